// The 16-byte pieces in which qv_kernel copies rows of Q (M x K, row-major, on any 8-byte boundary) to shared memory: plain
// address arithmetic, which host code can compile and check as well.
#pragma once

#include <stddef.h>
#include <stdint.h>

#ifdef __CUDACC__
#define QV_FN __host__ __device__ __forceinline__
#else
#define QV_FN inline
#endif

constexpr int QV_K = 32, QV_PIECES = 17;  // columns of a stage; pieces of a row that starts off the 16-byte grid (else 16)

// 1 for a row whose window (from column kbeg) starts 8 bytes off the 16-byte grid: it is then copied from one element before
QV_FN int qv_phase(const double *Q, int K, int row, int kbeg) {
    return (int)(((reinterpret_cast<uintptr_t>(Q) >> 3) + (size_t)row * K + kbeg) & 1);
}

struct QvPiece {
    const double *src;  // on a 16-byte boundary, also where nothing is read: the copy instruction asks for it
    int left;           // elements from the piece's first to the end of the range (<= 0: nothing to read)
};

// piece pc of the first stage of a row; further stages begin QV_K columns on each
QV_FN QvPiece qv_piece(const double *Q, int M, int K, int row, int kbeg, int kend, int pc) {
    // rows beyond the matrix read nothing from a place in its last row (a piece further on, so not before a lone first row)
    const bool in = row < M;
    const int r = in ? row : M - 1;
    const int k = kbeg - qv_phase(Q, K, r, kbeg) + 2 * (in ? pc : pc + 1);
    return {Q + ((ptrdiff_t)r * K + k), in ? kend - k : 0};
}

// source of a copy of n elements in the stage at column k0: the piece's own start where there is nothing to read.  (A piece
// that starts before Q has elements to read in every stage of its range, so the sum in the second case is src; without it
// the kernel's registers are dealt differently and it takes 2 % longer at 336 atoms x 370881 pairs, 10 columns.)
QV_FN const double *qv_source(const QvPiece &p, const double *Q, int k0, int n) {
    return n > 0 ? p.src + k0 : p.src + (Q > p.src);
}
