// Coulomb products of few columns, T = q_ov (s o V), G = gamma T and us = epilogue(q_ov^T G), for the Davidson's
// blocks of expansion vectors.  Included by dftb_kernels.cu inside its anonymous namespace.
//
// With m <= ~20 columns both q_ov products are bound by reading q_ov (8 nat nov bytes each); beyond that by the
// FP64 tensor pipe.  So the kernels stream q_ov once per product with no column padding beyond 8, feed it to
// mma.m8n8k4.f64 and keep the m-wide operands in shared memory.  Measured on B200 (the general 64 x 64 GEMM kernel
// that they replace pads every block to 64 columns), C294H42, 336 atoms x 370881 pairs, 10 columns, Hermitian form:
// T 2533 -> 241 us, G 49 -> 3.4 us, us 1187 -> 201 us (q_ov is 1.0 GB, 152 us at the copy rate); C1014H90, 1104 x
// 1500625, 10 columns without the square roots: T 2.60 ms, G 5.8 us, us 2.33 ms (13.2 GB, 2.03 ms).
#pragma once

#include "dmma.cuh"
#include "qv_pieces.cuh"

__device__ __forceinline__ void cp_async8(void *dst, const double *src, bool valid) {
    // 8-byte asynchronous copy; with src-size 0 the destination is zero-filled and nothing is read
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(valid ? 8 : 0)
                 : "memory");
}

// 16-byte asynchronous copy (L2 only) of the first `bytes` bytes (0..16); the rest of the destination is zero-filled
__device__ __forceinline__ void cp_async16(void *dst, const double *src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(bytes)
                 : "memory");
}

// The three kernels of a product are launched to overlap at their seams: each lets its successor's CTAs start when all of
// its own have, and waits for its predecessor's results (T, G) before it reads them.  At the smallest sizes the seams are a
// quarter of the time (B200, C20H22, 42 atoms x 2601 pairs, 10 columns: 24.6 -> 20.5 us; 17.7 with the present K ranges).
__device__ __forceinline__ void grid_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// ---------------------------------------------------------------------------- T = Q (s o V)
// A CTA takes 64 rows of Q and one of ksplit ranges of its columns, in 32-column stages of a four-deep cp.async ring
// that holds Q and V.  Q comes in 16-byte pieces.  nov is odd as often as not, so a row may start 8 bytes off the
// 16-byte grid: its window then begins one element early (at the row's `phase`) and takes a 17th piece, and the
// fragment reads add the phase.  Warps are 4 (rows) x 2 (halves of a stage), two row tiles each; for the Hermitian
// form four warps turn omega into sqrt(omega) every fourth stage (a square root is a long serial chain, so it should
// hold the stage's barrier up as seldom as possible), and the V fragments are multiplied as they are read.  Two CTAs per SM
// keep ~100 KB in flight.  The row pitches are 4 (mod 16) doubles, which keeps the fragment reads (nearly) conflict-free.
constexpr int QV_M = 64, QV_P = 36, QV_STAGES = 4, QV_THREADS = 256;

template <int NT> struct Skinny {  // NT tiles of 8 columns
    static constexpr int PITCH = 8 * NT + 4;
    static constexpr int STAGE = QV_M * QV_P + QV_K * PITCH;                        // doubles: Q, V
    static constexpr int SMEM = (int)sizeof(double) * (QV_STAGES * STAGE + 16 * QV_K);  // + sqrt(omega), omega x 8
};

struct QvP {
    int M, K;            // rows and columns of Q
    const double *Q;     // row-major, leading dimension K
    const double *V;     // K x ncol, leading dimension ldv
    int ncol, ldv;
    double *T;           // M x ncol, leading dimension ldt; accumulated with atomics (zeroed by the caller)
    int ldt;
    const double *omega; // scale V rows by sqrt(omega) (HERM)
    int kper;            // columns of Q per CTA, a multiple of QV_K
    int after;           // V comes from the kernel before, which this one may overlap
};

template <int NT, bool HERM>
__global__ void __launch_bounds__(QV_THREADS, 2) qv_kernel(const QvP p) {
    extern __shared__ __align__(16) double qv_sm[];
    using C = Skinny<NT>;
    constexpr int PV = C::PITCH, NCOL = 8 * NT, ROWS = QV_M * 16 / QV_THREADS, VREG = QV_K * NCOL / QV_THREADS;
    double *Ws = qv_sm + QV_STAGES * C::STAGE, *Wraw = Ws + 8 * QV_K;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int row0 = blockIdx.x * QV_M, c0 = blockIdx.z * NCOL;
    const int ncol = min(NCOL, p.ncol - c0);
    const int kbeg = blockIdx.y * p.kper, kend = min(p.K, kbeg + p.kper);
    const int niter = kend > kbeg ? (kend - kbeg + QV_K - 1) / QV_K : 0;
    grid_launch_dependents();
    if (p.after) grid_wait();
    auto phase = [&](int row) { return qv_phase(p.Q, p.K, row, kbeg); };
    // this thread's pieces of Q: number tid % 16 of rows tid / 16 + 16 j, and the 17th of row tid
    const int pc = tid & 15;
    QvPiece piece[ROWS];
    const double *src17 = nullptr;
#pragma unroll
    for (int j = 0; j < ROWS; ++j) piece[j] = qv_piece(p.Q, p.M, p.K, row0 + (tid >> 4) + 16 * j, kbeg, kend, pc);
    if (tid < QV_M && row0 + tid < p.M && phase(row0 + tid))
        src17 = qv_piece(p.Q, p.M, p.K, row0 + tid, kbeg, kend, 16).src;
    auto stage = [&](int it) {
        if (it < niter) {
            double *q = qv_sm + (it % QV_STAGES) * C::STAGE, *v = q + QV_M * QV_P;
            const int k0 = it * QV_K;
#pragma unroll
            for (int j = 0; j < ROWS; ++j) {
                double *dst = q + ((tid >> 4) + 16 * j) * QV_P + 2 * pc;
                const int n = min(2, max(0, piece[j].left - k0));
                if (piece[j].src + k0 >= p.Q)
                    cp_async16(dst, qv_source(piece[j], p.Q, k0, n), 8 * n);
                else  // the very first element of a Q that is itself off the grid: nothing lies before it
                    cp_async8(dst + 1, p.Q, n > 1);
            }
            if (src17) {
                const int n = min(1, max(0, kend - (kbeg + k0 + 31)));
                cp_async16(q + tid * QV_P + 32, n > 0 ? src17 + k0 : src17, 8 * n);
            }
#pragma unroll
            for (int r = 0; r < VREG; ++r) {
                const int idx = tid + r * QV_THREADS, kk = idx / NCOL, c = idx % NCOL, k = kbeg + k0 + kk;
                const bool ok = c < ncol && k < kend;
                cp_async8(v + kk * PV + c, ok ? p.V + ((size_t)k * p.ldv + c0 + c) : p.V, ok);
            }
        }
        if (HERM && warp == 0) {
            // omega five stages further on, so that it has landed when its square root is taken
            const int k = kbeg + (it + 5) * QV_K + lane;
            cp_async8(Wraw + ((it + 5) & 7) * QV_K + lane, k < kend ? p.omega + k : p.omega, k < kend);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    double acc[2][NT][2];
#pragma unroll
    for (int t = 0; t < 2; ++t)
#pragma unroll
        for (int n = 0; n < NT; ++n) acc[t][n][0] = acc[t][n][1] = 0.0;
    for (int s = 0; s < QV_STAGES - 1; ++s) stage(s);
    if (HERM && warp < 6) {
        const int k = kbeg + warp * QV_K + lane;
        Ws[warp * QV_K + lane] = k < kend ? sqrt(p.omega[k]) : 0.0;
    }
    const int wr = 16 * (warp & 3), wk = 16 * (warp >> 2);  // this warp's rows and half of a stage
    int aoff[2];
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        const int rl = wr + 8 * t + (lane >> 2);
        aoff[t] = rl * QV_P + wk + (lane & 3) + (row0 + rl < p.M ? phase(row0 + rl) : 0);
    }
    for (int it = 0; it < niter; ++it) {
        asm volatile("cp.async.wait_group %0;" ::"n"(QV_STAGES - 2) : "memory");
        __syncthreads();  // stage it has landed, and every warp has left stage it - 1
        stage(it + QV_STAGES - 1);
        // stages it + 2 .. it + 5, whose omega came with the groups up to stage it's; their slots of Ws were last
        // read in stages before it - 2
        if (HERM && (it & 3) == 0 && it > 0 && (warp >> 2) == ((it >> 2) & 1)) {
            const int s = ((it + 2 + (warp & 3)) & 7) * QV_K + lane;
            Ws[s] = sqrt(Wraw[s]);
        }
        const double *a = qv_sm + (it % QV_STAGES) * C::STAGE;
        const double *b = a + QV_M * QV_P + (wk + (lane & 3)) * PV + (lane >> 2);
        const double *w = Ws + (it & 7) * QV_K + wk + (lane & 3);
#pragma unroll
        for (int ks = 0; ks < QV_K / 8; ++ks) {
            const double a0 = a[aoff[0] + 4 * ks], a1 = a[aoff[1] + 4 * ks];
            const double s = HERM ? w[4 * ks] : 1.0;
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                const double bv = HERM ? s * b[4 * ks * PV + 8 * n] : b[4 * ks * PV + 8 * n];
                dmma884(acc[0][n][0], acc[0][n][1], a0, bv);
                dmma884(acc[1][n][0], acc[1][n][1], a1, bv);
            }
        }
    }
    if (niter > 0) {
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            const int row = row0 + wr + 8 * t + (lane >> 2);
            if (row >= p.M) continue;
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int c = 8 * n + 2 * (lane & 3) + e;
                    if (c < ncol) atomicAdd(p.T + (size_t)row * p.ldt + c0 + c, acc[t][n][e]);
                }
        }
    }
}

// ---------------------------------------------------------------------------- us = epilogue(Q^T G)
// A warp takes 32 consecutive pairs ia (four row tiles of the MMA) and runs over all atoms: its fragment reads of
// Q are four 64-byte pieces of four atoms' rows, straight into registers (the 32 pairs use whole sectors between
// them), two MMA steps ahead; G comes through shared memory, 32 atoms at a time.  No split: every output is
// written once, with the omega terms applied.
constexpr int QG_THREADS = 128, QG_K = 32;

struct QgP {
    int nov, nat;
    const double *Q, *G;  // nat x nov; nat x ncol, leading dimension ldg
    int ncol, ldg;
    const double *omega, *V;
    double *U;            // nov x ncol, leading dimension ldg as V
    double fac;
    int square;           // 1: omega^2 v + fac sqrt(omega) acc (Hermitian), 0: omega v + fac acc
};

template <int NT>
__global__ void __launch_bounds__(QG_THREADS) qg_kernel(const QgP p) {
    constexpr int PV = Skinny<NT>::PITCH, NCOL = 8 * NT, GREG = QG_K * NCOL / QG_THREADS;
    __shared__ double Gs[2][QG_K * PV];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int c0 = blockIdx.y * NCOL, ncol = min(NCOL, p.ncol - c0);
    const int ia0 = (blockIdx.x * (QG_THREADS / 32) + warp) * 32;
    const int nchunk = (p.nat + QG_K - 1) / QG_K;
    grid_launch_dependents();
    double gr[GREG];
    auto load_g = [&](int ch) {
#pragma unroll
        for (int r = 0; r < GREG; ++r) {
            const int idx = tid + r * QG_THREADS, kk = idx / NCOL, c = idx % NCOL, A = ch * QG_K + kk;
            gr[r] = (A < p.nat && c < ncol) ? p.G[(size_t)A * p.ldg + c0 + c] : 0.0;
        }
    };
    auto store_g = [&](int ch) {
#pragma unroll
        for (int r = 0; r < GREG; ++r) {
            const int idx = tid + r * QG_THREADS, kk = idx / NCOL, c = idx % NCOL;
            Gs[ch & 1][kk * PV + c] = gr[r];
        }
    };
    // this lane's four pairs (clamped: rows beyond the last pair are computed and dropped)
    const double *q[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) q[t] = p.Q + min(ia0 + 8 * t + (lane >> 2), p.nov - 1);
    double acc[4][NT][2];
#pragma unroll
    for (int t = 0; t < 4; ++t)
#pragma unroll
        for (int n = 0; n < NT; ++n) acc[t][n][0] = acc[t][n][1] = 0.0;
    constexpr int GRP = NT <= 2 ? 4 : 2, NGRP = QG_K / (4 * GRP);  // MMA steps per register group, groups per chunk
    double a[2][GRP][4];
    auto load_a = [&](int ch, int g, double (&dst)[GRP][4]) {
#pragma unroll
        for (int s = 0; s < GRP; ++s) {
            const int A = ch * QG_K + 4 * (GRP * g + s) + (lane & 3);
            const bool v = A < p.nat;
            const size_t off = v ? (size_t)A * p.nov : 0;
#pragma unroll
            for (int t = 0; t < 4; ++t) dst[s][t] = v ? __ldcs(q[t] + off) : 0.0;
        }
    };
    load_a(0, 0, a[0]);
    grid_wait();  // G
    load_g(0);
    store_g(0);
    __syncthreads();
    for (int ch = 0; ch < nchunk; ++ch) {
        if (ch + 1 < nchunk) load_g(ch + 1);
        const double *b = Gs[ch & 1] + (lane & 3) * PV + (lane >> 2);
#pragma unroll
        for (int g = 0; g < NGRP; ++g) {
            if (g + 1 < NGRP)
                load_a(ch, g + 1, a[(g + 1) & 1]);
            else if (ch + 1 < nchunk)
                load_a(ch + 1, 0, a[(g + 1) & 1]);
#pragma unroll
            for (int s = 0; s < GRP; ++s)
#pragma unroll
                for (int n = 0; n < NT; ++n) {
                    const double bv = b[4 * (GRP * g + s) * PV + 8 * n];
#pragma unroll
                    for (int t = 0; t < 4; ++t) dmma884(acc[t][n][0], acc[t][n][1], a[g & 1][s][t], bv);
                }
        }
        if (ch + 1 < nchunk) {
            store_g(ch + 1);  // buffer (ch + 1) & 1 was last read in chunk ch - 1, before the barrier below
            __syncthreads();
        }
    }
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        const int ia = ia0 + 8 * t + (lane >> 2);
        if (ia >= p.nov) continue;
        const double om = p.omega[ia];
        const double dia = p.square ? om * om : om, f = p.square ? p.fac * sqrt(om) : p.fac;
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int c = 8 * n + 2 * (lane & 3) + e;
                if (c < ncol) {
                    const size_t o = (size_t)ia * p.ldg + c0 + c;
                    p.U[o] = dia * p.V[o] + f * acc[t][n][e];
                }
            }
    }
}
