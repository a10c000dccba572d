// dftbaby_b200: FP64 CUDA kernels for the LR-TD-DFTB path on B200 (sm_100a).
//
// Every extern "C" entry point is declared in include/dftbaby_b200.h, which
// also documents argument shapes and the DFTBaby interface each one replaces.
// All matrices are row-major FP64 in device memory.  Nothing here allocates:
// scratch space comes from caller-provided workspaces.

#include <cublas_v2.h>
#include <cuda_runtime.h>
#include <dlfcn.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

#include <mutex>
#include <type_traits>

#include "dftbaby_b200.h"

namespace {

thread_local char g_last_error[256] = "";

int fail(int code, const char *what) {
    snprintf(g_last_error, sizeof(g_last_error), "%s", what);
    return code;
}

int check_launch(const char *where) {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        snprintf(g_last_error, sizeof(g_last_error), "%s: %s", where, cudaGetErrorString(e));
        return DFTB_ERR_CUDA;
    }
    return DFTB_OK;
}

inline cudaStream_t S(void *s) { return reinterpret_cast<cudaStream_t>(s); }
inline unsigned cdiv(long long a, long long b) { return (unsigned)((a + b - 1) / b); }

#include "sk_device.cuh"
#include "coulomb.cuh"

// ----------------------------------------------------------------------------
// S, H0 and dipoles (slako.f90:77-394).  A block takes the orbitals of 8 row atoms x 32 column atoms.  Its 256 threads
// first evaluate the splines of one atom pair each (an element's own evaluation took up to four splines, 50 per
// carbon pair, with six divisions each), then write the elements from them, a warp along each row.  The value is the
// reference's lower-triangle element for (max, min), so both triangles are written directly.  Four blocks per SM: the
// phases are short chains of loads between barriers, and 64 registers with a few spills (125 us, below) beat 80 without
// (136 us).  B200, C1014H90 (4146 orbitals): S and H0 846 -> 125 us (275 MB written, 42 us), D 879 -> 167 us (412 MB);
// C20H22: 19 -> 15 us each.
// ----------------------------------------------------------------------------
constexpr int SK_TA = 8, SK_TB = 32, SK_PAIRS = SK_TA * SK_TB;
constexpr int SK_ROWS = 64, SK_COLS = 160;  // orbitals of a tile with their (atom, l, axis) in shared memory

struct SkTile {
    int first[SK_TA + SK_TB + 2];  // orbital ranges of the row atoms (0 .. SK_TA) and of the column atoms (SK_TA + 1 ..)
    int rinfo[SK_ROWS], cinfo[SK_COLS];
    unsigned present, mask[SK_SHARED_PAIRS];
    unsigned char flags[SK_PAIRS];  // 1: proximate, 2: read as (later atom, earlier atom)
};

// an atom pair: r and the direction from the first to the second centre in the order in which its tables are read
struct SkPair {
    double r, e[3];
    int i, j, ipair;
    bool near;
};

__device__ __forceinline__ int orb_info(const OrbTables &O, int mu, int atom0) {
    return (O.ind[mu] - atom0) | O.ls[mu] << 8 | axis_of_m(O.ms[mu]) << 16;
}

// ranges, orbital tables, the thread's atom pair and the type pairs of the tile
__device__ __forceinline__ SkPair sk_tile_setup(SkTile &t, const OrbTables &O, int norb, int nat, const double *r,
                                                const double *x, const double *y, const double *z, const int *mprox,
                                                int A0, int B0) {
    const int tid = threadIdx.x;
    if (tid <= SK_TA) t.first[tid] = first_orbital(O.ind, norb, min(nat, A0 + tid));
    else if (tid <= SK_TA + 1 + SK_TB) t.first[tid] = first_orbital(O.ind, norb, min(nat, B0 + tid - SK_TA - 1));
    else if (tid < 64) {
        if (tid == 48) t.present = 0u;
        if (tid > 48 && tid <= 48 + SK_SHARED_PAIRS) t.mask[tid - 49] = 0u;
    }
    const int ia = tid / SK_TB, ib = tid % SK_TB, A = A0 + ia, B = B0 + ib;
    const bool in = A < nat && B < nat;
    SkPair p;
    p.i = max(A, B);
    p.j = min(A, B);
    p.r = p.e[0] = p.e[1] = p.e[2] = 0.0;
    p.near = in && mprox[(size_t)p.i * nat + p.j] != 0;
    if (in) pair_dir(nat, r, x, y, z, p.i, p.j, p.r, p.e);
    __syncthreads();
    const int row0 = t.first[0], row1 = t.first[SK_TA], col0 = t.first[SK_TA + 1], col1 = t.first[SK_TA + 1 + SK_TB];
    if (tid < SK_ROWS && row0 + tid < row1) t.rinfo[tid] = orb_info(O, row0 + tid, A0);
    const int c = tid - (SK_PAIRS - SK_COLS);
    if (c >= 0 && col0 + c < col1) t.cinfo[c] = orb_info(O, col0 + c, B0);
    const int fa = t.first[ia], fb = t.first[SK_TA + 1 + ib];
    bool straight = true;
    p.ipair = 0;
    p.near = p.near && fa < t.first[ia + 1] && fb < t.first[SK_TA + 2 + ib];
    if (p.near) {
        const int ta = O.typ[fa], tb = O.typ[fb], tmin = min(ta, tb), tmax = max(ta, tb);
        p.ipair = tmax * (tmax + 1) / 2 + tmin;
        straight = A >= B ? ta <= tb : tb <= ta;  // type of the later atom <= type of the earlier one
        if (!straight)
            for (int k = 0; k < 3; ++k) p.e[k] = -p.e[k];
    }
    t.flags[tid] = (p.near ? 1 : 0) | (straight ? 2 : 0);
    const unsigned here = __reduce_or_sync(0xffffffffu, p.near && p.ipair < SK_SHARED_PAIRS ? 1u << p.ipair : 0u);
    if ((tid & 31) == 0 && here) atomicOr(&t.present, here);
    __syncthreads();
    return p;
}

// filled and shared bits of a pair's tables; pairs beyond SK_SHARED_PAIRS look their own tables up
template <int NT>
__device__ __forceinline__ unsigned sk_pair_mask(const SkTile &t, const SkTables &TA, const SkTables *TB, int ipair,
                                                 const int (&tabs)[NT]) {
    if (ipair < SK_SHARED_PAIRS) return t.mask[ipair];
    unsigned m = 0;
#pragma unroll
    for (int q = 0; q < NT; ++q) {
        if (tabs[q] < TA.nsk && TA.filled[ipair * TA.nsk + tabs[q]] == 1) m |= 1u << q;
        if (TB && tabs[q] < TB->nsk && TB->filled[ipair * TB->nsk + tabs[q]] == 1) m |= 1u << (NT + q);
    }
    return m;
}

__global__ void __launch_bounds__(SK_PAIRS, 4) h0_and_s_kernel(int norb, int nat, OrbTables O, const double *r,
                                                               const double *x, const double *y, const double *z,
                                                               const int *mprox, const double *orben, SkTables TS,
                                                               SkTables TH, double *S, double *H0) {
    constexpr int tabs[5] = {0, 2, 4, 5, 6};  // ss, sp, ps, pp-pi, pp-sigma
    __shared__ double vals[13][SK_PAIRS];     // S tables, H tables, direction
    __shared__ SkTile t;
    const int A0 = blockIdx.y * SK_TA, B0 = blockIdx.x * SK_TB, tid = threadIdx.x;
    {
        const SkPair p = sk_tile_setup(t, O, norb, nat, r, x, y, z, mprox, A0, B0);
        sk_shared_tables(TS, &TH, tabs, t.present, t.mask);
        __syncthreads();
        if (p.near && p.i != p.j) {
            const unsigned m = sk_pair_mask(t, TS, &TH, p.ipair, tabs);
            SkBasis b = {};
            if (m >> 16)
                b = sk_basis(TS.knots + ((size_t)p.ipair * TS.nsk + sk_first_filled(TS, p.ipair, tabs)) * TS.npts,
                             TS.npts, p.r);
            sk_values(TS, p.ipair, tabs, p.r, b, m & 31u, m >> 16 & 31u, &vals[0][tid], SK_PAIRS);
            sk_values(TH, p.ipair, tabs, p.r, b, m >> 5 & 31u, m >> 21 & 31u, &vals[5][tid], SK_PAIRS);
        }
        for (int c = 0; c < 3; ++c) vals[10 + c][tid] = p.e[c];
    }
    __syncthreads();
    const int warp = tid >> 5, lane = tid & 31;
    const int row0 = t.first[0], row1 = t.first[SK_TA], col0 = t.first[SK_TA + 1], col1 = t.first[SK_TA + 1 + SK_TB];
    const double nan = __longlong_as_double(0x7ff8000000000000ULL);
    for (int col = col0 + lane; col < col1; col += 32) {
        const int ci = col - col0 < SK_COLS ? t.cinfo[col - col0] : orb_info(O, col, B0);
        const int ib = ci & 255, lc = ci >> 8 & 255, ac = ci >> 16;
        for (int row = row0 + warp; row < row1; row += SK_PAIRS / 32) {
            const int ri = row - row0 < SK_ROWS ? t.rinfo[row - row0] : orb_info(O, row, A0);
            const int ia = ri & 255, lr = ri >> 8 & 255, ar = ri >> 16;
            const int q = ia * SK_TB + ib, f = t.flags[q];
            const double *v = &vals[0][q];
            double s = 0.0, h = 0.0;
            if (A0 + ia == B0 + ib) {
                if (row == col && (f & 1)) {
                    s = 1.0;
                    h = orben[row];
                }
            } else if (f & 1) {
                const bool rf = (row > col) == ((f & 2) != 0);  // the row's orbital is the first one
                const double ang = (lr ? v[(10 + ar) * SK_PAIRS] : 1.0) * (lc ? v[(10 + ac) * SK_PAIRS] : 1.0);
                const int k = lr + lc < 2 ? (lr == lc ? 0 : ((lr == 1) == rf ? 2 : 1)) : 4;  // ss, ps, sp, pp-sigma
                s = v[k * SK_PAIRS];
                h = v[(5 + k) * SK_PAIRS];
                if (k == 4) {
                    const double spi = v[3 * SK_PAIRS], hpi = v[8 * SK_PAIRS], on = ar == ac ? 1.0 : 0.0;
                    s = on * spi + ang * (s - spi);
                    h = on * hpi + ang * (h - hpi);
                } else {
                    s *= ang;
                    h *= ang;
                }
                if (max(lr, lc) > 1) s = h = nan;
            }
            const size_t o = (size_t)row * norb + col;
            S[o] = s;
            H0[o] = h;
        }
    }
}

// D planes (3, norb, norb)
__global__ void __launch_bounds__(SK_PAIRS, 4) dipole_kernel(int norb, int nat, OrbTables O, const double *r,
                                                             const double *x, const double *y, const double *z,
                                                             const double *pos, const int *mprox, const double *Smat,
                                                             SkTables TD, double *D) {
    constexpr int tabs[8] = {3, 1, 4, 6, 13, 7, 8, 14};  // ss; sp pi, sigma; ps pi, sigma; pp
    __shared__ double vals[11][SK_PAIRS];                 // tables, direction
    __shared__ double centre[SK_TA + SK_TB][3];
    __shared__ SkTile t;
    const int A0 = blockIdx.y * SK_TA, B0 = blockIdx.x * SK_TB, tid = threadIdx.x;
    if (tid < 3 * (SK_TA + SK_TB)) {
        const int k = tid / 3, atom = k < SK_TA ? A0 + k : B0 + k - SK_TA;
        centre[k][tid % 3] = atom < nat ? pos[3 * atom + tid % 3] : 0.0;
    }
    {
        const SkPair p = sk_tile_setup(t, O, norb, nat, r, x, y, z, mprox, A0, B0);
        sk_shared_tables(TD, nullptr, tabs, t.present, t.mask);
        __syncthreads();
        if (p.near) {
            const unsigned m = sk_pair_mask(t, TD, nullptr, p.ipair, tabs);
            SkBasis b = {};
            if (m >> 16)
                b = sk_basis(TD.knots + ((size_t)p.ipair * TD.nsk + sk_first_filled(TD, p.ipair, tabs)) * TD.npts,
                             TD.npts, p.r);
            sk_values(TD, p.ipair, tabs, p.r, b, m & 255u, m >> 16 & 255u, &vals[0][tid], SK_PAIRS);
        }
        for (int c = 0; c < 3; ++c) vals[8 + c][tid] = p.e[c];
    }
    __syncthreads();
    const size_t plane = (size_t)norb * norb;
    const int warp = tid >> 5, lane = tid & 31;
    const int row0 = t.first[0], row1 = t.first[SK_TA], col0 = t.first[SK_TA + 1], col1 = t.first[SK_TA + 1 + SK_TB];
    for (int col = col0 + lane; col < col1; col += 32) {
        const int ci = col - col0 < SK_COLS ? t.cinfo[col - col0] : orb_info(O, col, B0);
        const int ib = ci & 255, lc = ci >> 8 & 255, ac = ci >> 16;
        for (int row = row0 + warp; row < row1; row += SK_PAIRS / 32) {
            const int ri = row - row0 < SK_ROWS ? t.rinfo[row - row0] : orb_info(O, row, A0);
            const int ia = ri & 255, lr = ri >> 8 & 255, ar = ri >> 16;
            const int q = ia * SK_TB + ib, f = t.flags[q];
            const double *v = &vals[0][q];
            double d[3] = {0.0, 0.0, 0.0};
            if (f & 1) {
                const bool lower = row >= col, st = (f & 2) != 0, rf = lower == st;
                const double s = Smat[lower ? (size_t)row * norb + col : (size_t)col * norb + row];
                // the second centre: the earlier atom where straight
                const double *o = centre[st == (A0 + ia >= B0 + ib) ? SK_TA + ib : ia];
                const int a1 = rf ? ar : ac, a2 = rf ? ac : ar;
                if (max(lr, lc) > 1) {
                    d[0] = d[1] = d[2] = __longlong_as_double(0x7ff8000000000000ULL);
                } else if (lr + lc == 0) {
                    const double d3 = v[0];
#pragma unroll
                    for (int c = 0; c < 3; ++c) d[c] = v[(8 + c) * SK_PAIRS] * d3;
                } else if (lr + lc == 1) {
                    const int b = lr == 1 ? ar : ac, tb = (lr == 1) == rf ? 3 : 1;  // ps or sp
                    const double dpi = v[tb * SK_PAIRS], w = v[(8 + b) * SK_PAIRS] * (v[(tb + 1) * SK_PAIRS] - dpi);
#pragma unroll
                    for (int c = 0; c < 3; ++c) d[c] = (c == b ? dpi : 0.0) + v[(8 + c) * SK_PAIRS] * w;
                } else {
                    const double d7 = v[5 * SK_PAIRS], d8 = v[6 * SK_PAIRS], cub = v[7 * SK_PAIRS] - d7 - 2.0 * d8;
                    const double ea = v[(8 + a1) * SK_PAIRS], eb = v[(8 + a2) * SK_PAIRS], w = ea * eb * cub;
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        const double ec = v[(8 + c) * SK_PAIRS];
                        double u = ec * w;
                        if (a1 == c) u += eb * d7;
                        if (c == a2) u += ea * d8;
                        if (a1 == a2) u += ec * d8;
                        d[c] = u;
                    }
                }
#pragma unroll
                for (int c = 0; c < 3; ++c) d[c] += o[c] * s;
            }
            const size_t out = (size_t)row * norb + col;
#pragma unroll
            for (int c = 0; c < 3; ++c) D[c * plane + out] = d[c];
        }
    }
}

__global__ void dircos_kernel(int nat, const double *pos, double *r, double *x, double *y, double *z) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = blockIdx.y;
    if (j >= nat || i >= nat) return;
    const double xc = pos[3 * i] - pos[3 * j], yc = pos[3 * i + 1] - pos[3 * j + 1],
                 zc = pos[3 * i + 2] - pos[3 * j + 2];
    const double rr = sqrt(xc * xc + yc * yc + zc * zc);
    const size_t o = (size_t)i * nat + j;
    r[o] = rr;
    if (rr > 0.0) {
        x[o] = xc / rr;
        y[o] = yc / rr;
        z[o] = zc / rr;
    } else {
        x[o] = 0.0;
        y[o] = 0.0;
        z[o] = 1.0;
    }
}

__global__ void gamma_kernel(int nat, const double *r, const double *sigma, double r_lr, double *g, double *glr) {
    const int B = blockIdx.x * blockDim.x + threadIdx.x;
    const int A = blockIdx.y;
    if (A >= nat || B >= nat) return;
    const size_t o = (size_t)A * nat + B;
    const double sa = sigma[A], sb = sigma[B];
    const double s2 = sa * sa + sb * sb;
    if (A == B) {
        g[o] = 1.0 / (sqrt(M_PI) * sa);
        if (glr) glr[o] = 1.0 / sqrt(M_PI * (sa * sa + 0.25 * r_lr * r_lr));
    } else {
        const double R = r[o];
        const double C = 1.0 / sqrt(2.0 * s2);
        g[o] = erf(C * R) / R;
        if (glr) {
            const double Clr = 1.0 / sqrt(2.0 * (s2 + 0.5 * r_lr * r_lr));
            glr[o] = erf(Clr * R) / R;
        }
    }
}

// rows per thread of the element-wise (norb, norb) kernels: enough loads and stores in flight to reach HBM speed
constexpr int AO_ROWS = 8;

__global__ void ao_expand_kernel(int norb, int nat, const int *ind, const double *g, double *G) {
    const int nu = blockIdx.x * blockDim.x + threadIdx.x;
    if (nu >= norb) return;
    const double *col = g + ind[nu];
    const int mu0 = blockIdx.y * AO_ROWS, mu1 = min(norb, mu0 + AO_ROWS);
#pragma unroll
    for (int mu = mu0; mu < mu0 + AO_ROWS; ++mu)
        if (mu < mu1) G[(size_t)mu * norb + nu] = col[(size_t)ind[mu] * nat];
}

// estat[A] = sum_B gamma[A][B] dq[B]; one warp per atom
__global__ void estat_kernel(int nat, const double *gamma, const double *dq, double *estat) {
    const int A = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
    const int lane = threadIdx.x % 32;
    if (A >= nat) return;
    double acc = 0.0;
    for (int B = lane; B < nat; B += 32) acc += gamma[(size_t)A * nat + B] * dq[B];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, off);
    if (lane == 0) estat[A] = acc;
}

__global__ void scc_h_kernel(int norb, const int *ind, const double *H0, const double *Smat, const double *estat,
                             double *H) {
    const int nu = blockIdx.x * blockDim.x + threadIdx.x;
    if (nu >= norb) return;
    const double en = estat[ind[nu]];
    const int mu0 = blockIdx.y * AO_ROWS, mu1 = min(norb, mu0 + AO_ROWS);
#pragma unroll
    for (int mu = mu0; mu < mu0 + AO_ROWS; ++mu)
        if (mu < mu1) {
            const size_t o = (size_t)mu * norb + nu;
            const double h1 = 0.5 * (estat[ind[mu]] + en);
            H[o] = H0[o] + h1 * Smat[o];
        }
}

// Mulliken monopoles: one block per atom, reduction over its rows.
__global__ void monopoles_kernel(int norb, int nat, const double *P, const double *P0, const double *Smat,
                                 const int *opa, double *q, double *dq) {
    const int A = blockIdx.x;
    __shared__ int first_s;
    __shared__ double red_q[32], red_d[32];
    if (threadIdx.x == 0) {
        int f = 0;
        for (int B = 0; B < A; ++B) f += opa[B];
        first_s = f;
    }
    __syncthreads();
    const int first = first_s, n = opa[A];
    double aq = 0.0, ad = 0.0;
    for (int k = 0; k < n; ++k) {
        const size_t row = (size_t)(first + k) * norb;
        for (int nu = threadIdx.x; nu < norb; nu += blockDim.x) {
            const double s = Smat[row + nu], p = P[row + nu];
            aq += p * s;
            ad += (p - P0[row + nu]) * s;
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        aq += __shfl_down_sync(0xffffffffu, aq, off);
        ad += __shfl_down_sync(0xffffffffu, ad, off);
    }
    const int w = threadIdx.x / 32, lane = threadIdx.x % 32;
    if (lane == 0) {
        red_q[w] = aq;
        red_d[w] = ad;
    }
    __syncthreads();
    if (w == 0) {
        const int nw = blockDim.x / 32;
        aq = lane < nw ? red_q[lane] : 0.0;
        ad = lane < nw ? red_d[lane] : 0.0;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            aq += __shfl_down_sync(0xffffffffu, aq, off);
            ad += __shfl_down_sync(0xffffffffu, ad, off);
        }
        if (lane == 0) {
            q[A] = aq;
            dq[A] = ad;
        }
    }
}

// ----------------------------------------------------------------------------
// FP64 GEMM engine on the FP64 tensor tiles (mma.m8n8k4):
//   C(m,n) = alpha * sum_k A(m,k) B(k,n) [+ beta C]
// with arbitrary element strides, a batch index, optional split-K (atomic accumulation) and two-level indices: k in A
// as (k / K2, k % K2), n in B and C as (n / N2, n % N2), so that a sum over (atom, orbital) pairs or an output of
// (orbital, vector) columns is one product without reordering its operands.
// A CTA of four warps takes a 64 x 64 tile (a warp 32 x 32) in 16-deep stages of a three-deep cp.async ring.  Each
// operand is staged in the order in which it is contiguous in memory, with a pitch of 4 (mod 16) doubles either way,
// so copies and fragment reads are both conflict-free; tiles of 8 rows beyond M are skipped.  Bound by the FP64 pipe:
// 30 TFLOP/s at 4096^3 on B200 (the 4 x 4 register-tile form it replaces ran at 9 to 13; cuBLAS 35).
// ----------------------------------------------------------------------------
enum { EPI_STORE = 0, EPI_ATOMIC = 1 };

struct GemmP {
    int M, N, K;
    const double *A;
    long long sam, sak, sak1, sa1;  // strides of m, k % K2, k / K2, batch
    int K2;                         // two-level k needs sak == 1 (else K2 = K)
    const double *B;
    long long sbk, sbn, sbn1, sb1;  // strides of k, n % N2, n / N2, batch
    double *C;
    long long scm, scn, scn1, sc1;
    int N2;
    double alpha, beta;
    int ksplit;  // gridDim.z = nbatch * ksplit
    int mstep;   // rows per CTA, a multiple of 8 and at most BM: the 8-row tiles of M dealt evenly to the CTAs
};

constexpr int BM = 64, BN = 64, BK = 16, GEMM_STAGES = 3, GEMM_THREADS = 128;
constexpr int PITCH_K = BK + 4, PITCH_MN = BM + 4;  // operand tiles [m or n][k] and [k][m or n]

// AK: A is contiguous along k (else staged along m); BNC: B is contiguous along n (else staged along k)
template <int EPI, bool AK, bool BNC>
__device__ __forceinline__ void dgemm_tile(const GemmP &p, int bx, int by, int bz) {
    constexpr int A_ELEMS = AK ? BM * PITCH_K : BK * PITCH_MN, B_ELEMS = BNC ? BK * PITCH_MN : BN * PITCH_K;
    extern __shared__ __align__(16) double gemm_sm[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int bm = by * p.mstep, bn = bx * BN, M = min(p.M, bm + p.mstep);
    const int zb = bz / p.ksplit, zk = bz % p.ksplit;
    const double *A = p.A + zb * p.sa1, *B = p.B + zb * p.sb1;
    double *C = p.C + zb * p.sc1;
    const int kchunk = ((p.K + p.ksplit - 1) / p.ksplit + BK - 1) / BK * BK;
    const int k0 = zk * kchunk, k1 = min(p.K, k0 + kchunk);
    const int niter = k1 > k0 ? (k1 - k0 + BK - 1) / BK : 0;
    auto noff = [&](int n, long long s1, long long s2) {
        const int q = p.N2 >= p.N ? 0 : n / p.N2;  // no division for a plain index
        return q * s1 + (n - q * p.N2) * s2;
    };

    // this thread's part of a stage: eight elements of each operand, along its contiguous index from thread to thread
    const int ka = AK ? tid & 15 : tid >> 6, ma = AK ? tid >> 4 : tid & 63;
    const int kb = BNC ? tid >> 6 : tid & 15, nb = BNC ? tid & 63 : tid >> 4;
    int kq = p.K2 >= p.K ? 0 : (k0 + ka) / p.K2, kr = k0 + ka - kq * p.K2;  // two-level k of A (AK)
    const double *bcol = B + (BNC && bn + nb < p.N ? noff(bn + nb, p.sbn1, p.sbn) : 0);
    long long boff[8];
    if (!BNC) {
#pragma unroll
        for (int i = 0; i < 8; ++i) boff[i] = bn + nb + 8 * i < p.N ? noff(bn + nb + 8 * i, p.sbn1, p.sbn) : -1;
    }
    auto stage = [&](int it) {
        if (it < niter) {
            double *as = gemm_sm + (it % GEMM_STAGES) * (A_ELEMS + B_ELEMS), *bs = as + A_ELEMS;
            const int kt = k0 + it * BK;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int mm = AK ? ma + 8 * i : ma, kk = AK ? ka : ka + 2 * i;
                const bool v = bm + mm < M && kt + kk < k1;
                const long long ko = AK ? kq * p.sak1 + kr * p.sak : (long long)(kt + kk) * p.sak;
                cp_async8(as + (AK ? mm * PITCH_K + kk : kk * PITCH_MN + mm),
                          v ? A + ((long long)(bm + mm) * p.sam + ko) : A, v);
            }
            if (AK) {
                kr += BK;
                while (kr >= p.K2) {
                    kr -= p.K2;
                    ++kq;
                }
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int nn = BNC ? nb : nb + 8 * i, kk = BNC ? kb + 2 * i : kb;
                const bool v = bn + nn < p.N && kt + kk < k1;
                const double *src = (BNC ? bcol : B + (v ? boff[BNC ? 0 : i] : 0)) + (v ? (kt + kk) * p.sbk : 0);
                cp_async8(bs + (BNC ? kk * PITCH_MN + nn : nn * PITCH_K + kk), v ? src : B, v);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    double acc[4][4][2];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
    // neighbouring CTAs swap the upper and lower warps, so that short tiles do not all fall to the same SM quarters
    const int wm = 32 * ((warp ^ bx) & 1), wn = 32 * (warp >> 1);
    const int mtiles = min(4, max(0, (M - bm - wm + 7) / 8)), ntiles = min(4, max(0, (p.N - bn - wn + 7) / 8));
    const int arow = wm + (lane >> 2), acol = lane & 3, bcol_l = wn + (lane >> 2);
    for (int s = 0; s < GEMM_STAGES - 1; ++s) stage(s);
    for (int it = 0; it < niter; ++it) {
        asm volatile("cp.async.wait_group %0;" ::"n"(GEMM_STAGES - 2) : "memory");
        __syncthreads();  // stage it has landed, and every warp has left stage it - 1
        stage(it + GEMM_STAGES - 1);
        const double *as = gemm_sm + (it % GEMM_STAGES) * (A_ELEMS + B_ELEMS), *bs = as + A_ELEMS;
        auto step = [&](int ks, auto full) {
            double a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
                a[i] = AK ? as[(arow + 8 * i) * PITCH_K + ks + acol] : as[(ks + acol) * PITCH_MN + arow + 8 * i];
#pragma unroll
            for (int j = 0; j < 4; ++j)
                b[j] = BNC ? bs[(ks + acol) * PITCH_MN + bcol_l + 8 * j] : bs[(bcol_l + 8 * j) * PITCH_K + ks + acol];
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (decltype(full)::value || i < mtiles) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) dmma884(acc[i][j][0], acc[i][j][1], a[i], b[j]);
                }
        };
        if (ntiles == 0) continue;
        if (mtiles == 4) {  // without branches between the MMAs
#pragma unroll
            for (int ks = 0; ks < BK; ks += 4) step(ks, std::true_type());
        } else {
#pragma unroll
            for (int ks = 0; ks < BK; ks += 4) step(ks, std::false_type());
        }
    }
    if (EPI == EPI_ATOMIC && niter == 0) return;
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int n = bn + wn + 8 * j + 2 * (lane & 3) + e;
            if (n >= p.N) continue;
            double *col = C + noff(n, p.scn1, p.scn);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int m = bm + arow + 8 * i;
                if (m >= M) continue;
                double *c = col + m * p.scm;
                const double val = p.alpha * acc[i][j][e];
                if (EPI == EPI_STORE)
                    *c = (p.beta == 0.0) ? val : val + p.beta * (*c);
                else
                    atomicAdd(c, val);
            }
        }
}

template <int EPI, bool AK, bool BNC>
__global__ void __launch_bounds__(GEMM_THREADS) dgemm_kernel(const GemmP p) {
    dgemm_tile<EPI, AK, BNC>(p, blockIdx.x, blockIdx.y, blockIdx.z);
}

// Several independent products in one launch: CTAs first[t] .. first[t + 1] - 1 take the tiles of product t.
constexpr int GROUP = 4;
struct GemmGroup {
    GemmP p[GROUP];
    int gx[GROUP], gy[GROUP], first[GROUP + 1];
    int n;
};

// WAIT_FIRST: the operands come from the kernel before, which this launch may overlap; else they do not, and the wait at the
// end only hands the order of the launches on to the next one.
template <int EPI, bool WAIT_FIRST>
__global__ void __launch_bounds__(GEMM_THREADS) dgemm_group_kernel(const __grid_constant__ GemmGroup g) {
    int t = 0;
    while (t + 1 < g.n && (int)blockIdx.x >= g.first[t + 1]) ++t;
    const GemmP &p = g.p[t];
    const int b = blockIdx.x - g.first[t], bx = b % g.gx[t], r = b / g.gx[t], by = r % g.gy[t], bz = r / g.gy[t];
    grid_launch_dependents();
    if (WAIT_FIRST) grid_wait();
    if (p.sbn == 1) {
        if (p.sak == 1)
            dgemm_tile<EPI, true, true>(p, bx, by, bz);
        else
            dgemm_tile<EPI, false, true>(p, bx, by, bz);
    } else {
        if (p.sak == 1)
            dgemm_tile<EPI, true, false>(p, bx, by, bz);
        else
            dgemm_tile<EPI, false, false>(p, bx, by, bz);
    }
    if (!WAIT_FIRST) grid_wait();
}

// a launch that may overlap the end of the kernel before it on the stream
template <typename K, typename P>
cudaError_t launch_overlapped(K kernel, dim3 grid, unsigned threads, size_t smem, cudaStream_t st, const P &p, bool overlap) {
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = overlap ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, p);
}

GemmP gemm_defaults() {
    GemmP p;
    memset(&p, 0, sizeof(p));
    p.alpha = 1.0;
    p.ksplit = 1;
    return p;
}

template <int EPI, bool AK, bool BNC>
int launch_gemm_as(const GemmP &p, dim3 grid, cudaStream_t st) {
    constexpr int smem =
        GEMM_STAGES * (int)sizeof(double) * ((AK ? BM * PITCH_K : BK * PITCH_MN) + (BNC ? BK * PITCH_MN : BN * PITCH_K));
    static bool attr_set[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !attr_set[dev]) {
        if (cudaFuncSetAttribute(dgemm_kernel<EPI, AK, BNC>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) !=
            cudaSuccess)
            return fail(DFTB_ERR_CUDA, "gemm: shared memory");
        if (dev >= 0 && dev < 64) attr_set[dev] = true;
    }
    dgemm_kernel<EPI, AK, BNC><<<grid, GEMM_THREADS, smem, st>>>(p);
    return check_launch("dgemm_kernel");
}

// the grid of a product, and its parameters brought to the form that the kernel reads; an error code
int plan_gemm(GemmP &p, int nbatch, dim3 &grid) {
    if (p.K <= 0) return fail(DFTB_ERR_BAD_SIZE, "gemm: K <= 0");
    if (p.K2 == 0) p.K2 = p.K;
    if (p.N2 == 0) p.N2 = p.N;
    // an inner index of one value: its stride is never taken, and the outer one says how the operand lies in memory
    if (p.K2 == 1) {
        p.sak = p.sak1;
        p.K2 = p.K;
    }
    if (p.N2 == 1) {
        p.sbn = p.sbn1;
        p.scn = p.scn1;
        p.N2 = p.N;
    }
    const int mblocks = (int)cdiv(p.M, BM);
    p.mstep = 8 * (int)cdiv(cdiv(p.M, 8), mblocks);
    grid = dim3(cdiv(p.N, BN), mblocks, (unsigned)(nbatch * p.ksplit));
    if (grid.y > 65535u || grid.z > 65535u) return fail(DFTB_ERR_BAD_SIZE, "gemm: grid too large");
    if (p.K2 != p.K && p.sak != 1) return fail(DFTB_ERR_BAD_SIZE, "gemm: two-level k");
    return DFTB_OK;
}

int launch_gemm(GemmP p, int epi, int nbatch, cudaStream_t st) {
    if (p.M <= 0 || p.N <= 0 || nbatch <= 0) return DFTB_OK;
    dim3 grid;
    const int rc = plan_gemm(p, nbatch, grid);
    if (rc) return rc;
    const bool ak = p.sak == 1, bn = p.sbn == 1;
    if (epi == EPI_STORE)
        return ak ? (bn ? launch_gemm_as<EPI_STORE, true, true>(p, grid, st)
                        : launch_gemm_as<EPI_STORE, true, false>(p, grid, st))
                  : (bn ? launch_gemm_as<EPI_STORE, false, true>(p, grid, st)
                        : launch_gemm_as<EPI_STORE, false, false>(p, grid, st));
    return ak ? (bn ? launch_gemm_as<EPI_ATOMIC, true, true>(p, grid, st)
                    : launch_gemm_as<EPI_ATOMIC, true, false>(p, grid, st))
              : (bn ? launch_gemm_as<EPI_ATOMIC, false, true>(p, grid, st)
                    : launch_gemm_as<EPI_ATOMIC, false, false>(p, grid, st));
}

// n products in one launch that may overlap the end of the kernel before it
template <int EPI, bool WAIT_FIRST>
int launch_gemm_group(const GemmP *p, const int *nbatch, int n, cudaStream_t st) {
    constexpr int smem = GEMM_STAGES * (int)sizeof(double) * 2 * BM * PITCH_K;  // the larger staging order of both operands
    GemmGroup g;
    memset(&g, 0, sizeof(g));
    g.n = n;
    long long ctas = 0;
    for (int t = 0; t < n; ++t) {
        dim3 grid;
        g.p[t] = p[t];
        const int rc = plan_gemm(g.p[t], nbatch[t], grid);
        if (rc) return rc;
        g.gx[t] = (int)grid.x;
        g.gy[t] = (int)grid.y;
        g.first[t] = (int)ctas;
        ctas += (long long)grid.x * grid.y * grid.z;
    }
    if (ctas > (1LL << 30)) return fail(DFTB_ERR_BAD_SIZE, "gemm: grid too large");
    g.first[n] = (int)ctas;
    cudaError_t e = cudaFuncSetAttribute(dgemm_group_kernel<EPI, WAIT_FIRST>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         smem);
    if (e != cudaSuccess) return fail(DFTB_ERR_CUDA, "gemm: shared memory");
    launch_overlapped(dgemm_group_kernel<EPI, WAIT_FIRST>, dim3((unsigned)ctas), GEMM_THREADS, smem, st, g, true);
    return check_launch("dgemm_group_kernel");
}

// K ranges so that about `ctas` CTAs are in flight, of at least `stages` stages each
int pick_ksplit(int M, int N, int K, int ctas, int stages) {
    const long long tiles = (long long)cdiv(M, BM) * cdiv(N, BN);
    const long long want = ctas / tiles, most = K / (stages * BK);
    return (int)(want < 1 || most < 1 ? 1 : (want < most ? want : most));
}

// ----------------------------------------------------------------------------
// transition charges
// ----------------------------------------------------------------------------
// first[A] = orbitals before atom A, first[nat] = all of them: one block scans (one thread did, 17 us at 336 atoms)
constexpr int PREFIX_THREADS = 512;

__global__ void __launch_bounds__(PREFIX_THREADS) prefix_kernel(int nat, const int *opa, int *first) {
    __shared__ int wsum[PREFIX_THREADS / 32];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    int base = 0;
    for (int A0 = 0; A0 < nat; A0 += PREFIX_THREADS) {
        const int A = A0 + t, v = A < nat ? opa[A] : 0;
        int x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) wsum[warp] = x;
        __syncthreads();
        int before = base, all = 0;
        for (int w = 0; w < PREFIX_THREADS / 32; ++w) {
            if (w < warp) before += wsum[w];
            all += wsum[w];
        }
        if (A < nat) first[A] = before + x - v;
        base += all;
        __syncthreads();
    }
    if (t == 0) first[nat] = base;
}

// q[A][p][q] = 1/2 sum_{mu in A} (C1[mu][p] Sc2[mu][q] + Sc1[mu][p] C2[mu][q]).
// The output (nat x n1 x n2 doubles) is the only large stream and its rows start at any multiple of 8 bytes.  A warp
// owns one atom and TC_Q columns, holds the atom's S c and c of those columns as B fragments of the FP64 tensor
// instruction (K = up to four orbitals, twice) in registers, and walks over blocks of 8 rows p: two loads, 32
// instructions, and the 8 x TC_Q block goes to the warp's own shared-memory buffer and from there to memory by one
// asynchronous bulk copy per row, 16-byte aligned, with the odd element of a row's ends stored singly.  Two buffers a
// warp; no barriers.  Bound by the writes.  (Outputs from registers, 16-byte stores through shuffles, two FP64 units'
// worth of FMAs each: L1 80 % and FP64 67 % busy, 3.7 TB/s of writes.  B200, C294H42 with 609 x 609 orbitals, 3.0 GB:
// 747 us so, 530 us here; filling the same memory takes 402 us.)
constexpr int TC_Q = 128, TC_WARPS = 4, TC_THREADS = 32 * TC_WARPS, TC_BLOCKS = 8;
// Row pitch of the staging buffer.  Rows that all start on a 16-byte boundary are staged by 16-byte stores, free of
// bank conflicts at 136; rows of both alignments by 8-byte stores, free of them at 130.
constexpr int TC_PITCH16 = 136, TC_PITCH8 = 130;
constexpr int TC_BUF = 8 * TC_PITCH16;
constexpr int TC_SMEM = TC_WARPS * 2 * TC_BUF * (int)sizeof(double);

__global__ void __launch_bounds__(TC_THREADS, 3) tc_kernel(int n1, int n2, const int *first,
                                                           const double *__restrict__ C1,
                                                           const double *__restrict__ Sc1,
                                                           const double *__restrict__ C2,
                                                           const double *__restrict__ Sc2, double *q) {
    extern __shared__ __align__(16) double tc_buf[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, kk = lane & 3, rr = lane >> 2;
    double *buf = tc_buf + warp * 2 * TC_BUF;
    const int A = blockIdx.z, q0 = blockIdx.x * TC_Q, ncols = min(TC_Q, n2 - q0);
    const int f0 = first[A], nA = first[A + 1] - f0;
    const int nblocks = (n1 + 7) / 8, stride = gridDim.y * TC_WARPS;
    double *qA = q + (size_t)A * n1 * n2 + q0;
    const bool vec = (n2 & 1) == 0 && (reinterpret_cast<uintptr_t>(q) & 15) == 0;
    const int pitch = vec ? TC_PITCH16 : TC_PITCH8;
    // one value of a (norb x n) matrix, zero outside
    auto at = [&](const double *X, int n, int j, int c) {
        return j < nA && c < n ? __ldg(X + (size_t)(f0 + j) * n + c) : 0.0;
    };
    double bs[TC_Q / 8], bc[TC_Q / 8];
#pragma unroll
    for (int t = 0; t < TC_Q / 8; ++t) {
        bs[t] = at(Sc2, n2, kk, q0 + 8 * t + rr);
        bc[t] = at(C2, n2, kk, q0 + 8 * t + rr);
    }
    int pb = blockIdx.y * TC_WARPS + warp;
    double ac = at(C1, n1, kk, 8 * pb + rr), as = at(Sc1, n1, kk, 8 * pb + rr);
    for (int step = 0; pb < nblocks; pb += stride, ++step) {
        double *out = buf + (step & 1) * TC_BUF;
        const int p0 = 8 * pb;
        const double ac0 = 0.5 * ac, as0 = 0.5 * as;
        ac = at(C1, n1, kk, p0 + 8 * stride + rr);  // the next block's
        as = at(Sc1, n1, kk, p0 + 8 * stride + rr);
        // the copies issued two steps ago have read this buffer
        asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
        __syncwarp();
        const int phase = (int)((reinterpret_cast<uintptr_t>(qA + (size_t)(p0 + rr) * n2) >> 3) & 1);
        double *o = out + rr * pitch + phase + 2 * kk;
#pragma unroll
        for (int t = 0; t < TC_Q / 8; ++t) {
            if (8 * t >= ncols) break;
            double d0 = 0.0, d1 = 0.0;
            dmma884(d0, d1, ac0, bs[t]);
            dmma884(d0, d1, as0, bc[t]);
            for (int j = 4; j < nA; j += 4) {  // atoms with d shells: the further orbitals, four at a time
                dmma884(d0, d1, 0.5 * at(C1, n1, j + kk, p0 + rr), at(Sc2, n2, j + kk, q0 + 8 * t + rr));
                dmma884(d0, d1, 0.5 * at(Sc1, n1, j + kk, p0 + rr), at(C2, n2, j + kk, q0 + 8 * t + rr));
            }
            if (vec) {
                *reinterpret_cast<double2 *>(o + 8 * t) = make_double2(d0, d1);
            } else {
                o[8 * t] = d0;
                o[8 * t + 1] = d1;
            }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        // lanes 0..7: the 16-byte aligned part of row lane; 8..15 an odd first element, 16..23 an odd last one
        const int r = lane & 7;
        if (p0 + r < n1) {
            double *dst = qA + (size_t)(p0 + r) * n2;
            const int head = (int)((reinterpret_cast<uintptr_t>(dst) >> 3) & 1), body = (ncols - head) & ~1;
            const double *src = out + r * pitch + head;
            if (lane < 8) {
                if (body > 0)
                    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst + head),
                                 "r"(static_cast<uint32_t>(__cvta_generic_to_shared(src + head))), "r"(body * 8)
                                 : "memory");
            } else if (lane < 16) {
                if (head) dst[0] = src[0];
            } else if (lane < 24) {
                if (head + body < ncols) dst[ncols - 1] = src[ncols - 1];
            }
        }
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    }
    asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

// one (n1 x n2) block of transition charges for all atoms
int launch_tc(int nat, int n1, int n2, const int *first, const double *C1, const double *Sc1, const double *C2,
              const double *Sc2, double *out, cudaStream_t st, const char *where) {
    // about TC_BLOCKS row blocks a warp: enough to pay for its B fragments, few enough to fill the GPU (609 x 609 orbitals,
    // 336 atoms: 552, 530, 543 and 582 us with 4, 8, 16 and 32)
    dim3 grid(cdiv(n2, TC_Q), cdiv(cdiv(n1, 8), TC_WARPS * TC_BLOCKS), nat);
    if (grid.y > 65535u || grid.z > 65535u) return fail(DFTB_ERR_BAD_SIZE, "trans_charges: grid too large");
    cudaError_t e = cudaFuncSetAttribute(tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, TC_SMEM);
    if (e != cudaSuccess) return fail(DFTB_ERR_CUDA, "trans_charges: shared memory");
    tc_kernel<<<grid, TC_THREADS, TC_SMEM, st>>>(n1, n2, first, C1, Sc1, C2, Sc2, out);
    return check_launch(where);
}

// diagonal q^{pp}_A
__global__ void tc_diag_kernel(int n, const int *first, const double *C, const double *Sc, double *q) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    const int A = blockIdx.y;
    if (p >= n) return;
    double acc = 0.0;
    for (int mu = first[A]; mu < first[A + 1]; ++mu)
        acc += C[(size_t)mu * n + p] * Sc[(size_t)mu * n + p] + C[(size_t)mu * n + p] * Sc[(size_t)mu * n + p];
    q[(size_t)A * n + p] = 0.5 * acc;
}

// cuBLAS for plain FP64 GEMMs (the wide Coulomb product's two, the transition charges' S.C).  The library is resolved at run
// time (dlopen / dlsym, reusing the copy the process has already loaded), so the shared library
// loads without it and the product falls back to dgemm_kernel.
using blas_create_t = cublasStatus_t (*)(cublasHandle_t *);
using blas_stream_t = cublasStatus_t (*)(cublasHandle_t, cudaStream_t);
using blas_dgemm_t = cublasStatus_t (*)(cublasHandle_t, cublasOperation_t, cublasOperation_t, int, int, int,
                                        const double *, const double *, int, const double *, int, const double *,
                                        double *, int);
struct Blas {
    blas_create_t create = nullptr;
    blas_stream_t set_stream = nullptr;
    blas_dgemm_t dgemm = nullptr;
    bool ok = false;
};

Blas &blas() {
    static Blas b;
    static std::once_flag once;
    std::call_once(once, [] {
        void *h = dlopen("libcublas.so.12", RTLD_NOW | RTLD_NOLOAD);
        if (!h) h = dlopen("libcublas.so.12", RTLD_NOW | RTLD_GLOBAL);
        if (!h) h = dlopen("libcublas.so", RTLD_NOW | RTLD_GLOBAL);
        if (!h) return;
        b.create = reinterpret_cast<blas_create_t>(dlsym(h, "cublasCreate_v2"));
        b.set_stream = reinterpret_cast<blas_stream_t>(dlsym(h, "cublasSetStream_v2"));
        b.dgemm = reinterpret_cast<blas_dgemm_t>(dlsym(h, "cublasDgemm_v2"));
        b.ok = b.create && b.set_stream && b.dgemm;
    });
    return b;
}

// one handle per host thread and device, bound to the caller's stream; nullptr if unavailable
cublasHandle_t blas_handle(cudaStream_t st) {
    Blas &b = blas();
    if (!b.ok) return nullptr;
    thread_local cublasHandle_t handles[64] = {nullptr};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
    if (!handles[dev] && b.create(&handles[dev]) != CUBLAS_STATUS_SUCCESS) {
        handles[dev] = nullptr;
        return nullptr;
    }
    if (b.set_stream(handles[dev], st) != CUBLAS_STATUS_SUCCESS) return nullptr;
    return handles[dev];
}

size_t align256(size_t b) { return (b + 255) / 256 * 256; }

// use_blas: S.C by cuBLAS when it resolves (the entry points that may allocate; the allocation-free one
// keeps the library's own dgemm_kernel)
int trans_charges_common(int norb, int nat, int nocc, int nvirt, const double *co, const double *cv,
                         const double *Smat, const int *opa, void *work, size_t work_bytes, cudaStream_t st,
                         double **sco, double **scv, int **first, bool use_blas = true) {
    if (norb <= 0 || nat <= 0 || nocc < 0 || nvirt < 0) return fail(DFTB_ERR_BAD_SIZE, "trans_charges: sizes");
    if (!Smat || !opa || (nocc > 0 && !co) || (nvirt > 0 && !cv)) return fail(DFTB_ERR_NULL, "trans_charges: null");
    if (!work || work_bytes < dftb_trans_charges_workspace_size(norb, nocc, nvirt))
        return fail(DFTB_ERR_WORKSPACE, "trans_charges: workspace too small");
    char *w = (char *)work;
    *sco = (double *)w;
    w += align256(sizeof(double) * (size_t)norb * nocc);
    *scv = (double *)w;
    w += align256(sizeof(double) * (size_t)norb * nvirt);
    *first = (int *)w;
    prefix_kernel<<<1, PREFIX_THREADS, 0, st>>>(nat, opa, *first);
    int rc = check_launch("prefix_kernel");
    if (rc) return rc;
    // Sc = S . C (S is symmetric)
    cublasHandle_t bh = use_blas ? blas_handle(st) : nullptr;
    for (int b = 0; b < 2; ++b) {
        const int n = b == 0 ? nocc : nvirt;
        if (n == 0) continue;
        if (bh) {
            // row-major Sc (norb x n) is the column-major Sc^T = C^T S^T = C^T S
            const double one = 1.0, zero = 0.0;
            if (blas().dgemm(bh, CUBLAS_OP_N, CUBLAS_OP_N, n, norb, norb, &one, b == 0 ? co : cv, n, Smat, norb, &zero,
                             b == 0 ? *sco : *scv, n) != CUBLAS_STATUS_SUCCESS)
                return fail(DFTB_ERR_CUDA, "trans_charges: cublasDgemm (S C) failed");
            continue;
        }
        GemmP p = gemm_defaults();
        p.M = norb;
        p.N = n;
        p.K = norb;
        p.A = Smat;
        p.sam = norb;
        p.sak = 1;
        p.B = b == 0 ? co : cv;
        p.sbk = n;
        p.sbn = 1;
        p.C = b == 0 ? *sco : *scv;
        p.scm = n;
        p.scn = 1;
        rc = launch_gemm(p, EPI_STORE, 1, st);
        if (rc) return rc;
    }
    return DFTB_OK;
}

// ----------------------------------------------------------------------------
// Davidson helpers
// ----------------------------------------------------------------------------
__global__ void precondition_kernel(int nov, int nnew, const double *W, int ldw, const int *src, const int *state,
                                    const double *w, const double *omega, double *Q, int ldq) {
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long long)nov * nnew) return;
    const int ia = (int)(idx / nnew), c = (int)(idx % nnew);
    const double om = omega[ia];
    double wd = w[state[c]] - om;
    if (fabs(wd) < 1.0e-6) wd = 1.0e-6 * om;
    Q[(size_t)ia * ldq + c] = W[(size_t)ia * ldw + src[c]] / wd;
}

__global__ void residual_kernel(int nov, int ncol, const double *AV, int ldav, const double *X, int ldx,
                                const double *lam, double *W, int ldw, double *nrm2) {
    const int c = blockIdx.y;
    double acc = 0.0;
    for (int ia = blockIdx.x * blockDim.x + threadIdx.x; ia < nov; ia += gridDim.x * blockDim.x) {
        const double r = AV[(size_t)ia * ldav + c] - lam[c] * X[(size_t)ia * ldx + c];
        W[(size_t)ia * ldw + c] = r;
        acc += r * r;
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, off);
    __shared__ double red[32];
    const int wi = threadIdx.x / 32, lane = threadIdx.x % 32;
    if (lane == 0) red[wi] = acc;
    __syncthreads();
    if (wi == 0) {
        acc = lane < (int)(blockDim.x / 32) ? red[lane] : 0.0;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, off);
        if (lane == 0) atomicAdd(&nrm2[c], acc);
    }
}

// Row-blocked form for ncol <= 256: a block of 256 threads covers R = 256 / ncol rows x all columns
// per step (consecutive threads read consecutive elements of a row), so each thread keeps one
// column and its squared norm in a register; the R partial sums of a column meet in shared memory.
__global__ void residual_rows_kernel(int nov, int ncol, const double *AV, int ldav, const double *X, int ldx,
                                     const double *lam, double *W, int ldw, double *nrm2) {
    __shared__ double red[256];
    const int R = blockDim.x / ncol;
    const int tc = threadIdx.x % ncol, tr = threadIdx.x / ncol;
    double acc = 0.0;
    if (tr < R) {
        const double l = lam[tc];
        for (long long ia = (long long)blockIdx.x * R + tr; ia < nov; ia += (long long)gridDim.x * R) {
            const double r = AV[ia * ldav + tc] - l * X[ia * ldx + tc];
            W[ia * ldw + tc] = r;
            acc += r * r;
        }
    }
    red[threadIdx.x] = acc;
    __syncthreads();
    if (threadIdx.x < ncol) {
        double sum = 0.0;
        for (int j = 0; j < R; ++j) sum += red[threadIdx.x + j * ncol];
        atomicAdd(&nrm2[threadIdx.x], sum);
    }
}

__global__ void sqrt_kernel(int n, double *x) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) x[i] = sqrt(x[i]);
}

// us = omega o vs (the first term of (A-B).v without Coulomb)
__global__ void omega_scale_kernel(long long nov, int nvec, const double *omega, const double *vs, double *us) {
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    grid_launch_dependents();  // the exchange products may start
    if (idx >= nov * nvec) return;
    us[idx] = omega[idx / nvec] * vs[idx];
}

// Coulomb part shared by the Hermitian and (A+B) products (cuBLAS handle: blas() above).
// us(ia, n) = omega_ia v(ia, n) + fac us(ia, n)   (in place; the non-Hermitian Coulomb epilogue)
__global__ void rv_inplace_kernel(long long total, int nvec, const double *omega, const double *vs, double *us,
                                  double fac) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    us[i] = omega[i / nvec] * vs[i] + fac * us[i];
}

template <int NT, bool HERM>
int launch_qv(const QvP &p, unsigned rows, unsigned ks, unsigned cols, cudaStream_t st) {
    static bool attr_set[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !attr_set[dev]) {
        if (cudaFuncSetAttribute(qv_kernel<NT, HERM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 Skinny<NT>::SMEM) != cudaSuccess)
            return fail(DFTB_ERR_CUDA, "coulomb: shared memory");
        if (dev >= 0 && dev < 64) attr_set[dev] = true;
    }
    if (p.after)
        launch_overlapped(qv_kernel<NT, HERM>, dim3(rows, ks, cols), QV_THREADS, Skinny<NT>::SMEM, st, p, true);
    else
        qv_kernel<NT, HERM><<<dim3(rows, ks, cols), QV_THREADS, Skinny<NT>::SMEM, st>>>(p);
    return check_launch("qv_kernel");
}

template <int NT>
int launch_qv(const QvP &p, unsigned rows, unsigned ks, unsigned cols, cudaStream_t st) {
    return p.omega ? launch_qv<NT, true>(p, rows, ks, cols, st) : launch_qv<NT, false>(p, rows, ks, cols, st);
}

// T = Q (s o V) for up to 32 columns at a time (T zeroed by the caller): the columns of Q are cut so that two
// CTAs per SM are in flight
int skinny_product(int M, int K, const double *Q, const double *V, int ncol, double *T, const double *omega,
                   cudaStream_t st, bool after = false) {
    const unsigned rows = cdiv(M, QV_M), cols = cdiv(ncol, 32);
    const long long want = 296 / ((long long)rows * cols);
    const long long chunks = cdiv(K, QV_K);
    // Up to four stages a range where there are ranges enough: each range adds all of T once more, to the same few elements
    // where Q has few rows.  B200, Hermitian product, us with one, two and four stages at least: 54 atoms x 6084 pairs, 10
    // columns 24.3, 18.5, 16.4, 32 columns 32.1, 25.4, 23.5; 90 x 12321, 10 columns 28.9 (three) and 23.1; but 14 x 256 12.3,
    // 12.3 and 14.4.
    const long long least = chunks < 48 ? 1 : (chunks < 96 ? chunks / 24 : 4);
    long long ks = want < 1 ? 1 : (want > chunks ? chunks : want);
    if (ks > chunks / least) ks = chunks / least;
    const long long per = (chunks + ks - 1) / ks;
    ks = (chunks + per - 1) / per;
    const QvP p{M, K, Q, V, ncol, ncol, T, ncol, omega, (int)(per * QV_K), after};
    switch (cols > 1 ? 4 : (int)cdiv(ncol, 8)) {
        case 1: return launch_qv<1>(p, rows, (unsigned)ks, cols, st);
        case 2: return launch_qv<2>(p, rows, (unsigned)ks, cols, st);
        case 3: return launch_qv<3>(p, rows, (unsigned)ks, cols, st);
        default: return launch_qv<4>(p, rows, (unsigned)ks, cols, st);
    }
}

//   T = q_ov . (s o V)   (atomic over the column ranges), G = gamma . T,  us = epilogue(q_ov^T G)
// The Hermitian form takes as many blocks of 32 columns as it needs.  The non-Hermitian form (s = 1) runs its two large
// GEMMs in cuBLAS, when it is available, where that is faster: row-major X (r x c) is the column-major X^T, so
// T^T = V^T q_ov^T and us^T = G^T q_ov.  B200, us here and in cuBLAS:
//   - more than 32 columns, where q_ov would be read a third and fourth time: 1104 atoms x 1225 x 1225, 60 columns 17000 and
//     12600;
//   - 25 to 32 columns, bound by the FP64 pipe, for many pairs: 1104 x 109k 661 and 690, 336 x 40k 116 and 147, but
//     600 x 160k 570 and 542, 336 x 371k 765 and 655, 1104 x 1.5M 9050 and 7800 (24 columns: 589 and 650, 7470 and 7700);
//   - one column of a long odd number of pairs, where every other row is off the 16-byte grid: 336 x 371k 346 and 374, but
//     1104 x 642k 2005 and 1953, 700 x 1.5M 3430 and 2650 (even, 1104 x 1.0M: 2840 and 3010; two columns: 5000 and 7560).
bool coulomb_in_blas(int nov, int nvec) {
    return nvec > 32 || (nvec > 24 && nov > 120000) || (nvec == 1 && nov % 2 == 1 && nov > 500000);
}
// Atoms up to which the cuBLAS route forms gamma . T in one plain product: two launches less count for more there than
// splitting the sum (14 atoms, 33 columns: 26 -> 23 us a call).
constexpr int COULOMB_PLAIN = 48;
// Kernels overlap at their seams up to this size of q_ov.  B200, 10 columns, overlapped and in turn: 0.1 MB 14.2 and 16.4 us,
// 0.9 MB 20.5 and 24.6, 6.7 MB 27.6 and 29.7, 22 MB 38.1 and 37.9, 66 MB 52.0 and 51.8; beyond, the waiting CTAs of the last
// kernel cost the first one more than the seams (997 MB, 30 columns: 841 and 799 us).
constexpr long long OVERLAP_BYTES = 16 << 20;
int coulomb_product(int nat, int nov, int nvec, const double *gamma, const double *q_ov, const double *omega,
                    const double *vs, double *us, double *T, double *G, int hermitian, cudaStream_t st) {
    int rc;
    cublasHandle_t bh = hermitian || !coulomb_in_blas(nov, nvec) ? nullptr : blas_handle(st);
    const bool plain = bh && nat <= COULOMB_PLAIN;
    if (!plain) {
        // T and G are adjacent in the workspace: one memset zeroes both
        const size_t bytes = (size_t)((char *)G - (char *)T) + sizeof(double) * (size_t)nat * nvec;
        if (cudaMemsetAsync(T, 0, bytes, st) != cudaSuccess) return fail(DFTB_ERR_CUDA, "memset T");
    }
    if (bh) {
        const double one = 1.0, zero = 0.0;
        if (blas().dgemm(bh, CUBLAS_OP_N, CUBLAS_OP_N, nvec, nat, nov, &one, vs, nvec, q_ov, nov, &zero, T, nvec) !=
            CUBLAS_STATUS_SUCCESS)
            return fail(DFTB_ERR_CUDA, "coulomb: cublasDgemm (q_ov V) failed");
        if (plain) {
            GemmP p = gemm_defaults();
            p.M = nat;
            p.N = nvec;
            p.K = nat;
            p.A = gamma;
            p.sam = nat;
            p.sak = 1;
            p.B = T;
            p.sbk = nvec;
            p.sbn = 1;
            p.C = G;
            p.scm = nvec;
            p.scn = 1;
            rc = launch_gemm(p, EPI_STORE, 1, st);
        } else {
            rc = skinny_product(nat, nat, gamma, T, nvec, G, nullptr, st);
        }
        if (rc) return rc;
        if (blas().dgemm(bh, CUBLAS_OP_N, CUBLAS_OP_T, nvec, nov, nat, &one, G, nvec, q_ov, nov, &zero, us, nvec) !=
            CUBLAS_STATUS_SUCCESS)
            return fail(DFTB_ERR_CUDA, "coulomb: cublasDgemm (q_ov^T G) failed");
        const long long total = (long long)nov * nvec;
        rv_inplace_kernel<<<(unsigned)((total + 255) / 256), 256, 0, st>>>(total, nvec, omega, vs, us, 4.0);
        return check_launch("rv_inplace_kernel");
    }
    const bool overlap = 8LL * nat * nov <= OVERLAP_BYTES;
    if ((rc = skinny_product(nat, nov, q_ov, vs, nvec, T, hermitian ? omega : nullptr, st))) return rc;
    if ((rc = skinny_product(nat, nat, gamma, T, nvec, G, nullptr, st, overlap))) return rc;
    const QgP p{nov, nat, q_ov, G, nvec, nvec, omega, vs, us, 4.0, hermitian};
    const unsigned cols = cdiv(nvec, 32);
    const dim3 grid(cdiv(nov, QG_THREADS), cols);
    switch (cols > 1 ? 4 : (int)cdiv(nvec, 8)) {
        case 1: launch_overlapped(qg_kernel<1>, grid, QG_THREADS, 0, st, p, overlap); break;
        case 2: launch_overlapped(qg_kernel<2>, grid, QG_THREADS, 0, st, p, overlap); break;
        case 3: launch_overlapped(qg_kernel<3>, grid, QG_THREADS, 0, st, p, overlap); break;
        default: launch_overlapped(qg_kernel<4>, grid, QG_THREADS, 0, st, p, overlap); break;
    }
    return check_launch("qg_kernel");
}

// Exchange terms in the transition-charge form, accumulated into us:
//   us += sK1 * K1 v + sK2 * K2 v
//   K1 v(i; a,c) = sum_{B,j} Z[B](i,j) Y[B][j](a,c),  Z[B](i,j) = sum_A g_lr[A][B] q_oo[A](i,j),
//                                                     Y[B][j](a,c) = sum_b q_vv[B](a,b) v(j,b,c)
//   K2 v(i; a,c) = sum_{B,b} Z2[B](i,b) W[B][b](a,c),  Z2[B](i,b) = sum_A g_lr[A][B] q_ov[A](i,b),
//                                                      W[B][b](a,c) = sum_j q_ov[B](j,a) v(j,b,c)
// Y and W are batched products per atom, laid out so that the sum over atoms and one orbital index is then a single
// product of that length with whole (orbital, vector) rows (a product per atom and vector, added into us with atomics,
// ran at 7 TFLOP/s).  B200, C40H42 (82 atoms, 101 x 101 orbitals), 10 vectors, (A+B).V and (A-B).V: 1820 -> 840 us.
//
// Small molecules are bound by launches and by the latency of a chain of short products: for them Z, Y, Z2 and W, which do
// not depend on one another, are one launch, and the two sums another; the first runs beside the Coulomb product's last
// kernel.  (A+B).V on B200, us with six launches and with two: C6H8 (14 atoms, 16 x 16 orbitals), 1 vector 37 and 16 (a
// product per atom and vector: 25), C10H12 46 and 22 (40), C20H22, 10 vectors 78 and 55 (125).  Up to this much scratch for
// both terms: C44H46, 1 vector, 35 MB, 126 and 120 us; C30H32, 10 vectors, 63 MB, 199 and 228.
constexpr size_t EXCHANGE_GROUPED_BYTES = (size_t)36 << 20;

// scratch elements of the two terms
void exchange_scratch(int nat, int nocc, int nvirt, int nvec, size_t *k1, size_t *k2) {
    const size_t no = nocc, nv = nvirt, m = nvec, na = nat;
    *k1 = na * no * no + na * no * nv * m;
    *k2 = na * no * nv + na * nv * nv * m;
}

int exchange_products(int nat, int nocc, int nvirt, int nvec, const double *g_lr, const double *q_oo,
                      const double *q_ov, const double *q_vv, const double *vs, double *us, double sK1, double sK2,
                      double *work, size_t work_bytes, cudaStream_t st) {
    const long long no = nocc, nv = nvirt, m = nvec;
    size_t k1, k2;
    exchange_scratch(nat, nocc, nvirt, nvec, &k1, &k2);
    const size_t both = sizeof(double) * (k1 + k2);
    const bool grouped = both <= EXCHANGE_GROUPED_BYTES && work_bytes >= both;
    double *Z = work, *Y = Z + nat * no * no, *Z2 = grouped ? work + k1 : work, *W = Z2 + nat * no * nv;
    GemmP q[4], k[2];  // Z, Y, Z2, W; K1 v, K2 v
    for (int t = 0; t < 4; t += 2) {  // (A, orbital pairs) from the charges of all atoms
        GemmP &p = q[t] = gemm_defaults();
        const long long pairs = no * (t ? nv : no);
        p.M = nat;
        p.N = (int)pairs;
        p.K = nat;
        p.A = g_lr;
        p.sam = 1;
        p.sak = nat;
        p.B = t ? q_ov : q_oo;
        p.sbk = pairs;
        p.sbn = 1;
        p.C = t ? Z2 : Z;
        p.scm = pairs;
        p.scn = 1;
    }
    {
        GemmP &p = q[1] = gemm_defaults();
        p.M = (int)nv;        // a
        p.N = (int)(no * m);  // (j, c)
        p.N2 = (int)m;
        p.K = (int)nv;  // b
        p.A = q_vv;
        p.sam = nv;
        p.sak = 1;
        p.sa1 = nv * nv;
        p.B = vs;
        p.sbk = m;
        p.sbn1 = nv * m;
        p.sbn = 1;
        p.C = Y;
        p.scm = m;
        p.scn1 = nv * m;
        p.scn = 1;
        p.sc1 = no * nv * m;
    }
    {
        GemmP &p = q[3] = gemm_defaults();
        p.M = (int)nv;        // a
        p.N = (int)(nv * m);  // (b, c)
        p.N2 = (int)m;
        p.K = (int)no;  // j
        p.A = q_ov;
        p.sam = 1;
        p.sak = nv;
        p.sa1 = no * nv;
        p.B = vs;
        p.sbk = nv * m;
        p.sbn1 = m;
        p.sbn = 1;
        p.C = W;
        p.scm = m;
        p.scn1 = nv * m;
        p.scn = 1;
        p.sc1 = nv * nv * m;
    }
    for (int t = 0; t < 2; ++t) {
        GemmP &p = k[t] = gemm_defaults();
        const long long n = t ? nv : no;  // the orbital of the sum
        p.M = (int)no;                    // i
        p.N = (int)(nv * m);              // (a, c)
        p.K = (int)(nat * n);
        p.K2 = (int)n;
        p.A = t ? Z2 : Z;
        p.sam = n;
        p.sak1 = no * n;
        p.sak = 1;
        p.B = t ? W : Y;
        p.sbk = nv * m;
        p.sbn = 1;
        p.C = us;
        p.scm = nv * m;
        p.scn = 1;
        p.alpha = t ? sK2 : sK1;
        // Two CTAs per SM: C40H42's 32 tiles of K = 8282 take 76 us, with four 80; C20H22's five of K = 2142 9 us in ranges of
        // four stages, 21 of sixteen.  Side by side the terms share them, and shorter ranges pay: C6H8's one tile of K = 224
        // 19 us a call with four stages, 16 with two.
        p.ksplit = grouped ? pick_ksplit(p.M, p.N, p.K, 148, 2) : pick_ksplit(p.M, p.N, p.K, 296, 4);
    }
    const int batch[4] = {1, nat, 1, nat};
    int rc;
    if (grouped) {
        if ((rc = launch_gemm_group<EPI_STORE, false>(q, batch, 4, st))) return rc;
        const int one[2] = {1, 1};
        return launch_gemm_group<EPI_ATOMIC, true>(k, one, 2, st);
    }
    for (int t = 0; t < 2; ++t) {  // one term after the other in the same scratch
        for (int h = 2 * t; h < 2 * t + 2; ++h)
            if ((rc = launch_gemm(q[h], EPI_STORE, batch[h], st))) return rc;
        if ((rc = launch_gemm(k[t], EPI_ATOMIC, 1, st))) return rc;
    }
    return DFTB_OK;
}

int check_products(int nat, int nocc, int nvirt, int nvec, int lc, const double *g, const double *g_lr,
                   const double *q_oo, const double *q_ov, const double *q_vv, const double *omega, const double *vs,
                   double *us, void *work, size_t work_bytes) {
    if (nat <= 0 || nocc <= 0 || nvirt <= 0 || nvec <= 0) return fail(DFTB_ERR_BAD_SIZE, "apbv: sizes");
    if (!g || !q_ov || !omega || !vs || !us) return fail(DFTB_ERR_NULL, "apbv: null");
    if (lc && (!g_lr || !q_oo || !q_vv)) return fail(DFTB_ERR_NULL, "apbv: lc needs g_lr, q_oo, q_vv");
    size_t need = dftb_hermitian_rv_workspace_size(nat, nvec);
    if (lc) {  // one exchange term at a time; dftb_apbv_workspace_size may ask for more, to run both side by side
        size_t k1, k2;
        exchange_scratch(nat, nocc, nvirt, nvec, &k1, &k2);
        need += align256(sizeof(double) * (k1 > k2 ? k1 : k2));
    }
    if (!work || work_bytes < need) return fail(DFTB_ERR_WORKSPACE, "apbv: workspace too small");
    return DFTB_OK;
}

// ---------------------------------------------------------------------------- layout changes of column blocks

// Y (cols x rows) = X^T through a 32 x 32 shared-memory tile: reads and writes run along rows of 256 bytes
// (a strided element copy moves a whole 32-byte sector per 8-byte element on one side)
__global__ void __launch_bounds__(256) transpose_f64_kernel(int rows, int cols, const double *__restrict__ X,
                                                            long long ldx, double *__restrict__ Y, long long ldy) {
    __shared__ double t[32][33];
    const int r0 = blockIdx.x * 32, c0 = blockIdx.y * 32;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    for (int k = ty; k < 32; k += 8) {
        const int r = r0 + k, c = c0 + tx;
        if (r < rows && c < cols) t[k][tx] = X[(long long)r * ldx + c];
    }
    __syncthreads();
    for (int k = ty; k < 32; k += 8) {
        const int c = c0 + k, r = r0 + tx;
        if (c < cols && r < rows) Y[(long long)c * ldy + r] = t[tx][k];
    }
}

// K_y[(i nvirt + a) m + c] = Kall[c][2a + y][i] (FP32 -> FP64): the exchange's last launch writes, for each
// product column c, K1^T and K2^T with their rows interleaved.  A CTA takes one a and a run of 32 i for
// every c: it reads 128-byte pieces of Kall rows and writes whole m-long rows of K1 and K2.
__global__ void __launch_bounds__(256) exchange_unpack_kernel(int m, int nv, int no, const float *__restrict__ Kall,
                                                              double *__restrict__ K1, double *__restrict__ K2) {
    __shared__ float t[2][64][33];
    const int a = blockIdx.y, i0 = blockIdx.x * 32;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int c0 = 0; c0 < m; c0 += 64) {
        const int mc = min(64, m - c0);
        for (int row = wid; row < 2 * mc; row += 8) {
            const int c = row >> 1, y = row & 1, i = i0 + lane;
            t[y][c][lane] = i < no ? Kall[((long long)(c0 + c) * 2 * nv + 2 * a + y) * no + i] : 0.0f;
        }
        __syncthreads();
        for (int row = wid; row < 64; row += 8) {
            const int il = row >> 1, y = row & 1, i = i0 + il;
            if (i < no) {
                double *dst = (y ? K2 : K1) + ((long long)i * nv + a) * m + c0;
                for (int c = lane; c < mc; c += 32) dst[c] = (double)t[y][c][il];
            }
        }
        __syncthreads();
    }
}

// (A+B) v = (u - K1) - K2 and (A-B) v = (omega v + K2) - K1 from the same Kall (FP32 or FP64), u = Coulomb products, in
// place of one pass that unpacks K1 and K2 and five element-wise ones; each operand moves once, at 3.1 to 3.5 TB/s, half the
// rate of a copy: the warps wait for the transposed tile in shared memory (two thirds of their stalls) and for its index
// divisions.  A block takes 32 i and as many a as make 64 of the contiguous (a, c); rounded as the separate passes were.  B200, 1225 x 1225: 700 us -> 315 us
// (FP32, 16 columns, 0.96 GB), 253 -> 91 us (FP64, 4 columns, 0.29 GB).  Four elements a thread in flight made it 450 us.
template <typename T>
__global__ void __launch_bounds__(256) exchange_combine_kernel(int m, int nv, int no, const T *__restrict__ Kall,
                                                               const double *__restrict__ omega,
                                                               const double *__restrict__ V, double *U,
                                                               double *__restrict__ W) {
    __shared__ T t[2][64][33];
    const int na_max = max(1, 64 / m), a0 = blockIdx.y * na_max, na = min(na_max, nv - a0), i0 = blockIdx.x * 32;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, i = i0 + lane;
    for (int c0 = 0; c0 < m; c0 += 64) {  // one round unless m > 64, where na = 1
        const int mc = min(64, m - c0), run = na * mc;
        for (int row = wid; row < 2 * run; row += 8) {
            const int c = row / (2 * na), ay = row % (2 * na);
            t[ay & 1][(ay >> 1) * mc + c][lane] =
                i < no ? Kall[((long long)(c0 + c) * 2 * nv + 2 * a0 + ay) * no + i] : (T)0;
        }
        __syncthreads();
        for (int e = threadIdx.x; e < 32 * run; e += 256) {
            const int il = e / run, k = e % run;
            if (i0 + il >= no) break;
            const long long ia = (long long)(i0 + il) * nv + a0, o = ia * m + c0 + k;
            const double k1 = t[0][k][il], k2 = t[1][k][il], w = omega[ia + k / mc];
            U[o] = __dadd_rn(__dadd_rn(U[o], -k1), -k2);
            W[o] = __dadd_rn(__dadd_rn(__dmul_rn(w, V[o]), k2), -k1);
        }
        __syncthreads();
    }
}

}  // namespace

// ============================================================================
// extern "C" entry points
// ============================================================================
extern "C" {

const char *dftb_version(void) { return "dftbaby_b200 0.1 (sm_100a, fp64)"; }
const char *dftb_last_error(void) { return g_last_error; }

int dftb_directional_cosines(int nat, const double *pos, double *r, double *x, double *y, double *z, void *stream) {
    if (nat <= 0) return fail(DFTB_ERR_BAD_SIZE, "directional_cosines: nat");
    if (!pos || !r || !x || !y || !z) return fail(DFTB_ERR_NULL, "directional_cosines: null");
    dim3 grid(cdiv(nat, 128), nat);
    dircos_kernel<<<grid, 128, 0, S(stream)>>>(nat, pos, r, x, y, z);
    return check_launch("dircos_kernel");
}

int dftb_h0_and_s(int norb, int nat, const int *ind, const int *typ, const int *ls, const int *ms, const double *r,
                  const double *x, const double *y, const double *z, const int *mprox, const double *orben, int deg,
                  const int *tab_filled, const double *S_knots, const double *S_coefs, const double *H_knots,
                  const double *H_coefs, int npair, int nsk, int npts, double *Sm, double *H0, void *stream) {
    if (norb <= 0 || nat <= 0 || npair <= 0 || nsk <= 0 || npts < 8) return fail(DFTB_ERR_BAD_SIZE, "h0_and_s: sizes");
    if (deg != 3) return fail(DFTB_ERR_UNSUPPORTED, "h0_and_s: only cubic splines");
    if (!ind || !typ || !ls || !ms || !r || !x || !y || !z || !mprox || !orben || !tab_filled || !S_knots ||
        !S_coefs || !H_knots || !H_coefs || !Sm || !H0)
        return fail(DFTB_ERR_NULL, "h0_and_s: null");
    OrbTables O{ind, typ, ls, ms};
    SkTables TS{tab_filled, S_knots, S_coefs, nsk, npts};
    SkTables TH{tab_filled, H_knots, H_coefs, nsk, npts};
    dim3 grid(cdiv(nat, SK_TB), cdiv(nat, SK_TA));
    if (grid.y > 65535u) return fail(DFTB_ERR_BAD_SIZE, "h0_and_s: more than 524280 atoms");
    h0_and_s_kernel<<<grid, SK_PAIRS, 0, S(stream)>>>(norb, nat, O, r, x, y, z, mprox, orben, TS, TH, Sm, H0);
    return check_launch("h0_and_s_kernel");
}

int dftb_dipole_matrix(int norb, int nat, const int *ind, const int *typ, const int *ls, const int *ms,
                       const double *r, const double *x, const double *y, const double *z, const double *pos,
                       const int *mprox, const double *Sm, int deg, const int *tab_filled_D, const double *D_knots,
                       const double *D_coefs, int npair, int nskd, int npts, double *D, void *stream) {
    if (norb <= 0 || nat <= 0 || npair <= 0 || nskd <= 0 || npts < 8)
        return fail(DFTB_ERR_BAD_SIZE, "dipole_matrix: sizes");
    if (deg != 3) return fail(DFTB_ERR_UNSUPPORTED, "dipole_matrix: only cubic splines");
    if (!ind || !typ || !ls || !ms || !r || !x || !y || !z || !pos || !mprox || !Sm || !tab_filled_D ||
        !D_knots || !D_coefs || !D)
        return fail(DFTB_ERR_NULL, "dipole_matrix: null");
    OrbTables O{ind, typ, ls, ms};
    SkTables TD{tab_filled_D, D_knots, D_coefs, nskd, npts};
    dim3 grid(cdiv(nat, SK_TB), cdiv(nat, SK_TA));
    if (grid.y > 65535u) return fail(DFTB_ERR_BAD_SIZE, "dipole_matrix: more than 524280 atoms");
    dipole_kernel<<<grid, SK_PAIRS, 0, S(stream)>>>(norb, nat, O, r, x, y, z, pos, mprox, Sm, TD, D);
    return check_launch("dipole_kernel");
}

int dftb_gamma_matrices(int nat, const double *r, const double *sigma, double r_lr, double *gamma, double *gamma_lr,
                        void *stream) {
    if (nat <= 0) return fail(DFTB_ERR_BAD_SIZE, "gamma: nat");
    if (!r || !sigma || !gamma) return fail(DFTB_ERR_NULL, "gamma: null");
    dim3 grid(cdiv(nat, 128), nat);
    gamma_kernel<<<grid, 128, 0, S(stream)>>>(nat, r, sigma, r_lr, gamma, gamma_lr);
    return check_launch("gamma_kernel");
}

int dftb_ao_expand(int norb, int nat, const int *ind, const double *g, double *G, void *stream) {
    if (norb <= 0 || nat <= 0) return fail(DFTB_ERR_BAD_SIZE, "ao_expand: sizes");
    if (!ind || !g || !G) return fail(DFTB_ERR_NULL, "ao_expand: null");
    dim3 grid(cdiv(norb, 128), cdiv(norb, AO_ROWS));
    ao_expand_kernel<<<grid, 128, 0, S(stream)>>>(norb, nat, ind, g, G);
    return check_launch("ao_expand_kernel");
}

int dftb_scc_hamiltonian(int norb, int nat, const int *ind, const double *H0, const double *Sm, const double *gamma,
                         const double *dq, double *estat, double *H, void *stream) {
    if (norb <= 0 || nat <= 0) return fail(DFTB_ERR_BAD_SIZE, "scc_hamiltonian: sizes");
    if (!ind || !H0 || !Sm || !gamma || !dq || !estat || !H) return fail(DFTB_ERR_NULL, "scc_hamiltonian: null");
    estat_kernel<<<cdiv(nat, 8), 256, 0, S(stream)>>>(nat, gamma, dq, estat);
    int rc = check_launch("estat_kernel");
    if (rc) return rc;
    dim3 grid(cdiv(norb, 128), cdiv(norb, AO_ROWS));
    scc_h_kernel<<<grid, 128, 0, S(stream)>>>(norb, ind, H0, Sm, estat, H);
    return check_launch("scc_h_kernel");
}

int dftb_monopoles(int norb, int nat, const double *P, const double *P0, const double *Sm, const int *opa, double *q,
                   double *dq, void *stream) {
    if (norb <= 0 || nat <= 0) return fail(DFTB_ERR_BAD_SIZE, "monopoles: sizes");
    if (!P || !P0 || !Sm || !opa || !q || !dq) return fail(DFTB_ERR_NULL, "monopoles: null");
    monopoles_kernel<<<nat, 256, 0, S(stream)>>>(norb, nat, P, P0, Sm, opa, q, dq);
    return check_launch("monopoles_kernel");
}

size_t dftb_trans_charges_workspace_size(int norb, int nocc, int nvirt) {
    if (norb <= 0 || nocc < 0 || nvirt < 0) return 0;
    return align256(sizeof(double) * (size_t)norb * nocc) + align256(sizeof(double) * (size_t)norb * nvirt) +
           align256(sizeof(int) * ((size_t)norb + 1));
}

int dftb_trans_charges(int norb, int nat, int nocc, int nvirt, const double *co, const double *cv, const double *Sm,
                       const int *opa, double *q_oo, double *q_ov, double *q_vv, void *work, size_t work_bytes,
                       void *stream) {
    cudaStream_t st = S(stream);
    double *sco, *scv;
    int *first;
    if (nat > norb) return fail(DFTB_ERR_BAD_SIZE, "trans_charges: nat > norb");
    if (nat > 65535) return fail(DFTB_ERR_BAD_SIZE, "trans_charges: nat > 65535");
    int rc = trans_charges_common(norb, nat, nocc, nvirt, co, cv, Sm, opa, work, work_bytes, st, &sco, &scv, &first);
    if (rc) return rc;
    struct Blk {
        double *out;
        const double *c1, *s1, *c2, *s2;
        int n1, n2;
    } blks[3] = {{q_oo, co, sco, co, sco, nocc, nocc},
                 {q_ov, co, sco, cv, scv, nocc, nvirt},
                 {q_vv, cv, scv, cv, scv, nvirt, nvirt}};
    for (auto &b : blks) {
        if (!b.out || b.n1 == 0 || b.n2 == 0) continue;
        if ((rc = launch_tc(nat, b.n1, b.n2, first, b.c1, b.s1, b.c2, b.s2, b.out, st, "tc_kernel")))
            return rc;
    }
    return DFTB_OK;
}

int dftb_trans_charges_diag(int norb, int nat, int nocc, int nvirt, const double *co, const double *cv,
                            const double *Sm, const int *opa, double *q_ii, double *q_aa, void *work,
                            size_t work_bytes, void *stream) {
    cudaStream_t st = S(stream);
    double *sco, *scv;
    int *first;
    if (nat > norb) return fail(DFTB_ERR_BAD_SIZE, "trans_charges_diag: nat > norb");
    int rc = trans_charges_common(norb, nat, nocc, nvirt, co, cv, Sm, opa, work, work_bytes, st, &sco, &scv, &first);
    if (rc) return rc;
    if (q_ii && nocc > 0) {
        tc_diag_kernel<<<dim3(cdiv(nocc, 128), nat), 128, 0, st>>>(nocc, first, co, sco, q_ii);
        if ((rc = check_launch("tc_diag_kernel"))) return rc;
    }
    if (q_aa && nvirt > 0) {
        tc_diag_kernel<<<dim3(cdiv(nvirt, 128), nat), 128, 0, st>>>(nvirt, first, cv, scv, q_aa);
        if ((rc = check_launch("tc_diag_kernel"))) return rc;
    }
    return DFTB_OK;
}

size_t dftb_hermitian_rv_workspace_size(int nat, int nvec) {
    if (nat <= 0 || nvec <= 0) return 0;
    return 2 * align256(sizeof(double) * (size_t)nat * nvec);
}

int dftb_hermitian_rv(int nat, int nocc, int nvirt, int nvec, const double *gamma, const double *q_ov,
                      const double *omega, const double *vs, double *us, void *work, size_t work_bytes,
                      void *stream) {
    if (nat <= 0 || nocc <= 0 || nvirt <= 0 || nvec <= 0) return fail(DFTB_ERR_BAD_SIZE, "hermitian_rv: sizes");
    if (!gamma || !q_ov || !omega || !vs || !us) return fail(DFTB_ERR_NULL, "hermitian_rv: null");
    if (!work || work_bytes < dftb_hermitian_rv_workspace_size(nat, nvec))
        return fail(DFTB_ERR_WORKSPACE, "hermitian_rv: workspace too small");
    double *T = (double *)work;
    double *G = (double *)((char *)work + align256(sizeof(double) * (size_t)nat * nvec));
    return coulomb_product(nat, nocc * nvirt, nvec, gamma, q_ov, omega, vs, us, T, G, 1, S(stream));
}

size_t dftb_apbv_workspace_size(int nat, int nocc, int nvirt, int nvec) {
    if (nat <= 0 || nocc <= 0 || nvirt <= 0 || nvec <= 0) return 0;
    size_t k1, k2;
    exchange_scratch(nat, nocc, nvirt, nvec, &k1, &k2);
    const size_t serial = sizeof(double) * (k1 > k2 ? k1 : k2), both = sizeof(double) * (k1 + k2);
    // never less for more atoms, orbitals or vectors, so that the size of the largest call serves the smaller ones
    const size_t grouped = both < EXCHANGE_GROUPED_BYTES ? both : EXCHANGE_GROUPED_BYTES;
    return align256(serial > grouped ? serial : grouped) + dftb_hermitian_rv_workspace_size(nat, nvec);
}

int dftb_apbv(int nat, int nocc, int nvirt, int nvec, int lc, const double *g, const double *g_lr,
              const double *q_oo, const double *q_ov, const double *q_vv, const double *omega, const double *vs,
              double *us, void *work, size_t work_bytes, void *stream) {
    int rc = check_products(nat, nocc, nvirt, nvec, lc, g, g_lr, q_oo, q_ov, q_vv, omega, vs, us, work, work_bytes);
    if (rc) return rc;
    cudaStream_t st = S(stream);
    // workspace: [T | G] for the Coulomb term, then the exchange scratch
    const size_t coul = dftb_hermitian_rv_workspace_size(nat, nvec);
    double *T = (double *)work;
    double *G = (double *)((char *)work + align256(sizeof(double) * (size_t)nat * nvec));
    rc = coulomb_product(nat, nocc * nvirt, nvec, g, q_ov, omega, vs, us, T, G, 0, st);
    if (rc || !lc) return rc;
    return exchange_products(nat, nocc, nvirt, nvec, g_lr, q_oo, q_ov, q_vv, vs, us, -1.0, -1.0,
                             (double *)((char *)work + coul), work_bytes - coul, st);
}

int dftb_ambv(int nat, int nocc, int nvirt, int nvec, int lc, const double *g, const double *g_lr,
              const double *q_oo, const double *q_ov, const double *q_vv, const double *omega, const double *vs,
              double *us, void *work, size_t work_bytes, void *stream) {
    int rc = check_products(nat, nocc, nvirt, nvec, lc, g, g_lr, q_oo, q_ov, q_vv, omega, vs, us, work, work_bytes);
    if (rc) return rc;
    cudaStream_t st = S(stream);
    const long long n = (long long)nocc * nvirt * nvec;
    omega_scale_kernel<<<cdiv(n, 256), 256, 0, st>>>((long long)nocc * nvirt, nvec, omega, vs, us);
    if ((rc = check_launch("omega_scale_kernel"))) return rc;
    if (!lc) return DFTB_OK;
    const size_t coul = dftb_hermitian_rv_workspace_size(nat, nvec);
    return exchange_products(nat, nocc, nvirt, nvec, g_lr, q_oo, q_ov, q_vv, vs, us, -1.0, +1.0,
                             (double *)((char *)work + coul), work_bytes - coul, st);
}

int dftb_davidson_precondition(int nov, int nnew, const double *W, int ldw, const int *src, const int *state,
                               const double *w, const double *omega, double *Q, int ldq, void *stream) {
    if (nov <= 0 || nnew < 0 || ldw <= 0 || ldq < nnew) return fail(DFTB_ERR_BAD_SIZE, "precondition: sizes");
    if (nnew == 0) return DFTB_OK;
    if (!W || !src || !state || !w || !omega || !Q) return fail(DFTB_ERR_NULL, "precondition: null");
    const long long n = (long long)nov * nnew;
    precondition_kernel<<<cdiv(n, 256), 256, 0, S(stream)>>>(nov, nnew, W, ldw, src, state, w, omega, Q, ldq);
    return check_launch("precondition_kernel");
}

int dftb_davidson_residual(int nov, int ncol, const double *AV, int ldav, const double *X, int ldx, const double *lam,
                           double *W, int ldw, double *norms, void *stream) {
    if (nov <= 0 || ncol <= 0 || ldav < ncol || ldx < ncol || ldw < ncol)
        return fail(DFTB_ERR_BAD_SIZE, "residual: sizes");
    if (!AV || !X || !lam || !W || !norms) return fail(DFTB_ERR_NULL, "residual: null");
    cudaStream_t st = S(stream);
    if (cudaMemsetAsync(norms, 0, sizeof(double) * ncol, st) != cudaSuccess)
        return fail(DFTB_ERR_CUDA, "residual: memset");
    int rc;
    if (ncol <= 256) {
        const int R = 256 / ncol;
        unsigned gx = cdiv(nov, R);
        if (gx > 148 * 8) gx = 148 * 8;
        residual_rows_kernel<<<gx, 256, 0, st>>>(nov, ncol, AV, ldav, X, ldx, lam, W, ldw, norms);
        rc = check_launch("residual_rows_kernel");
    } else {
        unsigned gx = cdiv(nov, 256);
        if (gx > 592) gx = 592;
        residual_kernel<<<dim3(gx, ncol), 256, 0, st>>>(nov, ncol, AV, ldav, X, ldx, lam, W, ldw, norms);
        rc = check_launch("residual_kernel");
    }
    if (rc) return rc;
    sqrt_kernel<<<cdiv(ncol, 128), 128, 0, st>>>(ncol, norms);
    return check_launch("sqrt_kernel");
}

int dftb_transpose_f64(int rows, int cols, const double *X, int ldx, double *Y, int ldy, void *stream) {
    if (rows < 0 || cols < 0 || ldx < cols || ldy < rows) return fail(DFTB_ERR_BAD_SIZE, "transpose_f64: sizes");
    if (rows == 0 || cols == 0) return DFTB_OK;
    if (!X || !Y) return fail(DFTB_ERR_NULL, "transpose_f64: null");
    if (cdiv(cols, 32) > 65535) return fail(DFTB_ERR_BAD_SIZE, "transpose_f64: more than 2097120 columns");
    transpose_f64_kernel<<<dim3(cdiv(rows, 32), cdiv(cols, 32)), 256, 0, S(stream)>>>(rows, cols, X, ldx, Y, ldy);
    return check_launch("transpose_f64_kernel");
}

int dftb_exchange_unpack(int m, int nvirt, int nocc, const float *Kall, double *K1, double *K2, void *stream) {
    if (m < 0 || nvirt < 0 || nocc < 0) return fail(DFTB_ERR_BAD_SIZE, "exchange_unpack: sizes");
    if (m == 0 || nvirt == 0 || nocc == 0) return DFTB_OK;
    if (!Kall || !K1 || !K2) return fail(DFTB_ERR_NULL, "exchange_unpack: null");
    if (nvirt > 65535) return fail(DFTB_ERR_BAD_SIZE, "exchange_unpack: more than 65535 virtual orbitals");
    exchange_unpack_kernel<<<dim3(cdiv(nocc, 32), nvirt), 256, 0, S(stream)>>>(m, nvirt, nocc, Kall, K1, K2);
    return check_launch("exchange_unpack_kernel");
}

int dftb_exchange_combine(int m, int nvirt, int nocc, int fp64, const void *Kall, const double *omega, const double *V,
                          double *U, double *W, void *stream) {
    if (m < 0 || nvirt < 0 || nocc < 0) return fail(DFTB_ERR_BAD_SIZE, "exchange_combine: sizes");
    if (m == 0 || nvirt == 0 || nocc == 0) return DFTB_OK;
    if (!Kall || !omega || !V || !U || !W) return fail(DFTB_ERR_NULL, "exchange_combine: null");
    const dim3 grid(cdiv(nocc, 32), cdiv(nvirt, m < 64 ? 64 / m : 1));
    if (grid.y > 65535u) return fail(DFTB_ERR_BAD_SIZE, "exchange_combine: too many virtual orbitals");
    if (fp64)
        exchange_combine_kernel<<<grid, 256, 0, S(stream)>>>(m, nvirt, nocc, (const double *)Kall, omega, V, U, W);
    else
        exchange_combine_kernel<<<grid, 256, 0, S(stream)>>>(m, nvirt, nocc, (const float *)Kall, omega, V, U, W);
    return check_launch("exchange_combine_kernel");
}

int dftb_dgemm(int transa, int transb, int m, int n, int k, double alpha, const double *A, int lda, const double *B,
               int ldb, double beta, double *C, int ldc, void *stream) {
    if (m < 0 || n < 0 || k < 0) return fail(DFTB_ERR_BAD_SIZE, "dgemm: sizes");
    if (m == 0 || n == 0) return DFTB_OK;
    if (!A || !B || !C) return fail(DFTB_ERR_NULL, "dgemm: null");
    GemmP p = gemm_defaults();
    p.M = m;
    p.N = n;
    p.K = k;
    p.A = A;
    p.sam = transa ? 1 : lda;
    p.sak = transa ? lda : 1;
    p.B = B;
    p.sbk = transb ? 1 : ldb;
    p.sbn = transb ? ldb : 1;
    p.C = C;
    p.scm = ldc;
    p.scn = 1;
    p.alpha = alpha;
    p.beta = beta;
    return launch_gemm(p, EPI_STORE, 1, S(stream));
}

}  // extern "C"

// ============================================================================
// Allocation-free variant of dftb_trans_charges.
//
// Some callers cannot allocate device memory at the point where they need the
// transition charges: applications that reserve the GPU's memory up front in
// their own pool and forbid any further cudaMalloc, or language bindings that
// only receive device pointers from their host program and have no allocator
// of their own.  dftb_trans_charges wants a caller-provided workspace; this
// variant instead keeps its scratch (S.C for both orbital blocks and the
// per-atom orbital offsets) in a fixed file-scope device array.
//
// The array exists once per GPU that loads this library and stays resident
// until the process exits.  On the host its name is only a stand-in symbol,
// so its device address is looked up with cudaGetSymbolAddress, once per
// device, the first time the entry point runs with that device current (the
// first call should therefore come before any stream capture).  Under lazy
// module loading the array is committed when this module is first used on a
// device, possibly by that first call.  The cached address belongs to the
// device's primary context; it is not looked up again after cudaDeviceReset.
// All calls on one device share the array: calls that can run at the same time on the GPU
// (unordered streams, concurrent host threads) race on it and must be
// serialised by the caller.  Every call rewrites the parts of the scratch it
// reads, so nothing has to be cleared between calls.
// ============================================================================
namespace {

constexpr size_t kNoAllocScratchBytes = size_t(8) << 20;  // 8 MiB per device
static __device__ __align__(256) unsigned char g_tc_scratch[kNoAllocScratchBytes];

constexpr int kMaxDevices = 64;
void *g_tc_scratch_addr[kMaxDevices] = {nullptr};
std::mutex g_tc_scratch_mutex;

int tc_scratch_address(void **out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) {
        snprintf(g_last_error, sizeof(g_last_error), "trans_charges_noalloc: cudaGetDevice: %s",
                 cudaGetErrorString(e));
        return DFTB_ERR_CUDA;
    }
    if (dev < 0 || dev >= kMaxDevices) return fail(DFTB_ERR_BAD_SIZE, "trans_charges_noalloc: device index");
    std::lock_guard<std::mutex> lock(g_tc_scratch_mutex);
    if (!g_tc_scratch_addr[dev]) {
        void *ptr = nullptr;
        e = cudaGetSymbolAddress(&ptr, g_tc_scratch);
        if (e != cudaSuccess || !ptr) {
            snprintf(g_last_error, sizeof(g_last_error), "trans_charges_noalloc: cudaGetSymbolAddress: %s",
                     cudaGetErrorString(e));
            return DFTB_ERR_CUDA;
        }
        g_tc_scratch_addr[dev] = ptr;
    }
    *out = g_tc_scratch_addr[dev];
    return DFTB_OK;
}

}  // namespace

extern "C" size_t dftb_trans_charges_noalloc_max_bytes(void) { return kNoAllocScratchBytes; }

extern "C" int dftb_trans_charges_noalloc(int norb, int nat, int nocc, int nvirt, const double *co, const double *cv,
                                          const double *Sm, const int *opa, double *q_oo, double *q_ov,
                                          double *q_vv, void *stream) {
    if (norb <= 0 || nat <= 0 || nocc < 0 || nvirt < 0 || nat > norb)
        return fail(DFTB_ERR_BAD_SIZE, "trans_charges_noalloc: sizes");
    // the atom index is the grid's z extent; refuse before anything is launched
    if (nat > 65535) return fail(DFTB_ERR_BAD_SIZE, "trans_charges_noalloc: nat > 65535");
    const size_t need = dftb_trans_charges_workspace_size(norb, nocc, nvirt);
    if (need > kNoAllocScratchBytes) {
        snprintf(g_last_error, sizeof(g_last_error),
                 "trans_charges_noalloc: needs %zu bytes of scratch, the static array holds %zu "
                 "(use dftb_trans_charges with a workspace)",
                 need, kNoAllocScratchBytes);
        return DFTB_ERR_WORKSPACE;
    }
    void *scratch = nullptr;
    int rc = tc_scratch_address(&scratch);
    if (rc) return rc;
    cudaStream_t st = S(stream);
    double *sco, *scv;
    int *first;
    rc = trans_charges_common(norb, nat, nocc, nvirt, co, cv, Sm, opa, scratch, kNoAllocScratchBytes, st, &sco, &scv,
                              &first, false);
    if (rc) return rc;
    struct Blk {
        double *out;
        const double *c1, *s1, *c2, *s2;
        int n1, n2;
    } blks[3] = {{q_oo, co, sco, co, sco, nocc, nocc},
                 {q_ov, co, sco, cv, scv, nocc, nvirt},
                 {q_vv, cv, scv, cv, scv, nvirt, nvirt}};
    for (auto &b : blks) {
        if (!b.out || b.n1 == 0 || b.n2 == 0) continue;
        if ((rc = launch_tc(nat, b.n1, b.n2, first, b.c1, b.s1, b.c2, b.s2, b.out, st, "tc_kernel (noalloc)")))
            return rc;
    }
    return DFTB_OK;
}
