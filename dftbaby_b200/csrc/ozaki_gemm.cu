// FP64 matrix products emulated exactly on the int8 tensor cores of B200 (tcgen05 kind::i8), after the
// "Ozaki scheme II" of Ozaki, Uchino and Imamura (integer modular GEMMs plus the Chinese remainder theorem):
//
//   C = alpha * op(A) op(B) + beta * C            (row-major FP64; op = transpose when trans != 0)
//
// 1. Row m of op(A) is scaled by 2^sa[m] and column n of op(B) by 2^sb[n] and rounded to integers A', B'
//    of at most `bits` bits, chosen so that every entry of A'B' (K terms) stays below P/2 in magnitude,
//    P = p_1 ... p_N the product of N pairwise coprime moduli p_i <= 256.
// 2. For each modulus the symmetric residues A' mod p_i and B' mod p_i (|r| <= 128, int8) are multiplied on
//    the tensor cores with exact int32 accumulation (K < 2^17), and the epilogue keeps the product's residue
//    mod p_i as int8.
// 3. Per element, the Chinese remainder sum is formed from pairs of residues in exact FP64 limbs and reduced modulo P,
//    which gives A'B' to within FP64 rounding, and C = 2^-(sa[m] + sb[n]) A'B'.
//
// The only approximation is step 1: each entry of op(A) (op(B)) is carried with `bits` bits relative to
// the largest entry of its row (column); with N = 16 moduli and K <= 2^17 that is the full 53-bit FP64
// mantissa.  The tensor-core work is N int8 GEMMs (B200: 4.5 dense int8 POPS against ~35 TFLOP/s of FP64
// DGEMM).
//
// Kernels: ozaki_rowscale_kernel and ozaki_colscale_kernel (exponents), ozaki_residue_kernel (int8 residue planes, K-major,
// zero-padded), ozaki_mma_kernel (persistent tcgen05 GEMM over (M tile, N tile, modulus), TMA operand ring,
// double-buffered TMEM accumulators, residue epilogue), ozaki_crt_kernel (reconstruction and scaling).

#include <cuda.h>
#include <cudaTypedefs.h>
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

#include <mutex>

#include "dftbaby_b200.h"
#include "tcgen05.cuh"

namespace ozk {

using namespace tc5;

constexpr int MAXMOD = 16;
// pairwise coprime: 2^8, 3*5*17, 11*23, 13*19 and primes
constexpr int kModuli[MAXMOD] = {256, 255, 253, 251, 247, 241, 239, 233, 229, 227, 223, 211, 199, 197, 193, 191};
constexpr int KMAX = 131071;                // 128 * 128 * K < 2^31: exact int32 accumulation
constexpr int SCALE_NONFINITE = -(1 << 20);  // row/column exponent marking an Inf or NaN entry

// Per modulus p; residues are symmetric (|r| <= p / 2) and formed in FP32, see symres2().
struct Tables {
    float2 np[MAXMOD], invp[MAXMOD];    // -p and 1 / p, twice: the FP32 pair operands
    uint32_t blo[MAXMOD], bhi[MAXMOD];  // int8 weights 2^(8 j) mod p of the bytes j = 0..3 and 4..7
    int rinit[MAXMOD];                  // kMagicBits + (-2^54 mod p): undoes the offset that makes the bytes unsigned
    int c16[MAXMOD];                    // 2^16 mod p, |c16| <= 85
};

// Reconstruction from the first NM moduli, two at a time: with P_k = p_a p_b and W_k = P / P_k,
//   X = sum_k W_k u_k mod P,  u_k = r_a A_a + r_b A_b,  A_a = p_b ((P / p_a)^-1 mod p_a) mod P_k
// (int16 coefficients; |u_k| < 2^23).  W_k and P are held as balanced 28-bit limbs in FP64.
struct CrtTables {
    int a[MAXMOD / 2];           // A_a | A_b << 16
    double w[MAXMOD / 2][4];     // limbs of W_k
    double p[4];                 // limbs of P
    double qscale;               // 2^(28 (limbs - 1)) / P
};

constexpr int kMagicBits = 0x4B400000;     // 1.5 2^23: adding it to an integer |t| < 2^22 gives the float 1.5 2^23 + t
constexpr float kMagic = 12582912.0f;

// FP32 pair arithmetic: one instruction slot for two operations (the residue and epilogue loops are issue-bound)
__device__ __forceinline__ uint64_t f32x2(float a, float b) {
    return (uint64_t)__float_as_uint(a) | (uint64_t)__float_as_uint(b) << 32;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

// Two words whose low bytes are the symmetric residues of t modulo p, from the bits of the floats 1.5 2^23 + t,
// |t| < 2^22: t / p is rounded to an integer q with an error below 2^-11 (FP32 product against 1.5 2^23, whose ulp
// is 1), so t - p q is within p / 2 + 0.1 of zero, exact, and for odd p the canonical residue (for p = 256, +-128
// are one byte).
__device__ __forceinline__ void symres2(int tm0, int tm1, uint64_t np, uint64_t invp, uint32_t &r0, uint32_t &r1) {
    const uint64_t magic = f32x2(kMagic, kMagic), nmagic = f32x2(-kMagic, -kMagic);
    const uint64_t tm = (uint64_t)(uint32_t)tm0 | (uint64_t)(uint32_t)tm1 << 32;
    const uint64_t q = add2(fma2(add2(tm, nmagic), invp, magic), nmagic);
    const uint64_t r = fma2(np, q, tm);
    r0 = (uint32_t)r;
    r1 = (uint32_t)(r >> 32);
}

__device__ __forceinline__ uint32_t pack4(uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    return __byte_perm(__byte_perm(a, b, 0x0040), __byte_perm(c, d, 0x0040), 0x5410);
}

__device__ __forceinline__ int dp4a_us(uint32_t a, uint32_t b, int c) {  // unsigned bytes of a, signed bytes of b
    int d;
    asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}

// 2^e as a double, |e| <= 1022
__device__ __forceinline__ double pow2(int e) { return __hiloint2double((1023 + e) << 20, 0); }

// x 2^e for any e (exact unless the result leaves the normal range)
__device__ __forceinline__ double scale2(double x, int e) {
    return (unsigned)(e + 1000) <= 2000u ? x * pow2(e) : ldexp(x, e);
}

// ---------------------------------------------------------------------------- scaling and residues

// Y(r, k) = X[r * ldx + k]; s[r] = bits - 1 - ilogb(max_k |Y(r, k)|) so that
// |Y(r, k)| 2^s[r] < 2^bits (0 for a zero row, SCALE_NONFINITE for a row holding Inf or NaN); rows in
// [rows, rpad) get 0.
__global__ void ozaki_rowscale_kernel(int rows, int rpad, int K, const double *X, long long ldx, int bits, int *s) {
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (warp >= rpad) return;
    double m = 0.0;
    bool bad = false;
    if (warp < rows) {
        const double *x = X + (long long)warp * ldx;
        int k = lane;
        for (; k + 96 < K; k += 128) {
            // four independent loads in flight per lane
            const double a0 = fabs(x[k]), a1 = fabs(x[k + 32]), a2 = fabs(x[k + 64]), a3 = fabs(x[k + 96]);
            bad |= !(a0 <= 1.7976931348623157e308 && a1 <= 1.7976931348623157e308 &&
                     a2 <= 1.7976931348623157e308 && a3 <= 1.7976931348623157e308);
            m = fmax(fmax(m, fmax(a0, a1)), fmax(a2, a3));
        }
        for (; k < K; k += 32) {
            const double a = fabs(x[k]);
            bad |= !(a <= 1.7976931348623157e308);
            m = fmax(m, a);
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
        bad |= __shfl_xor_sync(0xffffffffu, (int)bad, o) != 0;
    }
    if (lane == 0) s[warp] = bad ? SCALE_NONFINITE : (m > 0.0 ? bits - 1 - ilogb(m) : 0);
}

// The same for rows that are strided in memory (Y(r, k) = X[k * ldx + r]): a cluster of RC_SPLIT CTAs takes 32 rows
// (consecutive in memory), each CTA a range of k with RC_PHASES phases, and the first CTA joins their maxima.
// Split because 4146 rows are 130 blocks, too few loads in flight for one pass over 137 MB: 42 -> 39 us for 4146 x 4146,
// and 96 us before with 32 phases in one block.
constexpr int RC_SPLIT = 8, RC_PHASES = 8;
__global__ void __cluster_dims__(1, RC_SPLIT, 1) __launch_bounds__(32 * RC_PHASES)
    ozaki_colscale_kernel(int rows, int rpad, int K, const double *X, long long ldx, int bits, int *s) {
    __shared__ double sm[RC_PHASES][32];
    __shared__ double best[32];  // this CTA's maximum per row; infinite for a row holding Inf or NaN
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    const int tx = threadIdx.x, ty = threadIdx.y, r = blockIdx.x * 32 + tx;
    const int kper = (K + RC_SPLIT - 1) / RC_SPLIT;
    const int k0 = blockIdx.y * kper, k1 = min(K, k0 + kper);
    const double inf = __longlong_as_double(0x7ff0000000000000ll);
    double m = 0.0;
    if (r < rows) {
        int k = k0 + ty;
        for (; k + 7 * RC_PHASES < k1; k += 8 * RC_PHASES) {
            double a[8];
            const double *x = X + (long long)k * ldx + r;
#pragma unroll
            for (int u = 0; u < 8; ++u, x += RC_PHASES * ldx) a[u] = fabs(*x);
#pragma unroll
            for (int u = 0; u < 8; ++u) m = a[u] <= m ? m : (a[u] < inf ? a[u] : inf);  // NaN fails both: infinite
        }
        for (; k < k1; k += RC_PHASES) {
            const double a = fabs(X[(long long)k * ldx + r]);
            m = a <= m ? m : (a < inf ? a : inf);
        }
    }
    sm[ty][tx] = m;
    __syncthreads();
    if (ty == 0) {
#pragma unroll
        for (int y = 1; y < RC_PHASES; ++y) m = fmax(m, sm[y][tx]);
        best[tx] = m;
    }
    cluster.sync();
    if (cluster.block_rank() == 0 && ty == 0 && r < rpad) {
        for (int c = 1; c < RC_SPLIT; ++c) m = fmax(m, *cluster.map_shared_rank(&best[tx], c));
        s[r] = m == inf ? SCALE_NONFINITE : (m > 0.0 ? bits - 1 - ilogb(m) : 0);
    }
    cluster.sync();  // the other CTAs' shared memory stays until it has been read
}

constexpr int RT_ROWS = 32, RT_K = 128;

// Residue planes R[i][r][k] (i < nmod, r < rows_write, k < kpad; zero outside rows x K) of the scaled,
// rounded Y(r, k) 2^s[r].  One block per 32 x 128 tile of Y; a warp takes four rows, a lane four consecutive k of each,
// so the int8 writes are 128 contiguous bytes.  Rows that are contiguous in memory are read straight into registers;
// strided ones (TRANS) are read along r and turned in shared memory, in 16-byte slots swizzled by the row.  Bound by
// instruction issue, then by DRAM: about 6 instructions per entry and modulus (two dp4a, two FP32 pair operations for
// two entries, packing).  B200, 4146 x 4146, 16 moduli (430 MB): 187 -> 90 us (rows contiguous) and 95 us (strided).
template <int NM, bool TRANS>
__global__ void __launch_bounds__(256) ozaki_residue_kernel(int rows, int rows_write, int K, const double *X,
                                                            long long ldx, const int *s,
                                                            const __grid_constant__ Tables tb, int8_t *R,
                                                            long long plane, int kpad) {
    __shared__ __align__(16) double tile[TRANS ? RT_ROWS * RT_K : 2];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r0 = blockIdx.y * RT_ROWS, k0 = blockIdx.x * RT_K;
    const int k = k0 + 4 * lane;
    double x[4][4];
    if (TRANS) {
        const double *p = X + (long long)(k0 + warp) * ldx + r0 + lane;
        const bool in = r0 + lane < rows;
        double v[RT_K / 8];
#pragma unroll
        for (int j = 0; j < RT_K / 8; ++j, p += 8 * ldx) v[j] = (in && k0 + warp + 8 * j < K) ? *p : 0.0;
#pragma unroll
        for (int j = 0; j < RT_K / 8; ++j) {
            const int kk = warp + 8 * j;
            tile[lane * RT_K + (((kk >> 1) ^ (lane & 7)) << 1) + (kk & 1)] = v[j];
        }
        __syncthreads();
    } else {
        const bool vec = ((ldx & 1) | (reinterpret_cast<uintptr_t>(X) & 8)) == 0 && k + 3 < K;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int r = r0 + warp + 8 * j;
            const double *p = X + (long long)r * ldx + k;
            if (r < rows && vec) {
                const double2 a = *reinterpret_cast<const double2 *>(p), b = *reinterpret_cast<const double2 *>(p + 2);
                x[j][0] = a.x, x[j][1] = a.y, x[j][2] = b.x, x[j][3] = b.y;
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e) x[j][e] = (r < rows && k + e < K) ? p[e] : 0.0;
            }
        }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int rr = warp + 8 * j, r = r0 + rr;
        if (r >= rows_write) break;
        if (TRANS) {
            const double2 a = *reinterpret_cast<const double2 *>(tile + rr * RT_K + (((2 * lane) ^ (rr & 7)) << 1));
            const double2 b = *reinterpret_cast<const double2 *>(tile + rr * RT_K + (((2 * lane + 1) ^ (rr & 7)) << 1));
            x[j][0] = a.x, x[j][1] = a.y, x[j][2] = b.x, x[j][3] = b.y;
        }
        const int sr = r < rows ? s[r] : SCALE_NONFINITE;
        // the scaled, rounded entries (at most 53 bits) plus 2^54, as seven unsigned bytes
        uint32_t lo[4], hi[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const long long ai = sr == SCALE_NONFINITE ? 0ll : __double2ll_rn(scale2(x[j][e], sr));
            const unsigned long long u = (unsigned long long)(ai + (1ll << 54));
            lo[e] = (uint32_t)u;
            hi[e] = (uint32_t)(u >> 32);
        }
        int8_t *out = R + (long long)r * kpad + k;
#pragma unroll
        for (int i = 0; i < NM; ++i, out += plane) {
            const uint64_t np = f32x2(tb.np[i].x, tb.np[i].y), invp = f32x2(tb.invp[i].x, tb.invp[i].y);
            int t[4];
            uint32_t rd[4];
#pragma unroll
            for (int e = 0; e < 4; ++e)  // seven products below 255 127: |t| < 2^18
                t[e] = dp4a_us(lo[e], tb.blo[i], dp4a_us(hi[e], tb.bhi[i], tb.rinit[i]));
            symres2(t[0], t[1], np, invp, rd[0], rd[1]);
            symres2(t[2], t[3], np, invp, rd[2], rd[3]);
            *reinterpret_cast<uint32_t *>(out) = pack4(rd[0], rd[1], rd[2], rd[3]);
        }
    }
}

// ---------------------------------------------------------------------------- int8 tensor-core GEMM

// 128 x 256 output tiles: per 128-byte K block a stage holds 16 KiB of A and 32 KiB of B for four
// 128 x 256 x 32 MMAs, a third fewer operand bytes per MMA than 128 x 128 tiles
constexpr int BM = 128, BN = 256, BKB = 128;  // tile rows, tile columns, K bytes (= int8 elements) per stage
constexpr int TILE_BYTES = BM * BKB;          // 16 KiB (A)
constexpr int TILE_B_BYTES = BN * BKB;        // 32 KiB (B)
constexpr int STAGES = 4;
constexpr int STAGE_BYTES = TILE_BYTES + TILE_B_BYTES;
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 /* alignment slack */ + 256 /* barriers */;
constexpr int EPI_THREADS = 128;
// instruction descriptor: D = S32 (bits 4-5 = 2), A = B = signed int8 (bits 7-9, 10-12 = 1), both K-major,
// N >> 3 at bit 17, M >> 4 at bit 24
constexpr uint32_t kIdescI8 = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) |
                              ((uint32_t)(BM >> 4) << 24);

__device__ __forceinline__ void umma_i8(uint32_t tmem_c, uint64_t da, uint64_t db, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_c),
        "l"(da), "l"(db), "r"(kIdescI8), "r"(accumulate));
}

struct Maps {
    CUtensorMap a;  // residue planes of the A operand: nmod * arows rows x kpad int8
    CUtensorMap b;  // residue planes of the B operand: nmod * brows rows x kpad int8
};

struct MmaParams {
    int M, N, kpad, nmod;
    int arows, brows;  // rows per residue plane of the A and B operands (multiples of 256)
    int8_t *RC;  // product residues: plane i at RC + i * planeC, row-major with ldr (multiple of 32)
    long long planeC;
    int ldr;
    int *err;
};

// Persistent kernel, one CTA per SM over the tiles t = (m tile, n tile, modulus), M fastest:
//   warp 0 lane 0 : TMA producer over a 4-stage ring of 128-byte-wide A (128 rows) and B (256 rows) tiles
//                   (128-byte swizzle);
//   warp 1 lane 0 : tcgen05.mma kind::i8 issuer (M = 128, N = 256, K = 32 per instruction) into one of two
//                   256-column int32 TMEM accumulators (tile j uses accumulator j % 2);
//   warps 2..5    : epilogue of tile j under the MMAs of tile j + 1: int32 -> residue mod p -> int8.  It must take less
//                   than a tile's MMAs (7k cycles at K = 1225): in FP64 it did not (8292 x 8292 x 1225, 14 moduli:
//                   1.49 ms), in FP32 pairs it does (1.06 ms).
// Every wait is bounded; on timeout the kernel records an error code, stops issuing, drains its copies
// and releases TMEM.
__global__ void __launch_bounds__(192, 1) ozaki_mma_kernel(const __grid_constant__ Maps maps, const MmaParams p,
                                                           const __grid_constant__ Tables tb) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + STAGES * STAGE_BYTES);
    uint64_t *empty = full + STAGES;
    uint64_t *tfull = empty + STAGES;
    uint64_t *tempty = tfull + 2;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(tempty + 2);
    int *abort_flag = reinterpret_cast<int *>(tmem_slot + 1);

    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const int mt = (p.M + BM - 1) / BM, nt = (p.N + BN - 1) / BN;
    const int ntiles = mt * nt * p.nmod;
    const int kblocks = p.kpad / BKB;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(&tfull[a], 1);
            mbar_init(&tempty[a], EPI_THREADS);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncwarp();
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(2 * BN));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            // ---------------- TMA producer
            int it = 0;
            bool stop = false;
            for (int t = blockIdx.x; t < ntiles && !stop; t += gridDim.x) {
                const int mi = t % mt, ni = (t / mt) % nt, mod = t / (mt * nt);
                const int ya = mod * p.arows + mi * BM, yb = mod * p.brows + ni * BN;
                for (int kb = 0; kb < kblocks; ++kb) {
                    const int s = it % STAGES;
                    if (it >= STAGES && !mbar_wait(&empty[s], ((it / STAGES) - 1) & 1)) {
                        atomicExch(p.err, 1);
                        *(volatile int *)abort_flag = 1;
                        stop = true;
                        break;
                    }
                    if (*(volatile int *)abort_flag) {
                        stop = true;
                        break;
                    }
                    uint8_t *sa = smem + s * STAGE_BYTES;
                    mbar_expect_tx(&full[s], STAGE_BYTES);
                    tma_load_2d(sa, &maps.a, &full[s], kb * BKB, ya);
                    tma_load_2d(sa + TILE_BYTES, &maps.b, &full[s], kb * BKB, yb);
                    ++it;
                }
            }
            // drain: wait (bounded) until every copy that was started has landed
            for (int j = max(0, it - STAGES); j < it; ++j) mbar_wait(&full[j % STAGES], (j / STAGES) & 1);
        }
    } else if (warp == 1) {
        if (lane == 0) {
            // ---------------- MMA issuer
            int it = 0, j = 0;
            bool stop = false;
            for (int t = blockIdx.x; t < ntiles && !stop; t += gridDim.x, ++j) {
                const int acc = j & 1;
                const uint32_t tacc = tmem + (uint32_t)(acc * BN);
                if (j >= 2 && !mbar_wait(&tempty[acc], ((j >> 1) - 1) & 1)) {
                    atomicExch(p.err, 4);
                    *(volatile int *)abort_flag = 1;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                for (int kb = 0; kb < kblocks; ++kb) {
                    const int s = it % STAGES;
                    if (!mbar_wait(&full[s], (it / STAGES) & 1)) {
                        atomicExch(p.err, 2);
                        *(volatile int *)abort_flag = 1;
                        stop = true;
                        break;
                    }
                    if (*(volatile int *)abort_flag) {
                        stop = true;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t sa = smem_u32(smem + s * STAGE_BYTES), sb = sa + TILE_BYTES;
#pragma unroll
                    for (int k = 0; k < BKB / 32; ++k) {
                        // 32 int8 = 32 bytes along K per instruction, inside the 128-byte swizzle atom
                        umma_i8(tacc, smem_desc_k128(sa + k * 32), smem_desc_k128(sb + k * 32),
                                (kb > 0 || k > 0) ? 1u : 0u);
                    }
                    umma_commit(&empty[s]);
                    ++it;
                }
                umma_commit(&tfull[acc]);
            }
        }
    } else {
        // ---------------- epilogue (warps 2..5): TMEM lanes 32 (warp % 4) .. + 31 are this warp's rows
        const int rq = warp & 3;
        const int rloc = rq * 32 + lane;
        int j = 0;
        for (int t = blockIdx.x; t < ntiles; t += gridDim.x, ++j) {
            const int mi = t % mt, ni = (t / mt) % nt, mod = t / (mt * nt);
            const int acc = j & 1;
            const int row = mi * BM + rloc, n0 = ni * BN;
            const uint64_t np = f32x2(tb.np[mod].x, tb.np[mod].y), invp = f32x2(tb.invp[mod].x, tb.invp[mod].y);
            const int c16 = tb.c16[mod];
            const bool ok = __all_sync(0xffffffffu, mbar_wait(&tfull[acc], (j >> 1) & 1) ? 1 : 0) != 0;
            if (!ok && lane == 0) atomicExch(p.err, 3);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const bool live = ok && !*(volatile int *)abort_flag && kblocks > 0;  // warp-uniform
            for (int c0 = 0; c0 < BN; c0 += 32) {
                uint32_t v[32];
                tmem_ld32_raw(tmem + ((uint32_t)(rq * 32) << 16) + (uint32_t)(acc * BN + c0), v);
                const int col0 = n0 + c0;
                if (live && row < p.M && col0 < p.N) {
                    uint32_t w[8];
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        // a = ah 2^16 + al: |ah c16 + al| <= 2^15 85 + 2^16 < 2^22
                        int t[4];
                        uint32_t rd[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const int a = (int)v[4 * q + e];
                            t[e] = (a >> 16) * c16 + ((a & 0xffff) | kMagicBits);
                        }
                        symres2(t[0], t[1], np, invp, rd[0], rd[1]);
                        symres2(t[2], t[3], np, invp, rd[2], rd[3]);
                        w[q] = pack4(rd[0], rd[1], rd[2], rd[3]);
                    }
                    uint4 *dst = reinterpret_cast<uint4 *>(p.RC + mod * p.planeC + (long long)row * p.ldr + col0);
                    dst[0] = make_uint4(w[0], w[1], w[2], w[3]);
                    dst[1] = make_uint4(w[4], w[5], w[6], w[7]);
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            mbar_arrive(&tempty[acc]);
            if (!ok) break;
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * BN));
    }
}

// ---------------------------------------------------------------------------- reconstruction

constexpr __host__ __device__ int crt_limbs(int nmod) { return nmod >= 13 ? 4 : (nmod >= 9 ? 3 : 2); }

// C[m][n] = alpha G[m][n] 2^-(sa[m] + sb[n]) X + beta C[m][n] (G optional), X the integer with residues RC[i][m][n]:
// the limbs S_l = sum_k u_k W_k,l are exact in FP64 (|u_k| < 2^23, |W_k,l| <= 2^27, 8 terms), Q = round(S / P) from the
// three highest, and X = sum_l (S_l - Q P_l) 2^(28 l), rounded at most once per limb below the first that exceeds 53 bits.
// Four consecutive columns per thread (one 32-bit word per residue plane); NM moduli.  Per entry it costs 8 PRMT, 8 dp2a
// and ~55 FP64 operations, where the mixed-radix (Garner) form took 120 multiply-adds and 15 reductions: B200, 4146 x
// 4146 from 16 planes (413 MB) 282 -> 99 us, 8292 x 8292 from 14 planes 1080 -> 360 us.
template <int NM>
__global__ void __launch_bounds__(256) ozaki_crt_kernel(int M, int N, const int8_t *RC, long long planeC, int ldr,
                                                        const int *sa, const int *sb, double alpha, const double *G,
                                                        long long ldg, double beta, double *C, long long ldc,
                                                        const __grid_constant__ CrtTables tb) {
    constexpr int NP = (NM + 1) / 2, NL = crt_limbs(NM), NW = (NM + 3) / 4;
    const int nq = (N + 3) / 4;
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long long)M * nq) return;
    const int m = (int)(idx / nq), n0 = (int)(idx % nq) * 4;
    uint32_t wd[4 * NW];
#pragma unroll
    for (int i = 0; i < 4 * NW; ++i)
        wd[i] = i < NM ? *reinterpret_cast<const uint32_t *>(RC + i * planeC + (long long)m * ldr + n0) : 0u;
    // 4 x 4 byte transposes: word 4 g + e then holds the residues modulo p_4g .. p_4g+3 of column e
#pragma unroll
    for (int g = 0; g < NW; ++g) {
        uint32_t *w = wd + 4 * g;
        const uint32_t a = __byte_perm(w[0], w[1], 0x5140), b = __byte_perm(w[2], w[3], 0x5140);
        const uint32_t c = __byte_perm(w[0], w[1], 0x7362), d = __byte_perm(w[2], w[3], 0x7362);
        w[0] = __byte_perm(a, b, 0x5410);
        w[1] = __byte_perm(a, b, 0x7632);
        w[2] = __byte_perm(c, d, 0x5410);
        w[3] = __byte_perm(c, d, 0x7632);
    }
    const int sm = sa[m];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const int n = n0 + e;
        if (n >= N) break;
        double S[NL];
#pragma unroll
        for (int l = 0; l < NL; ++l) S[l] = 0.0;
#pragma unroll
        for (int k = 0; k < NP; ++k) {
            const int r = (int)wd[4 * (k / 2) + e];
            // u + 2^24 > 0 in the low word of 2^52 + (u + 2^24)
            const int u = (k & 1) ? __dp2a_hi(tb.a[k], r, 1 << 24) : __dp2a_lo(tb.a[k], r, 1 << 24);
            const double ud = __hiloint2double(0x43300000, u) - (4503599627370496.0 + 16777216.0);
#pragma unroll
            for (int l = 0; l < NL; ++l) S[l] = fma(ud, tb.w[k][l], S[l]);
        }
        double q = fma(S[NL - 2], 0x1p-28, S[NL - 1]);
        if (NL > 2) q = fma(S[NL > 2 ? NL - 3 : 0], 0x1p-56, q);
        q = __dsub_rn(fma(q, tb.qscale, 6755399441055744.0), 6755399441055744.0);  // rounded: 1.5 2^52 has ulp 1
        double x = fma(-q, tb.p[NL - 1], S[NL - 1]);
#pragma unroll
        for (int l = NL - 2; l >= 0; --l) x = fma(x, 0x1p28, fma(-q, tb.p[l], S[l]));
        const int sn = sb[n];
        double out;
        if (sm == SCALE_NONFINITE || sn == SCALE_NONFINITE)
            out = __longlong_as_double(0x7ff8000000000000ll);  // NaN
        else
            out = alpha * scale2(x, -(sm + sn));
        if (G) out *= G[(long long)m * ldg + n];
        double *c = C + (long long)m * ldc + n;
        *c = beta == 0.0 ? out : out + beta * *c;
    }
}

template <int NM>
void launch_crt(int M, int N, const int8_t *RC, long long planeC, int ldr, const int *sa, const int *sb, double alpha,
                const double *G, long long ldg, double beta, double *C, long long ldc, const CrtTables &tb,
                cudaStream_t st) {
    const long long nthreads = (long long)M * ((N + 3) / 4);
    ozaki_crt_kernel<NM><<<(unsigned)((nthreads + 255) / 256), 256, 0, st>>>(M, N, RC, planeC, ldr, sa, sb, alpha,
                                                                             G, ldg, beta, C, ldc, tb);
}

// ---------------------------------------------------------------------------- host side
thread_local char g_err[256] = "";
PFN_cuTensorMapEncodeTiled_v12000 g_encode = nullptr;
std::mutex g_mutex;
Tables g_tables;
CrtTables g_crt[MAXMOD + 1];
bool g_tables_ready = false;

using u128 = unsigned __int128;

// balanced 28-bit limbs of v, the highest unreduced
void limbs28(u128 v, int n, double *out) {
    for (int l = 0; l < n - 1; ++l) {
        long long d = (long long)(v & ((1u << 28) - 1));
        v >>= 28;
        if (d >= (1 << 27)) {
            d -= 1 << 28;
            v += 1;
        }
        out[l] = (double)d;
    }
    out[n - 1] = (double)(unsigned long long)v;
}

void init_crt(CrtTables &t, int nmod) {
    const int nl = crt_limbs(nmod);
    u128 P = 1;
    for (int i = 0; i < nmod; ++i) P *= (u128)kModuli[i];  // below 2^126
    limbs28(P, nl, t.p);
    double Pd = 0.0;
    for (int l = nl - 1; l >= 0; --l) Pd = Pd * 268435456.0 + t.p[l];
    t.qscale = ldexp(1.0, 28 * (nl - 1)) / Pd;
    for (int k = 0; 2 * k < nmod; ++k) {
        const int pa = kModuli[2 * k], pb = 2 * k + 1 < nmod ? kModuli[2 * k + 1] : 1;
        const int pk = pa * pb;
        limbs28(P / (u128)pk, nl, t.w[k]);
        int A[2] = {0, 0};
        for (int h = 0; h < 2; ++h) {
            const int p = h == 0 ? pa : pb, other = h == 0 ? pb : pa;
            if (p == 1) continue;
            const int rest = (int)((P / (u128)p) % (u128)p);
            int inv = 1;
            while ((long long)rest * inv % p != 1) ++inv;
            int c = (int)((long long)other * inv % pk);
            if (c > pk / 2) c -= pk;
            A[h] = c;
        }
        t.a[k] = (int)(((uint32_t)A[0] & 0xffffu) | ((uint32_t)A[1] << 16));
    }
}

int init_host() {
    std::lock_guard<std::mutex> lock(g_mutex);
    if (!g_encode) {
        cudaDriverEntryPointQueryResult q;
        void *fn = nullptr;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) !=
                cudaSuccess ||
            q != cudaDriverEntryPointSuccess || !fn) {
            snprintf(g_err, sizeof(g_err), "cuTensorMapEncodeTiled unavailable");
            return -1;
        }
        g_encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
    }
    if (!g_tables_ready) {
        Tables &t = g_tables;
        for (int i = 0; i < MAXMOD; ++i) {
            const int p = kModuli[i];
            auto sym = [p](long long v) {
                const int r = (int)(((v % p) + p) % p);
                return r > p / 2 ? r - p : r;
            };
            t.np[i] = make_float2(-(float)p, -(float)p);
            t.invp[i] = make_float2(1.0f / (float)p, 1.0f / (float)p);
            uint32_t w[2] = {0, 0};
            for (int j = 0; j < 7; ++j) w[j >> 2] |= (uint32_t)(uint8_t)(int8_t)sym(1ll << (8 * j)) << (8 * (j & 3));
            t.blo[i] = w[0];
            t.bhi[i] = w[1];
            t.rinit[i] = kMagicBits + sym(-(1ll << 54));
            t.c16[i] = sym(1ll << 16);
        }
        for (int nmod = 8; nmod <= MAXMOD; ++nmod) init_crt(g_crt[nmod], nmod);
        g_tables_ready = true;
    }
    return 0;
}

int make_map_i8(CUtensorMap *map, const void *base, long long rows, int kpad, int box_rows) {
    cuuint64_t dims[2] = {(cuuint64_t)kpad, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)kpad};
    cuuint32_t box[2] = {(cuuint32_t)BKB, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void *>(base), dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        snprintf(g_err, sizeof(g_err), "cuTensorMapEncodeTiled (int8) failed (%d): rows %lld kpad %d", (int)r, rows,
                 kpad);
        return -1;
    }
    return 0;
}

inline long long up(long long x, long long q) { return (x + q - 1) / q * q; }

// An operand in residue form: rows_total rows (padded to 256) of a K-major matrix, k columns (padded to 128):
//   int32 exponent per row | nmod int8 residue planes of rpad x kpad
struct OperandLayout {
    long long rpad, kpad, plane;
    size_t off_res, total;
};

OperandLayout operand_layout(int rows_total, int k, int nmod) {
    OperandLayout L;
    L.rpad = up(rows_total, 256);
    L.kpad = up(k, BKB);
    L.plane = L.rpad * L.kpad;
    L.off_res = (size_t)up(4 * L.rpad, 256);
    L.total = L.off_res + (size_t)nmod * L.plane;
    return L;
}

// product residues: nmod planes of m x ldr int8
inline long long product_ldr(int n) { return up(n, 32); }
inline size_t product_bytes(int m, int n, int nmod) { return (size_t)up((long long)nmod * m * product_ldr(n), 256); }

// largest bit count b with K 2^(2b) < P/2 (P the product of the first nmod moduli), at most 53
int scale_bits(int k, int nmod) {
    double log2P = 0.0;
    for (int i = 0; i < nmod; ++i) log2P += log2((double)kModuli[i]);
    const int b = (int)floor((log2P - 1.0 - log2((double)k) - 1e-6) / 2.0);
    return b < 53 ? b : 53;
}

int check_shape(int k, int nmod) {
    if (k <= 0 || k > KMAX || nmod < 8 || nmod > MAXMOD) {
        snprintf(g_err, sizeof(g_err), "ozaki: 0 < k <= %d and 8 <= nmod <= %d required", KMAX, MAXMOD);
        return DFTB_ERR_BAD_SIZE;
    }
    if (scale_bits(k, nmod) < 16) {
        snprintf(g_err, sizeof(g_err), "ozaki: %d moduli leave too few bits at k = %d", nmod, k);
        return DFTB_ERR_BAD_SIZE;
    }
    return DFTB_OK;
}

// rows [row0, row0 + rows) of the operand from Y(r, k) = trans ? X[k][r] : X[r][k]; when they are the last
// rows (row0 + rows == rows_total) the padding rows up to 256 are written as zeros too
int prepare(int trans, int rows, int k, const double *X, long long ldx, int nmod, uint8_t *op, int rows_total,
            int row0, cudaStream_t st) {
    const OperandLayout L = operand_layout(rows_total, k, nmod);
    const int bits = scale_bits(k, nmod);
    const int rows_write = (row0 + rows == rows_total) ? (int)(L.rpad - row0) : rows;
    int *s = reinterpret_cast<int *>(op) + row0;
    int8_t *R = reinterpret_cast<int8_t *>(op + L.off_res) + (long long)row0 * L.kpad;
    if (!trans) {
        const long long threads = (long long)rows_write * 32;
        ozaki_rowscale_kernel<<<(unsigned)((threads + 255) / 256), 256, 0, st>>>(rows, rows_write, k, X, ldx, bits, s);
    } else {
        ozaki_colscale_kernel<<<dim3((unsigned)((rows_write + 31) / 32), RC_SPLIT), dim3(32, RC_PHASES), 0, st>>>(
            rows, rows_write, k, X, ldx, bits, s);
    }
    dim3 g((unsigned)(L.kpad / RT_K), (unsigned)((rows_write + RT_ROWS - 1) / RT_ROWS));
    switch (nmod) {
#define OZK_RES(NMV)                                                                                            \
    case NMV:                                                                                                   \
        if (trans)                                                                                              \
            ozaki_residue_kernel<NMV, true><<<g, 256, 0, st>>>(rows, rows_write, k, X, ldx, s, g_tables, R,     \
                                                               L.plane, (int)L.kpad);                           \
        else                                                                                                    \
            ozaki_residue_kernel<NMV, false><<<g, 256, 0, st>>>(rows, rows_write, k, X, ldx, s, g_tables, R,    \
                                                                L.plane, (int)L.kpad);                          \
        break;
        OZK_RES(8)
        OZK_RES(9)
        OZK_RES(10)
        OZK_RES(11)
        OZK_RES(12)
        OZK_RES(13)
        OZK_RES(14)
        OZK_RES(15)
        OZK_RES(16)
#undef OZK_RES
    }
    return cudaGetLastError() == cudaSuccess ? DFTB_OK : DFTB_ERR_CUDA;
}

int product(int m, int n, int k, int nmod, const uint8_t *A, int rows_a, const uint8_t *B, int rows_b, double alpha,
            const double *G, long long ldg, double beta, double *C, long long ldc, int8_t *RC, int *err,
            cudaStream_t st) {
    const OperandLayout LA = operand_layout(rows_a, k, nmod), LB = operand_layout(rows_b, k, nmod);
    Maps maps;
    memset(&maps, 0, sizeof(maps));
    if (make_map_i8(&maps.a, A + LA.off_res, (long long)nmod * LA.rpad, (int)LA.kpad, BM) ||
        make_map_i8(&maps.b, B + LB.off_res, (long long)nmod * LB.rpad, (int)LB.kpad, BN))
        return DFTB_ERR_CUDA;
    MmaParams p;
    p.M = m;
    p.N = n;
    p.kpad = (int)LA.kpad;
    p.nmod = nmod;
    p.arows = (int)LA.rpad;
    p.brows = (int)LB.rpad;
    p.RC = RC;
    p.ldr = (int)product_ldr(n);
    p.planeC = (long long)m * p.ldr;
    p.err = err;
    static bool attr_set[64] = {false};
    static int sm_count[64] = {0};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !attr_set[dev]) {
        if (cudaFuncSetAttribute(ozaki_mma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES) !=
            cudaSuccess) {
            snprintf(g_err, sizeof(g_err), "ozaki: cannot reserve %d bytes of shared memory", SMEM_BYTES);
            return DFTB_ERR_CUDA;
        }
        int nsm = 0;
        if (cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || nsm <= 0) nsm = 148;
        sm_count[dev] = nsm;
        attr_set[dev] = true;
    }
    const int sms = (dev >= 0 && dev < 64) ? sm_count[dev] : 148;
    const long long ntiles = (long long)((m + BM - 1) / BM) * ((n + BN - 1) / BN) * nmod;
    if (ntiles > (1LL << 30)) return DFTB_ERR_BAD_SIZE;
    ozaki_mma_kernel<<<(unsigned)(ntiles < sms ? ntiles : sms), 192, SMEM_BYTES, st>>>(maps, p, g_tables);
    const int *sa = reinterpret_cast<const int *>(A), *sb = reinterpret_cast<const int *>(B);
    switch (nmod) {
#define OZK_CRT(NMV)                                                                                              \
    case NMV:                                                                                                     \
        launch_crt<NMV>(m, n, RC, p.planeC, p.ldr, sa, sb, alpha, G, ldg, beta, C, ldc, g_crt[nmod], st); \
        break;
        OZK_CRT(8)
        OZK_CRT(9)
        OZK_CRT(10)
        OZK_CRT(11)
        OZK_CRT(12)
        OZK_CRT(13)
        OZK_CRT(14)
        OZK_CRT(15)
        OZK_CRT(16)
#undef OZK_CRT
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        snprintf(g_err, sizeof(g_err), "ozaki: %s", cudaGetErrorString(e));
        return DFTB_ERR_CUDA;
    }
    return DFTB_OK;
}

}  // namespace ozk

extern "C" {

const char *dftb_ozaki_last_error(void) { return ozk::g_err; }

size_t dftb_ozaki_operand_size(int rows, int k, int nmod) {
    if (rows <= 0 || ozk::check_shape(k, nmod) != DFTB_OK) return 0;
    return ozk::operand_layout(rows, k, nmod).total;
}

int dftb_ozaki_prepare(int trans, int rows, int k, const double *X, int ldx, int nmod, void *operand, int rows_total,
                       int row0, void *stream) {
    using namespace ozk;
    if (int rc = check_shape(k, nmod)) return rc;
    if (rows <= 0 || row0 < 0 || row0 + rows > rows_total || ldx < (trans ? rows : k)) {
        snprintf(g_err, sizeof(g_err), "ozaki_prepare: rows %d at %d of %d, ldx %d", rows, row0, rows_total, ldx);
        return DFTB_ERR_BAD_SIZE;
    }
    if (!X || !operand) return DFTB_ERR_NULL;
    if (reinterpret_cast<uintptr_t>(operand) & 255) {
        snprintf(g_err, sizeof(g_err), "ozaki_prepare: the operand must be 256-byte aligned");
        return DFTB_ERR_BAD_SIZE;
    }
    if (init_host()) return DFTB_ERR_CUDA;
    return prepare(trans, rows, k, X, ldx, nmod, reinterpret_cast<uint8_t *>(operand), rows_total, row0,
                   reinterpret_cast<cudaStream_t>(stream));
}

size_t dftb_ozaki_product_workspace_size(int m, int n, int nmod) {
    if (m <= 0 || n <= 0 || nmod < 1 || nmod > ozk::MAXMOD) return 0;
    return ozk::product_bytes(m, n, nmod);
}

int dftb_ozaki_product(int m, int n, int k, int nmod, const void *A, int rows_a, const void *B, int rows_b,
                       double alpha, const double *G, int ldg, double beta, double *C, int ldc, void *work,
                       size_t work_bytes, int *err, void *stream) {
    using namespace ozk;
    if (int rc = check_shape(k, nmod)) return rc;
    if (m <= 0 || n <= 0 || m > rows_a || n > rows_b || ldc < n || (G && ldg < n)) {
        snprintf(g_err, sizeof(g_err), "ozaki_product: m %d of %d rows, n %d of %d rows, ldc %d", m, rows_a, n, rows_b,
                 ldc);
        return DFTB_ERR_BAD_SIZE;
    }
    if (!A || !B || !C || !work || !err) return DFTB_ERR_NULL;
    if (work_bytes < product_bytes(m, n, nmod) || ((reinterpret_cast<uintptr_t>(work) |
                                                    reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B)) &
                                                   255)) {
        snprintf(g_err, sizeof(g_err), "ozaki_product: workspace of %zu bytes and 256-byte aligned operands needed",
                 product_bytes(m, n, nmod));
        return DFTB_ERR_WORKSPACE;
    }
    if (init_host()) return DFTB_ERR_CUDA;
    return product(m, n, k, nmod, reinterpret_cast<const uint8_t *>(A), rows_a, reinterpret_cast<const uint8_t *>(B),
                   rows_b, alpha, G, ldg, beta, C, ldc, reinterpret_cast<int8_t *>(work), err,
                   reinterpret_cast<cudaStream_t>(stream));
}

size_t dftb_ozaki_workspace_size(int m, int n, int k, int nmod) {
    if (m <= 0 || n <= 0 || ozk::check_shape(k, nmod) != DFTB_OK) return 0;
    return ozk::operand_layout(m, k, nmod).total + ozk::operand_layout(n, k, nmod).total +
           ozk::product_bytes(m, n, nmod);
}

int dftb_ozaki_dgemm(int transa, int transb, int m, int n, int k, double alpha, const double *A, int lda,
                     const double *B, int ldb, double beta, double *C, int ldc, int nmod, void *work,
                     size_t work_bytes, int *err, void *stream) {
    using namespace ozk;
    if (int rc = check_shape(k, nmod)) return rc;
    if (m <= 0 || n <= 0) return DFTB_ERR_BAD_SIZE;
    if (!A || !B || !C || !work || !err) return DFTB_ERR_NULL;
    if (lda < (transa ? m : k) || ldb < (transb ? k : n) || ldc < n) {
        snprintf(g_err, sizeof(g_err), "ozaki_dgemm: leading dimension too small");
        return DFTB_ERR_BAD_SIZE;
    }
    const size_t need = dftb_ozaki_workspace_size(m, n, k, nmod);
    if (work_bytes < need || (reinterpret_cast<uintptr_t>(work) & 255)) {
        snprintf(g_err, sizeof(g_err), "ozaki_dgemm: workspace of %zu bytes (256-byte aligned) needed", need);
        return DFTB_ERR_WORKSPACE;
    }
    if (init_host()) return DFTB_ERR_CUDA;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    uint8_t *w = reinterpret_cast<uint8_t *>(work);
    uint8_t *opA = w, *opB = w + operand_layout(m, k, nmod).total;
    int8_t *RC = reinterpret_cast<int8_t *>(opB + operand_layout(n, k, nmod).total);
    // op(A)(r, k) = transa ? A[k][r] : A[r][k];  op(B)^T(r, k) = op(B)(k, r) = transb ? B[r][k] : B[k][r]
    int rc = prepare(transa ? 1 : 0, m, k, A, lda, nmod, opA, m, 0, st);
    if (rc == DFTB_OK) rc = prepare(transb ? 0 : 1, n, k, B, ldb, nmod, opB, n, 0, st);
    if (rc == DFTB_OK) rc = product(m, n, k, nmod, opA, m, opB, n, alpha, nullptr, 0, beta, C, ldc, RC, err, st);
    return rc;
}

}  // extern "C"
