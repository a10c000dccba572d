// Split-precision BF16 GEMM on the 5th-generation tensor cores (tcgen05) of B200.
//
//   C(m, n) = alpha * sum_s sum_k A_s(m, k) B_s(n, k)          (FP32 accumulation in TMEM)
//
// with up to three (A_s, B_s) operand pairs ("segments") that share M, N, K.
// Splitting an FP32 operand X into BF16 parts X = X_hi + X_lo and summing the
// segments (A_hi,B_hi), (A_hi,B_lo), (A_lo,B_hi) reproduces the FP32 product to
// ~2^-16 relative error at three BF16 tensor-core passes.
//
// Operands are K-major row-major BF16 matrices (A: M x K, B: N x K, leading
// dimensions multiples of 8 elements, 16-byte aligned base).  The epilogue can
//   * multiply elementwise by an FP32 matrix G (the AO-expanded gamma^lr),
//   * store FP32 C,
//   * store the result as a BF16 hi/lo pair, row-major and/or transposed
//     (the transposed store is coalesced across a warp).
//
// Structure per CTA (320 threads, 128 x 128 or 128 x 256 output tiles; pairs of CTAs: 256 x 256):
//   warp 0 lane 0 : TMA producer, ring of operand tiles, mbarrier::complete_tx completion;
//   warp 1 lane 0 : issues tcgen05.mma into one of two TMEM accumulators; tcgen05.commit frees ring slots and finally
//                   signals the epilogue;
//   warps 2..9    : epilogue, tcgen05.ld 32x32b of their 32 TMEM lanes, under the next tile's MMAs.
// Every mbarrier wait is bounded; on timeout the kernel records an error
// code, stops issuing work, drains the copies it started and releases TMEM.

#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

#include <mutex>

#include "dftbaby_b200.h"
#include "tcgen05.cuh"

namespace tcg {

using namespace tc5;

constexpr int BM = 128, BN = 128, BK = 64;
// segment mode: one (A, B) tile pair per stage, 4 stages;
// shared-split mode: A_hi, A_lo, B_hi, B_lo per stage (three MMAs reuse them), 3 stages
// Row-chunk moves of the epilogue: 16 consecutive elements of one row, as 16- or 8-byte words
// when the address is aligned and the chunk is whole, element by element otherwise.
__device__ __forceinline__ void load_row16(const float *src, int n, float out[16]) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(src);
    if (n == 16 && (a & 15) == 0) {
        const float4 *s4 = reinterpret_cast<const float4 *>(src);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float4 t = s4[q];
            out[4 * q] = t.x;
            out[4 * q + 1] = t.y;
            out[4 * q + 2] = t.z;
            out[4 * q + 3] = t.w;
        }
    } else if (n == 16 && (a & 7) == 0) {
        const float2 *s2 = reinterpret_cast<const float2 *>(src);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const float2 t = s2[q];
            out[2 * q] = t.x;
            out[2 * q + 1] = t.y;
        }
    } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) out[j] = j < n ? src[j] : 0.0f;
    }
}

// Eight epilogue warps, two per TMEM lane quarter with every other 32-column chunk each: the epilogues with a Hadamard
// factor or a transposed output are instruction-bound, and with four warps they outlasted the next tile's MMAs (a dense
// layer of 65536 x 256: 50 us with four warps, 32 us with eight).
constexpr int EPI_WARPS = 8, EPI_THREADS = 32 * EPI_WARPS, THREADS = 64 + EPI_THREADS;
// BF16 output staging: per epilogue warp a 32 x 32 block (row-major or transposed, hi, then lo), rows padded to 40
// elements (80 B, a multiple of 16 B for the 16-byte reads), so that a store instruction writes eight whole 64-byte
// pieces instead of 16 bytes of 32 rows (the exchange's W 83 -> 77 us, N 556 -> 522 us).
constexpr int TPITCH = 40;
constexpr int TSTAGE_BYTES = EPI_WARPS * 32 * TPITCH * 2;

template <bool SPLIT, bool WIDE = false, bool PAIR = false> struct Cfg {
    // 128 x 128 output tiles with 64-element K blocks (128-byte swizzle); WIDE (split mode only): 128 x 256
    // tiles with 32-element K blocks (64-byte swizzle), so four stages of A_hi, A_lo, B_hi, B_lo fit and a
    // stage carries the same MMA work with a quarter fewer operand bytes.  (128 x 256 tiles with 64-element
    // blocks leave room for two stages only, which measured slower.)  PAIR (WIDE only): 256 x 256 tiles of a
    // CTA pair, each CTA holding half the rows of A and of B.
    static constexpr int BMX = PAIR ? 2 * BM : BM;
    static constexpr int BNX = WIDE ? 256 : 128;
    static constexpr int BKX = WIDE && !PAIR ? 32 : BK;
    static constexpr int KU = WIDE ? 32 : BK;  // K ranges (split-K) come in multiples of this
    static constexpr int TILE_AX = BM * BKX * 2;
    static constexpr int TILE_BX = (PAIR ? BNX / 2 : BNX) * BKX * 2;
    static constexpr int STAGES = PAIR ? 3 : (WIDE ? 4 : (SPLIT ? 3 : 4));
    static constexpr int STAGE_BYTES = SPLIT ? 2 * (TILE_AX + TILE_BX) : TILE_AX + TILE_BX;
    static constexpr int SMEM_BYTES =
        STAGES * STAGE_BYTES + TSTAGE_BYTES + 1024 /* alignment slack */ + 256 /* barriers */;
    static constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BNX >> 3) << 17) |
                                      ((uint32_t)(BMX >> 4) << 24);
};

struct Maps {
    CUtensorMap a[3];
    CUtensorMap b[3];
};

struct Params {
    int M, N, K, nseg;
    int ksplit;  // K ranges per output tile (gridDim.z); > 1 accumulates C with atomics
    float alpha;
    const float *G;
    long long ldg;
    float *C;
    long long ldc;
    __nv_bfloat16 *Ohi, *Olo;  // row-major hi/lo output (ld = ldo)
    long long ldo;
    __nv_bfloat16 *Thi, *Tlo;  // transposed hi/lo output: T(n, m) (ld = ldt)
    long long ldt;
    int *err;  // device error word (0 = ok)
    // dense layer (MLP): relu(v + bias) or v o (mask > 0), rounded to Ohi and Thi; colsum += column sums of the
    // unrounded values
    const float *bias;
    const __nv_bfloat16 *mask;
    long long ldm;
    float *colsum;
};

// Sums over the warp's 32 lanes of 32 values per lane: lane q returns the sum of every lane's v[q] (halving the values
// with each exchange: 31 shuffles, where 32 separate reductions take 160).
__device__ __forceinline__ float warp_column_sums(float v[32]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int half = 16; half > 0; half >>= 1) {
        const bool up = (lane & half) != 0;
#pragma unroll
        for (int q = 0; q < half; ++q) {
            const float send = up ? v[q] : v[q + half], keep = up ? v[q + half] : v[q];
            v[q] = keep + __shfl_xor_sync(0xffffffffu, send, half);
        }
    }
    return v[0];
}

// UMMA shared-memory descriptor for K-major rows of 64 B with 64-byte swizzle: 8-row groups 512 B apart
__device__ __forceinline__ uint64_t smem_desc_k64(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFF) >> 4);  // start address
    d |= (uint64_t)1 << 16;                    // leading byte offset (unused for swizzled K-major)
    d |= (uint64_t)(512 >> 4) << 32;           // stride byte offset
    d |= (uint64_t)1 << 46;                    // descriptor version
    d |= (uint64_t)4 << 61;                    // SWIZZLE_64B
    return d;
}

template <bool WIDE>
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr) {
    return WIDE ? smem_desc_k64(saddr) : smem_desc_k128(saddr);
}

// instruction descriptor: D = F32, A = B = BF16, both K-major, M = 128, N = 128
constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) |
                            ((uint32_t)(BM >> 4) << 24);

__device__ __forceinline__ void umma_bf16(uint32_t tmem_c, uint64_t da, uint64_t db, uint32_t accumulate,
                                          uint32_t idesc = kIdesc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_c),
        "l"(da), "l"(db), "r"(idesc), "r"(accumulate));
}

__device__ __forceinline__ void umma_bf16_pair(uint32_t tmem_c, uint64_t da, uint64_t db, uint32_t accumulate,
                                               uint32_t idesc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_c),
        "l"(da), "l"(db), "r"(idesc), "r"(accumulate));
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float *v) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// 32 consecutive FP32 accumulator columns of this warp's 32 TMEM lanes
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float *v) {
    uint32_t r[32];
    tmem_ld32_raw(taddr, r);
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// Output tile t of a launch: tiles run M-fastest, then N, then the K range (split-K index), so the CTAs working at one
// time share B tiles and the A operand stays in L2.
struct TileCoords {
    int m0, n0, k0, kend, kblocks;  // kblocks of bkx elements cover k0 .. kend
};

// Pair tiles of tall outputs run in bands of BAND tile columns, N-fastest, so that the tiles at work at one time (74) span
// about as many rows as columns and touch little of both operands (33 x 33 tiles M-fastest send all 41 MB of A past the
// outputs' stream in every round).
// B200, N 8292 x 8292 x 1225: DRAM reads 883 -> 640 MB, 452 -> 427 us; the products' order is unchanged.
constexpr int BAND = 8, BAND_ROWS = 16;

// kper: units of ku elements in a K range
__device__ __forceinline__ TileCoords tile_coords(bool bands, int t, int mt, int nt, int bmx, int bnx, int bkx, int ku, int kper, int K) {
    TileCoords c;
    const int kr = t / (mt * nt), u = t % (mt * nt);
    int mi = u % mt, ni = u / mt;
    if (bands && mt > BAND_ROWS) {
        const int b = u / (mt * BAND), v = u - b * mt * BAND, width = min(BAND, nt - b * BAND);
        mi = v / width;
        ni = b * BAND + v % width;
    }
    c.m0 = mi * bmx;
    c.n0 = ni * bnx;
    c.k0 = kr * kper * ku;
    c.kend = min(K, c.k0 + kper * ku);
    c.kblocks = max(0, (c.kend - c.k0 + bkx - 1) / bkx);
    return c;
}

// Persistent kernel: one CTA per SM walks the tiles t = blockIdx.x, blockIdx.x + gridDim.x, ...
//   warp 0 lane 0 : TMA producer over the operand ring (continues across tiles);
//   warp 1 lane 0 : tcgen05.mma issuer into one of two 128-column TMEM accumulators
//                   (tile j uses accumulator j % 2);
//   warps 2..9    : epilogue of tile j while the MMAs of tile j + 1 run; warp w reads TMEM
//                   lanes 32 (w % 4) .. 32 (w % 4) + 31, every other 32-column chunk.
// Barriers: full/empty per ring slot, tfull (MMA -> epilogue, tcgen05.commit) and tempty
// (epilogue -> MMA, 256 arrivals) per accumulator.  Every wait is bounded.
// MLP (segment mode): the epilogue of a dense layer of the pair-scoring network, forward (bias and ReLU) or backward
// (ReLU mask and bias gradient), instead of an FP32 result that another kernel would read again.  B200, 65536 samples x
// 256 units: product and bias_relu 32 + 46 us, product and relu_backward 32 + 80 us; here 25 to 40 us.
// PAIR (clusters of two): a 128 x 256 split tile makes each SM read 12 KiB of operands per MMA of 128 cycles from shared
// memory while TMA writes 8 KiB, 160 of the 128 bytes a cycle that it moves, and all of B crosses the L2 for every 128 rows
// of A.  In cta_group::2 each CTA reads and is sent half of B: 8 KiB and 5.3 KiB.  The even CTA issues the MMAs of both; its
// full (bytes of both CTAs) and tempty barriers count for the pair, empty and tfull are committed to both.  The K order of an
// element is that of the other tiles, so the results are the same bits.  B200, the exchange's shapes, us without and with:
// W 8292 x 1225 x 1225 77 -> 71, N 8292 x 8292 x 1225 (Hadamard, both outputs) 514 -> 427, P 1225 x 16640 x 8292 723 -> 675
// (1.50 PFLOP/s), K 2450 x 1225 x 8292 164 -> 147.
template <bool SPLIT, bool WIDE, bool MLP = false, bool PAIR = false>
__global__ void __launch_bounds__(THREADS, 1) gemm_kernel(const __grid_constant__ Maps maps, const Params p) {
    using C = Cfg<SPLIT, WIDE, PAIR>;
    constexpr int STAGES = C::STAGES, STAGE_BYTES = C::STAGE_BYTES;
    constexpr int BMX = C::BMX, BNX = C::BNX, TILE_BX = C::TILE_BX, TILE_AX = C::TILE_AX, BKX = C::BKX;
    constexpr uint32_t IDESC = C::IDESC;
    static_assert(BNX % 32 == 0 && (!WIDE || SPLIT), "tile columns come in 32-column chunks; WIDE is split-only");
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    __nv_bfloat16 *tstage = reinterpret_cast<__nv_bfloat16 *>(smem + STAGES * STAGE_BYTES);
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + STAGES * STAGE_BYTES + TSTAGE_BYTES);
    uint64_t *empty = full + STAGES;
    uint64_t *tfull = empty + STAGES;
    uint64_t *tempty = tfull + 2;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(tempty + 2);
    int *abort_flag = reinterpret_cast<int *>(tmem_slot + 1);

    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const uint32_t rank = PAIR ? cluster_rank() : 0;
    const int tile0 = PAIR ? blockIdx.x / 2 : blockIdx.x, tstep = PAIR ? gridDim.x / 2 : gridDim.x;
    const int mt = (p.M + BMX - 1) / BMX, nt = (p.N + BNX - 1) / BNX;
    const int ntiles = mt * nt * p.ksplit;
    const int kblocks_all = (p.K + C::KU - 1) / C::KU;
    const int kper = (kblocks_all + p.ksplit - 1) / p.ksplit;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(&tfull[a], 1);
            mbar_init(&tempty[a], PAIR ? 2 * EPI_WARPS : EPI_THREADS);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncwarp();
    if (warp == 0) {
        // two accumulators of BNX columns (128 lanes x 2 BNX FP32)
        if constexpr (PAIR) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                         "r"(2 * BNX));
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                         "r"(2 * BNX));
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
        }
    }
    __syncthreads();
    if constexpr (PAIR) {
        __syncwarp();
        cluster_sync();  // both CTAs' barriers exist before either signals the other's
    }
    auto wait = [](uint64_t *bar, uint32_t parity) { return PAIR ? mbar_wait_cluster(bar, parity) : mbar_wait(bar, parity); };
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            // ---------------- TMA producer
            int it = 0;  // copies issued (ring position)
            bool stop = false;
            for (int t = tile0; t < ntiles && !stop; t += tstep) {
                const TileCoords tc = tile_coords(PAIR, t, mt, nt, BMX, BNX, BKX, C::KU, kper, p.K);
                const int total = SPLIT ? tc.kblocks : tc.kblocks * p.nseg;
                for (int i = 0; i < total; ++i) {
                    const int s = it % STAGES;
                    if (it >= STAGES && !wait(&empty[s], ((it / STAGES) - 1) & 1)) {
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
                    if (!PAIR) mbar_expect_tx(&full[s], STAGE_BYTES);
                    if constexpr (PAIR) {
                        // this CTA's halves; the even CTA's barrier counts the bytes of both
                        const int kx = tc.k0 + i * BKX, ya = tc.m0 + (int)rank * BM, yb = tc.n0 + (int)rank * (BNX / 2);
                        if (rank == 0) mbar_expect_tx(&full[s], 2 * STAGE_BYTES);
                        const uint32_t bar = map_cta(&full[s], 0);
                        tma_load_2d_pair(sa, &maps.a[0], bar, kx, ya);
                        tma_load_2d_pair(sa + TILE_AX, &maps.a[1], bar, kx, ya);
                        tma_load_2d_pair(sa + 2 * TILE_AX, &maps.b[0], bar, kx, yb);
                        tma_load_2d_pair(sa + 2 * TILE_AX + TILE_BX, &maps.b[1], bar, kx, yb);
                    } else if (SPLIT) {
                        // stage layout: A_hi | A_lo | B_hi | B_lo
                        const int kx = tc.k0 + i * BKX;
                        tma_load_2d(sa, &maps.a[0], &full[s], kx, tc.m0);
                        tma_load_2d(sa + TILE_AX, &maps.a[1], &full[s], kx, tc.m0);
                        tma_load_2d(sa + 2 * TILE_AX, &maps.b[0], &full[s], kx, tc.n0);
                        tma_load_2d(sa + 2 * TILE_AX + TILE_BX, &maps.b[1], &full[s], kx, tc.n0);
                    } else {
                        const int seg = i / tc.kblocks, kx = tc.k0 + i % tc.kblocks * BKX;
                        tma_load_2d(sa, &maps.a[seg], &full[s], kx, tc.m0);
                        tma_load_2d(sa + TILE_AX, &maps.b[seg], &full[s], kx, tc.n0);
                    }
                    ++it;
                }
            }
            // drain: wait (bounded) until every copy that was started has landed
            // (pairs: until the MMAs have read it, which both CTAs see)
            for (int j = max(0, it - STAGES); j < it; ++j) wait(PAIR ? &empty[j % STAGES] : &full[j % STAGES], (j / STAGES) & 1);
        }
    } else if (warp == 1) {
        if (lane == 0 && rank == 0) {
            // ---------------- MMA issuer (of both CTAs)
            int it = 0, j = 0;
            bool stop = false;
            for (int t = tile0; t < ntiles && !stop; t += tstep, ++j) {
                const TileCoords tc = tile_coords(PAIR, t, mt, nt, BMX, BNX, BKX, C::KU, kper, p.K);
                const int total = SPLIT ? tc.kblocks : tc.kblocks * p.nseg;
                const int acc = j & 1;
                const uint32_t tacc = tmem + (uint32_t)(acc * BNX);
                if (j >= 2 && !wait(&tempty[acc], ((j >> 1) - 1) & 1)) {
                    atomicExch(p.err, 4);
                    *(volatile int *)abort_flag = 1;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                for (int i = 0; i < total; ++i) {
                    const int s = it % STAGES;
                    if (!wait(&full[s], (it / STAGES) & 1)) {
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
                    const uint32_t sa = smem_u32(smem + s * STAGE_BYTES);
                    if constexpr (PAIR) {
                        const uint32_t sal = sa + TILE_AX, sb = sa + 2 * TILE_AX, sbl = sb + TILE_BX;
                        const int ks = min(BKX / 16, (tc.kend - tc.k0 - i * BKX + 15) / 16);  // none past the K range
                        for (int k = 0; k < ks; ++k) {
                            const uint32_t o = k * 32;
                            umma_bf16_pair(tacc, smem_desc_k128(sa + o), smem_desc_k128(sb + o), (i > 0 || k > 0) ? 1u : 0u,
                                           IDESC);
                            umma_bf16_pair(tacc, smem_desc_k128(sa + o), smem_desc_k128(sbl + o), 1u, IDESC);
                            umma_bf16_pair(tacc, smem_desc_k128(sal + o), smem_desc_k128(sb + o), 1u, IDESC);
                        }
                    } else if (SPLIT) {
                        const uint32_t sal = sa + TILE_AX, sb = sa + 2 * TILE_AX, sbl = sb + TILE_BX;
#pragma unroll
                        for (int k = 0; k < BKX / 16; ++k) {
                            // 16 BF16 = 32 bytes along K per instruction, inside the swizzle atom
                            const uint32_t o = k * 32;
                            umma_bf16(tacc, smem_desc<WIDE>(sa + o), smem_desc<WIDE>(sb + o),
                                      (i > 0 || k > 0) ? 1u : 0u, IDESC);
                            umma_bf16(tacc, smem_desc<WIDE>(sa + o), smem_desc<WIDE>(sbl + o), 1u, IDESC);
                            umma_bf16(tacc, smem_desc<WIDE>(sal + o), smem_desc<WIDE>(sb + o), 1u, IDESC);
                        }
                    } else {
                        const uint32_t sb = sa + TILE_AX;
#pragma unroll
                        for (int k = 0; k < BKX / 16; ++k) {
                            // advance 16 BF16 = 32 bytes along K inside the 128-byte swizzle atom
                            umma_bf16(tacc, smem_desc_k128(sa + k * 32), smem_desc_k128(sb + k * 32),
                                      (i > 0 || k > 0) ? 1u : 0u);
                        }
                    }
                    if constexpr (PAIR)
                        umma_commit_pair(&empty[s]);
                    else
                        umma_commit(&empty[s]);  // slot s may be refilled once these MMAs have read it
                    ++it;
                }
                if constexpr (PAIR)
                    umma_commit_pair(&tfull[acc]);
                else
                    umma_commit(&tfull[acc]);  // accumulator complete (or abandoned) -> epilogue
            }
        }
    } else {
        // ---------------- epilogue (warps 2..9, 256 threads)
        const int rq = warp & 3;  // TMEM lane quarter this warp may access
        const int rloc = rq * 32 + lane;
        const int chunk0 = 32 * ((warp - 2) >> 2);  // this warp's chunks start here, 64 columns apart
        __nv_bfloat16 *sh = tstage + (warp - 2) * (32 * TPITCH);
        // writes the staged 32 x 32 block to D rows r0 .., columns c0 .. (inside rows x cols)
        auto write_block = [&](__nv_bfloat16 *D, long long ld, int r0, int c0, int rows, int cols) {
            __syncwarp();
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int rl = q * 8 + (lane >> 2), part = lane & 3;
                const int r = r0 + rl, c = c0 + part * 8, nv = min(8, cols - c);
                if (r < rows && nv > 0) {
                    const __nv_bfloat16 *src = sh + rl * TPITCH + part * 8;
                    __nv_bfloat16 *dst = D + (long long)r * ld + c;
                    if (nv == 8 && (reinterpret_cast<uintptr_t>(dst) & 15) == 0)
                        *reinterpret_cast<uint4 *>(dst) = *reinterpret_cast<const uint4 *>(src);
                    else
                        for (int e = 0; e < nv; ++e) dst[e] = src[e];
                }
            }
            __syncwarp();
        };
        // this warp's block of BF16 values (a row per lane) to the row-major output O and the transposed one T
        auto write_bf16 = [&](const __nv_bfloat16 *x, __nv_bfloat16 *O, __nv_bfloat16 *T, int row0, int col0) {
            if (O) {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    uint32_t w[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const __nv_bfloat162 pr = __halves2bfloat162(x[8 * q + 2 * e], x[8 * q + 2 * e + 1]);
                        w[e] = *reinterpret_cast<const uint32_t *>(&pr);
                    }
                    *reinterpret_cast<uint4 *>(sh + lane * TPITCH + 8 * q) = make_uint4(w[0], w[1], w[2], w[3]);
                }
                write_block(O, p.ldo, row0, col0, p.M, p.N);
            }
            if (T) {
#pragma unroll
                for (int q = 0; q < 32; ++q) sh[q * TPITCH + lane] = x[q];
                write_block(T, p.ldt, col0, row0, p.N, p.M);
            }
        };
        // this warp's block of FP32 values (a row per lane) to C, 16 columns at a time through the same staging rows: 64-byte
        // pieces of eight rows a store, or of two where rows are off the 16-byte grid.  (16 bytes of 32 rows a store, by eight
        // warps at a time, took more: 8292 x 8292 x 1225 on 128 x 128 tiles 679 us, 2312 x 8252 x 44 45 us.)
        const bool vec_c = ((reinterpret_cast<uintptr_t>(p.C) | (uintptr_t)p.ldc * sizeof(float)) & 15) == 0;
        auto write_f32 = [&](const float *x, int row0, int col0) {
            float *sf = reinterpret_cast<float *>(sh);
            constexpr int PITCH = TPITCH / 2;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    *reinterpret_cast<float4 *>(sf + lane * PITCH + 4 * q) =
                        make_float4(x[16 * h + 4 * q], x[16 * h + 4 * q + 1], x[16 * h + 4 * q + 2], x[16 * h + 4 * q + 3]);
                __syncwarp();
                if (vec_c && p.N - col0 >= 32) {
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int rl = q * 8 + (lane >> 2), r = row0 + rl, cl = 4 * (lane & 3);
                        if (r < p.M)
                            *reinterpret_cast<float4 *>(p.C + (long long)r * p.ldc + col0 + 16 * h + cl) =
                                *reinterpret_cast<const float4 *>(sf + rl * PITCH + cl);
                    }
                } else {
                    const int cl = lane & 15, c = col0 + 16 * h + cl;
#pragma unroll
                    for (int q = 0; q < 16; ++q) {
                        const int rl = q * 2 + (lane >> 4), r = row0 + rl;
                        if (r < p.M && c < p.N) p.C[(long long)r * p.ldc + c] = sf[rl * PITCH + cl];
                    }
                }
                __syncwarp();
            }
        };
        int j = 0;
        for (int t = tile0; t < ntiles; t += tstep, ++j) {
            const TileCoords tc = tile_coords(PAIR, t, mt, nt, BMX, BNX, BKX, C::KU, kper, p.K);
            const int total = SPLIT ? tc.kblocks : tc.kblocks * p.nseg;
            const int acc = j & 1;
            const int m0 = tc.m0 + (int)rank * BM, n0 = tc.n0;
            const int row = m0 + rloc;
            if (p.G && p.ksplit == 1 && row < p.M) {
                // pull this tile's G row into L2 while its MMAs run (128-byte lines, inside the matrix)
                const float *g = p.G + (long long)row * p.ldg + n0;
                const int ncols = min(BNX, p.N - n0);
                for (int c = chunk0; c < ncols; c += 64) asm volatile("prefetch.global.L2 [%0];" ::"l"(g + c));
            }
            const float *bias_s = MLP && p.bias ? p.bias + n0 : nullptr;
            const bool ok = __all_sync(0xffffffffu, wait(&tfull[acc], (j >> 1) & 1) ? 1 : 0) != 0;
            if (!ok && lane == 0) atomicExch(p.err, 3);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const bool live = ok && !*(volatile int *)abort_flag && total > 0;  // warp-uniform
            for (int c0 = chunk0; c0 < BNX; c0 += 64) {
                float v[32];
                tmem_ld32(tmem + ((uint32_t)(rq * 32) << 16) + (uint32_t)(acc * BNX + c0), v);
                const int col0 = n0 + c0;
                if constexpr (MLP) {
                    const int ncol = min(32, p.N - col0);
                    const bool in = live && row < p.M && ncol > 0;
                    if (p.bias) {
                        // lane q holds the bias of column q; one shuffle each instead of one load each
                        const float bl = lane < ncol ? __ldg(bias_s + c0 + lane) : 0.0f;
#pragma unroll
                        for (int q = 0; q < 32; ++q) v[q] = fmaxf(v[q] + __shfl_sync(0xffffffffu, bl, q), 0.0f);
                        if (!in || ncol < 32) {
#pragma unroll
                            for (int q = 0; q < 32; ++q)
                                if (!in || q >= ncol) v[q] = 0.0f;
                        }
                    } else {
                        const __nv_bfloat16 *mk = p.mask + (long long)row * p.ldm + col0;
                        if (in && ncol == 32 && (reinterpret_cast<uintptr_t>(mk) & 15) == 0) {
                            uint32_t m[16];
#pragma unroll
                            for (int q = 0; q < 4; ++q)
                                *reinterpret_cast<uint4 *>(m + 4 * q) = reinterpret_cast<const uint4 *>(mk)[q];
#pragma unroll
                            for (int q = 0; q < 16; ++q) {  // a bf16 is above zero if its sign is clear and it is not zero
                                if ((int16_t)(m[q] & 0xffff) <= 0) v[2 * q] = 0.0f;
                                if ((int16_t)(m[q] >> 16) <= 0) v[2 * q + 1] = 0.0f;
                            }
                        } else {
#pragma unroll
                            for (int q = 0; q < 32; ++q)
                                if (!(in && q < ncol && __bfloat162float(mk[q]) > 0.0f)) v[q] = 0.0f;
                        }
                    }
                    __nv_bfloat16 hi[32];
#pragma unroll
                    for (int q = 0; q < 32; ++q) hi[q] = __float2bfloat16_rn(v[q]);
                    if (live && ncol > 0) write_bf16(hi, p.Ohi, p.Thi, m0 + rq * 32, col0);
                    if (p.colsum) {
                        const float sum = warp_column_sums(v);
                        if (live && lane < ncol) atomicAdd(p.colsum + col0 + lane, sum);
                    }
                    continue;
                }
                if (live && row < p.M && col0 < p.N) {
                    const int ncol = min(32, p.N - col0);
                    if (p.ksplit > 1) {  // partial sums over this tile's K range
                        float *c = &p.C[(long long)row * p.ldc + col0];
                        if (ncol == 32 && (reinterpret_cast<uintptr_t>(c) & 15) == 0) {
#pragma unroll
                            for (int q = 0; q < 32; q += 4)  // four elements per reduction where the row is aligned
                                atomicAdd(reinterpret_cast<float4 *>(c + q),
                                          make_float4(p.alpha * v[q], p.alpha * v[q + 1], p.alpha * v[q + 2],
                                                      p.alpha * v[q + 3]));
                        } else {
#pragma unroll
                            for (int q = 0; q < 32; ++q)
                                if (q < ncol) atomicAdd(c + q, p.alpha * v[q]);
                        }
                    } else {
                        const int n1 = min(16, ncol), n2 = ncol - 16;  // the two 16-column halves (n2 <= 0: none)
#pragma unroll
                        for (int q = 0; q < 32; ++q) v[q] *= p.alpha;
                        if (p.G) {
                            float g[32];
                            const float *gr = p.G + (long long)row * p.ldg + col0;
                            load_row16(gr, n1, g);
                            if (n2 > 0) load_row16(gr + 16, n2, g + 16);
#pragma unroll
                            for (int q = 0; q < 32; ++q) v[q] *= g[q];
                        }
                    }
                }
                if (p.C && p.ksplit == 1 && live && col0 < p.N) write_f32(v, m0 + rq * 32, col0);
                if ((p.Ohi || p.Thi) && p.ksplit == 1 && live && col0 < p.N) {  // rows beyond M are staged, not written
                    __nv_bfloat16 x[32];
#pragma unroll
                    for (int q = 0; q < 32; ++q) x[q] = __float2bfloat16_rn(v[q]);
                    write_bf16(x, p.Ohi, p.Thi, m0 + rq * 32, col0);
#pragma unroll
                    for (int q = 0; q < 32; ++q) x[q] = __float2bfloat16_rn(v[q] - __bfloat162float(x[q]));
                    write_bf16(x, p.Olo, p.Tlo, m0 + rq * 32, col0);
                }
            }
            // the accumulator has been read: hand it back to the MMA issuer
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            if constexpr (PAIR) {
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster(map_cta(&tempty[acc], 0));
            } else {
                mbar_arrive(&tempty[acc]);
            }
            if (!ok) break;
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if constexpr (PAIR) {
        __syncwarp();
        cluster_sync();  // neither CTA leaves while the other may signal its barriers or its MMAs read its memory
    }
    if (warp == 0) {
        if constexpr (PAIR)
            asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * BNX));
        else
            asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * BNX));
    }
}

// FP32 -> BF16 hi/lo split, with zero padding of the columns [cols, ld)
__global__ void split_kernel(int rows, int cols, const float *X, long long ldx, int transpose, __nv_bfloat16 *hi,
                             __nv_bfloat16 *lo, long long ld) {
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long outr = transpose ? cols : rows;
    if (idx >= outr * ld) return;
    const long long r = idx / ld, c = idx % ld;
    float x = 0.0f;
    const long long inr = transpose ? c : r, inc = transpose ? r : c;
    if (c < (transpose ? rows : cols)) x = X[inr * ldx + inc];
    const __nv_bfloat16 h = __float2bfloat16_rn(x);
    hi[idx] = h;
    lo[idx] = __float2bfloat16_rn(x - __bfloat162float(h));
}

__global__ void split64_kernel(int rows, int cols, const double *X, long long ldx, int transpose, __nv_bfloat16 *hi,
                               __nv_bfloat16 *lo, long long ld, double scale) {
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long outr = transpose ? cols : rows;
    if (idx >= outr * ld) return;
    const long long r = idx / ld, c = idx % ld;
    double x = 0.0;
    const long long inr = transpose ? c : r, inc = transpose ? r : c;
    if (c < (transpose ? rows : cols)) x = scale * X[inr * ldx + inc];
    const float xf = (float)x;
    const __nv_bfloat16 h = __float2bfloat16_rn(xf);
    hi[idx] = h;
    lo[idx] = __float2bfloat16_rn((float)(x - (double)__bfloat162float(h)));
}

// ---------------------------------------------------------------------------- host side
thread_local char g_err[256] = "";
PFN_cuTensorMapEncodeTiled_v12000 g_encode = nullptr;
std::mutex g_mutex;
int *g_errword[64] = {nullptr};

int get_encode() {
    std::lock_guard<std::mutex> lock(g_mutex);
    if (g_encode) return 0;
    cudaDriverEntryPointQueryResult q;
    void *fn = nullptr;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) !=
            cudaSuccess ||
        q != cudaDriverEntryPointSuccess || !fn) {
        snprintf(g_err, sizeof(g_err), "cuTensorMapEncodeTiled unavailable");
        return -1;
    }
    g_encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
    return 0;
}

int make_map(CUtensorMap *map, const void *base, int rows, int cols, long long ld, int box_rows = BM,
             int box_cols = BK) {
    // 2D BF16 tensor: innermost dimension = columns (K), box box_cols x box_rows, zero fill; rows of 64
    // elements (128 B) use the 128-byte swizzle, rows of 32 elements the 64-byte swizzle
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)(ld * 2)};
    cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    const CUtensorMapSwizzle sw = box_cols == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B;
    CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(base), dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        snprintf(g_err, sizeof(g_err), "cuTensorMapEncodeTiled failed (%d): rows %d cols %d ld %lld", (int)r, rows,
                 cols, ld);
        return -1;
    }
    return 0;
}

// 128 x 256 split tiles go to CTA pairs unless less than one round of tiles meets a short K range: there the pair's start
// and finish cost more than its main loop saves.  B200, cold L2, us with pairs and without: 1281 x 1281 x 640 (66 tiles)
// 26.6 and 24.6, 808 x 808 x 202 30.7 and 28.7; 385 x 8192 x 4096 (128 tiles) 78 and 84, 3000 x 3000 x 1000 (288) 49 and
// 51, 2436 x 2436 x 609 (200) 57 and 57, 2450 x 1225 x 8292 in four K ranges 171 and 194.  Nor are they better with few tiles
// (warm L2: 7234 x 131 x 1170, 57 tiles, 28.8 and 26.7, 256 x 8192 x 2000, 64 tiles, 39.0 and 37.6; 2048 x 1280 x 1100, 80
// tiles, 26.7 and 28.8), or where an odd number of row tiles gives the pairs more rounds of the GPU, a round of theirs being
// about a tenth shorter (1104 x 128 x 200000 in 16 K ranges, two rounds of 80 pairs or one of 144 tiles, 377 and 258).
bool pair_tiles(int M, int N, int K, int ksplit) {
    const long long columns = (long long)((N + 255) / 256) * ksplit;
    const long long tiles = (M + BM - 1) / BM * columns, pairs = (M + 2 * BM - 1) / (2 * BM) * columns;
    const long long rounds = (tiles + 147) / 148, pair_rounds = (pairs + 73) / 74;
    return M > BM && (tiles > 148 || (tiles >= 80 && K / ksplit >= 1024)) && 9 * pair_rounds <= 10 * rounds;
}

// mode: 0 segments, 1 split, 2 split with 128 x 256 tiles, 3 segments with a dense layer's epilogue, 4 split with pair tiles
int launch(const Maps &maps, const Params &p, int mode, void *stream) {
    using Kernel = void (*)(const Maps, const Params);
    static const Kernel kernels[5] = {gemm_kernel<false, false>, gemm_kernel<true, false>, gemm_kernel<true, true>,
                                      gemm_kernel<false, false, true>, gemm_kernel<true, true, false, true>};
    static const int smem[5] = {Cfg<false>::SMEM_BYTES, Cfg<true>::SMEM_BYTES, Cfg<true, true>::SMEM_BYTES,
                                Cfg<false>::SMEM_BYTES, Cfg<true, true, true>::SMEM_BYTES};
    static bool attr_set[5][64] = {{false}};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !attr_set[mode][dev]) {
        if (cudaFuncSetAttribute(kernels[mode], cudaFuncAttributeMaxDynamicSharedMemorySize, smem[mode]) != cudaSuccess) {
            snprintf(g_err, sizeof(g_err), "bf16x3_gemm: cannot reserve %d bytes of shared memory", smem[mode]);
            return DFTB_ERR_CUDA;
        }
        if (dev >= 0 && dev < 64) attr_set[mode][dev] = true;
    }
    const int group = mode == 4 ? 2 : 1, bmx = group * BM;  // CTAs that share a tile
    const int bnx = mode == 2 || mode == 4 ? Cfg<true, true>::BNX : Cfg<false>::BNX;
    // persistent launch: one CTA per SM (the shared-memory footprint admits one), each walking tiles
    const long long ntiles = (long long)((p.M + bmx - 1) / bmx) * ((p.N + bnx - 1) / bnx) * p.ksplit;
    if (ntiles > (1LL << 30)) return DFTB_ERR_BAD_SIZE;
    static int sm_count[64] = {0};
    if (dev >= 0 && dev < 64 && sm_count[dev] == 0) {
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
        sm_count[dev] = n;
    }
    const int sms = (dev >= 0 && dev < 64) ? sm_count[dev] : 148;
    const unsigned ctas = group * (unsigned)(ntiles < sms / group ? ntiles : sms / group);
    if (mode == 4) {
        cudaLaunchConfig_t cfg;
        memset(&cfg, 0, sizeof(cfg));
        cfg.gridDim = dim3(ctas);
        cfg.blockDim = dim3(THREADS);
        cfg.dynamicSmemBytes = smem[mode];
        cfg.stream = reinterpret_cast<cudaStream_t>(stream);
        cudaLaunchAttribute attr;
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = 2;
        attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        if (cudaLaunchKernelEx(&cfg, kernels[mode], maps, p) != cudaSuccess) {
            snprintf(g_err, sizeof(g_err), "gemm_kernel: %s", cudaGetErrorString(cudaGetLastError()));
            return DFTB_ERR_CUDA;
        }
    } else {
        kernels[mode]<<<ctas, THREADS, smem[mode], reinterpret_cast<cudaStream_t>(stream)>>>(maps, p);
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        snprintf(g_err, sizeof(g_err), "gemm_kernel: %s", cudaGetErrorString(e));
        return DFTB_ERR_CUDA;
    }
    return DFTB_OK;
}

}  // namespace tcg

extern "C" {

const char *dftb_tc_last_error(void) { return tcg::g_err; }

int dftb_bf16x3_gemm_ex(int M, int N, int K, int nseg, int shared_split, int ksplit, const void *const *A, int lda,
                        const void *const *B, int ldb, float alpha, const float *G, int ldg, float *C, int ldc,
                        void *Ohi, void *Olo, int ldo, void *Thi, void *Tlo, int ldt, int *err, void *stream);

int dftb_bf16x3_gemm(int M, int N, int K, int nseg, const void *const *A, int lda, const void *const *B, int ldb,
                     float alpha, const float *G, int ldg, float *C, int ldc, void *Ohi, void *Olo, int ldo, void *Thi,
                     void *Tlo, int ldt, int *err, void *stream) {
    return dftb_bf16x3_gemm_ex(M, N, K, nseg, 0, 1, A, lda, B, ldb, alpha, G, ldg, C, ldc, Ohi, Olo, ldo, Thi, Tlo,
                               ldt, err, stream);
}

int dftb_bf16x3_gemm_ex(int M, int N, int K, int nseg, int shared_split, int ksplit, const void *const *A, int lda,
                        const void *const *B, int ldb, float alpha, const float *G, int ldg, float *C, int ldc,
                        void *Ohi, void *Olo, int ldo, void *Thi, void *Tlo, int ldt, int *err, void *stream) {
    using namespace tcg;
    if (M <= 0 || N <= 0 || K <= 0 || nseg < 1 || nseg > 3 || ksplit < 1 || ksplit > 64) return DFTB_ERR_BAD_SIZE;
    if (shared_split < 0 || shared_split > 2 || (shared_split && nseg != 2)) {
        snprintf(g_err, sizeof(g_err), "bf16x3_gemm: shared-split mode (1, or 2 for 128 x 256 tiles) takes the pairs "
                 "(A_hi, A_lo), (B_hi, B_lo)");
        return DFTB_ERR_BAD_SIZE;
    }
    if (ksplit > 1 && (!C || G || Ohi || Thi)) {
        snprintf(g_err, sizeof(g_err), "bf16x3_gemm: split-K accumulates into C only (zeroed by the caller)");
        return DFTB_ERR_BAD_SIZE;
    }
    if (lda % 8 || ldb % 8 || lda < K || ldb < K) {
        snprintf(g_err, sizeof(g_err), "bf16x3_gemm: lda/ldb must be multiples of 8 and >= K");
        return DFTB_ERR_BAD_SIZE;
    }
    if (!A || !B || !err) return DFTB_ERR_NULL;
    if ((Ohi && (!Olo || ldo < N)) || (Thi && (!Tlo || ldt < M)) || (C && ldc < N) || (G && ldg < N))
        return DFTB_ERR_BAD_SIZE;
    if (get_encode()) return DFTB_ERR_CUDA;
    Maps maps;
    memset(&maps, 0, sizeof(maps));
    const bool pair = shared_split == 2 && pair_tiles(M, N, K, ksplit);
    for (int s = 0; s < nseg; ++s) {
        if (!A[s] || !B[s]) return DFTB_ERR_NULL;
        if ((reinterpret_cast<uintptr_t>(A[s]) & 15) || (reinterpret_cast<uintptr_t>(B[s]) & 15)) {
            snprintf(g_err, sizeof(g_err), "bf16x3_gemm: operands must be 16-byte aligned");
            return DFTB_ERR_BAD_SIZE;
        }
        const bool wide = shared_split == 2;
        const int bkx = wide && !pair ? Cfg<true, true>::BKX : BK;
        const int bnx = wide && !pair ? Cfg<true, true>::BNX : BN;
        if (make_map(&maps.a[s], A[s], M, K, lda, BM, bkx) || make_map(&maps.b[s], B[s], N, K, ldb, bnx, bkx))
            return DFTB_ERR_CUDA;
    }
    Params p;
    p.M = M;
    p.N = N;
    p.K = K;
    p.nseg = nseg;
    p.ksplit = ksplit;
    p.alpha = alpha;
    p.G = G;
    p.ldg = ldg;
    p.C = C;
    p.ldc = ldc;
    p.Ohi = reinterpret_cast<__nv_bfloat16 *>(Ohi);
    p.Olo = reinterpret_cast<__nv_bfloat16 *>(Olo);
    p.ldo = ldo;
    p.Thi = reinterpret_cast<__nv_bfloat16 *>(Thi);
    p.Tlo = reinterpret_cast<__nv_bfloat16 *>(Tlo);
    p.ldt = ldt;
    p.err = err;
    p.bias = nullptr;
    p.mask = nullptr;
    p.ldm = 0;
    p.colsum = nullptr;
    return tcg::launch(maps, p, pair ? 4 : shared_split, stream);
}

int dftb_mlp_dense(int ns, int nout, int nin, const void *X, int ldx, const void *W, int ldw, const float *bias,
                   const void *mask, int ldm, void *H, int ldh, void *HT, int ldht, float *colsum, int *err,
                   void *stream) {
    using namespace tcg;
    if (ns <= 0 || nout <= 0 || nin <= 0 || ldx % 8 || ldw % 8 || ldx < nin || ldw < nin || (H && ldh < nout) ||
        (HT && ldht < ns) || (mask && ldm < nout)) {
        snprintf(g_err, sizeof(g_err), "mlp_dense: sizes or leading dimensions");
        return DFTB_ERR_BAD_SIZE;
    }
    if (!X || !W || !err || (!bias == !mask) || (!H && !HT)) {
        snprintf(g_err, sizeof(g_err), "mlp_dense: operands, a bias or a mask, and an output");
        return DFTB_ERR_NULL;
    }
    if ((reinterpret_cast<uintptr_t>(X) | reinterpret_cast<uintptr_t>(W)) & 15) {
        snprintf(g_err, sizeof(g_err), "mlp_dense: operands must be 16-byte aligned");
        return DFTB_ERR_BAD_SIZE;
    }
    if (get_encode()) return DFTB_ERR_CUDA;
    Maps maps;
    memset(&maps, 0, sizeof(maps));
    if (make_map(&maps.a[0], X, ns, nin, ldx, BM, BK) || make_map(&maps.b[0], W, nout, nin, ldw, BN, BK))
        return DFTB_ERR_CUDA;
    Params p;
    memset(&p, 0, sizeof(p));
    p.M = ns;
    p.N = nout;
    p.K = nin;
    p.nseg = 1;
    p.ksplit = 1;
    p.alpha = 1.0f;
    p.Ohi = reinterpret_cast<__nv_bfloat16 *>(H);
    p.ldo = ldh;
    p.Thi = reinterpret_cast<__nv_bfloat16 *>(HT);
    p.ldt = ldht;
    p.bias = bias;
    p.mask = reinterpret_cast<const __nv_bfloat16 *>(mask);
    p.ldm = ldm;
    p.colsum = colsum;
    p.err = err;
    return launch(maps, p, 3, stream);
}

int dftb_split_bf16(int rows, int cols, const float *X, int ldx, int transpose, void *hi, void *lo, int ld,
                    void *stream) {
    using namespace tcg;
    if (rows <= 0 || cols <= 0 || ld < (transpose ? rows : cols)) return DFTB_ERR_BAD_SIZE;
    if (!X || !hi || !lo) return DFTB_ERR_NULL;
    const long long n = (long long)(transpose ? cols : rows) * ld;
    split_kernel<<<(unsigned)((n + 255) / 256), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
        rows, cols, X, ldx, transpose, reinterpret_cast<__nv_bfloat16 *>(hi), reinterpret_cast<__nv_bfloat16 *>(lo),
        ld);
    return cudaGetLastError() == cudaSuccess ? DFTB_OK : DFTB_ERR_CUDA;
}

int dftb_split_bf16_f64(int rows, int cols, const double *X, int ldx, int transpose, double scale, void *hi, void *lo,
                        int ld, void *stream) {
    using namespace tcg;
    if (rows <= 0 || cols <= 0 || ld < (transpose ? rows : cols)) return DFTB_ERR_BAD_SIZE;
    if (!X || !hi || !lo) return DFTB_ERR_NULL;
    const long long n = (long long)(transpose ? cols : rows) * ld;
    split64_kernel<<<(unsigned)((n + 255) / 256), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
        rows, cols, X, ldx, transpose, reinterpret_cast<__nv_bfloat16 *>(hi), reinterpret_cast<__nv_bfloat16 *>(lo),
        ld, scale);
    return cudaGetLastError() == cudaSuccess ? DFTB_OK : DFTB_ERR_CUDA;
}

}  // extern "C"
