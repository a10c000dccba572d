// dftbaby_b200: element-wise kernels of the small MLP behind the learned
// Davidson guess and preconditioner correction (no counterpart in DFTBaby).
//
// The network is x(64, zero-padded features) -> 256 -> 256 -> 2 with ReLU.
// Its matrix products run on the tcgen05 tensor cores (dftb_bf16x3_gemm_ex with
// one BF16 segment, FP32 accumulation); the kernels here do everything in
// between: bias + ReLU with BF16 row-major and transposed copies of the
// activations (the transposed copies are the K-major operands of the
// weight-gradient products), the weighted squared-error loss and its gradient,
// the ReLU backward pass with bias-gradient column sums, and Adam on FP32
// master weights with refreshed BF16 copies.  All matrices are row-major.

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include "dftbaby_b200.h"

namespace {

thread_local char g_mlp_err[256] = "";

int mlp_fail(int code, const char *what) {
    snprintf(g_mlp_err, sizeof(g_mlp_err), "%s", what);
    return code;
}

int mlp_check(const char *where) {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        snprintf(g_mlp_err, sizeof(g_mlp_err), "%s: %s", where, cudaGetErrorString(e));
        return DFTB_ERR_CUDA;
    }
    return DFTB_OK;
}

inline cudaStream_t S(void *s) { return reinterpret_cast<cudaStream_t>(s); }

constexpr int TILE = 32;

// H = relu(Z + b) on a 32 x 32 tile (samples x units); H row-major and, when
// HT is given, H^T through a shared-memory transpose so both writes coalesce.
__global__ void bias_relu_kernel(int ns, int nh, const float *__restrict__ Z, int ldz, const float *__restrict__ b,
                                 __nv_bfloat16 *__restrict__ H, int ldh, __nv_bfloat16 *__restrict__ HT, int ldht) {
    __shared__ float tile[TILE][TILE + 1];
    const int s0 = blockIdx.x * TILE, h0 = blockIdx.y * TILE;
    const int tx = threadIdx.x, ty = threadIdx.y;
    for (int r = ty; r < TILE; r += blockDim.y) {
        const int s = s0 + r, h = h0 + tx;
        float v = 0.0f;
        if (s < ns && h < nh) {
            v = fmaxf(Z[(size_t)s * ldz + h] + b[h], 0.0f);
            H[(size_t)s * ldh + h] = __float2bfloat16(v);
        }
        tile[r][tx] = v;
    }
    if (!HT) return;
    __syncthreads();
    for (int r = ty; r < TILE; r += blockDim.y) {
        const int h = h0 + r, s = s0 + tx;
        if (h < nh && s < ns) HT[(size_t)h * ldht + s] = __float2bfloat16(tile[tx][r]);
    }
}

// dZ = G o (H > 0) with the same tiling; db[h] += sum over the tile's samples.
__global__ void relu_backward_kernel(int ns, int nh, const float *__restrict__ G, int ldg,
                                     const __nv_bfloat16 *__restrict__ H, int ldh, __nv_bfloat16 *__restrict__ dZ,
                                     int lddz, __nv_bfloat16 *__restrict__ dZT, int lddzt, float *__restrict__ db) {
    __shared__ float tile[TILE][TILE + 1];
    const int s0 = blockIdx.x * TILE, h0 = blockIdx.y * TILE;
    const int tx = threadIdx.x, ty = threadIdx.y;
    for (int r = ty; r < TILE; r += blockDim.y) {
        const int s = s0 + r, h = h0 + tx;
        float v = 0.0f;
        if (s < ns && h < nh) {
            v = __bfloat162float(H[(size_t)s * ldh + h]) > 0.0f ? G[(size_t)s * ldg + h] : 0.0f;
            if (dZ) dZ[(size_t)s * lddz + h] = __float2bfloat16(v);
        }
        tile[r][tx] = v;
    }
    __syncthreads();
    if (ty == 0 && h0 + tx < nh) {
        float acc = 0.0f;
        for (int r = 0; r < TILE; ++r) acc += tile[r][tx];
        atomicAdd(&db[h0 + tx], acc);
    }
    for (int r = ty; r < TILE; r += blockDim.y) {
        const int h = h0 + r, s = s0 + tx;
        if (h < nh && s < ns) dZT[(size_t)h * lddzt + s] = __float2bfloat16(tile[tx][r]);
    }
}

// Output layer, one thread per sample:
//   y[s][o] = Z[s][o] + b[o];
//   with targets: loss += sum_o wout[o] m[s] (y - t)^2 * inv_norm and
//   dY[s][o] = 2 wout[o] m[s] (y - t) inv_norm (BF16, row-major dYp and rows o of dYT),
//   db[o] += dY[s][o].
__global__ void output_kernel(int ns, int no, const float *__restrict__ Z, int ldz, const float *__restrict__ b,
                              const float *__restrict__ T, const float *__restrict__ m,
                              const float *__restrict__ wout, float inv_norm, float *__restrict__ Y,
                              __nv_bfloat16 *__restrict__ dYp, int lddy, __nv_bfloat16 *__restrict__ dYT, int lddyt,
                              float *__restrict__ db, double *__restrict__ loss) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    double l = 0.0;
    if (s < ns) {
        for (int o = 0; o < no; ++o) {
            const float y = Z[(size_t)s * ldz + o] + b[o];
            Y[(size_t)s * no + o] = y;
            if (T) {
                const float d = y - T[(size_t)s * no + o];
                const float w = wout[o] * m[s];
                l += (double)w * d * d * inv_norm;
                const float g = 2.0f * w * d * inv_norm;
                dYp[(size_t)s * lddy + o] = __float2bfloat16(g);
                dYT[(size_t)o * lddyt + s] = __float2bfloat16(g);
                atomicAdd(&db[o], g);
            }
        }
    }
    if (!T) return;
    for (int off = 16; off > 0; off >>= 1) l += __shfl_xor_sync(0xffffffffu, l, off);
    if ((threadIdx.x & 31) == 0) atomicAdd(loss, l);
}

// Adam (with decoupled weight decay) on FP32 master weights W (rows x cols),
// followed by the BF16 copies Wb (row-major, ldwb) and optionally WbT (transposed, ldwbt).
__global__ void adam_kernel(int rows, int cols, float *__restrict__ W, const float *__restrict__ G,
                            float *__restrict__ mom1, float *__restrict__ mom2, float lr, float beta1, float beta2,
                            float eps, float bc1, float bc2, float wd, __nv_bfloat16 *__restrict__ Wb, int ldwb,
                            __nv_bfloat16 *__restrict__ WbT, int ldwbt) {
    const long long n = (long long)rows * cols;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float g = G[i];
        const float m1 = beta1 * mom1[i] + (1.0f - beta1) * g;
        const float m2 = beta2 * mom2[i] + (1.0f - beta2) * g * g;
        mom1[i] = m1;
        mom2[i] = m2;
        float w = W[i];
        w -= lr * ((m1 / bc1) / (sqrtf(m2 / bc2) + eps) + wd * w);
        W[i] = w;
        const int r = (int)(i / cols), c = (int)(i % cols);
        if (Wb) Wb[(size_t)r * ldwb + c] = __float2bfloat16(w);
        if (WbT) WbT[(size_t)c * ldwbt + r] = __float2bfloat16(w);
    }
}

// Standardised, zero-padded BF16 inputs: X[s][f] = (F[s][f] - mean[f]) / std[f] for s < n, f < nf, else 0, with X (ns x
// fpad) row-major and its transpose for the weight gradient, through a 64 x 64 tile.  msum += sum of the sample weights m
// (in FP64, so that the order of the blocks does not show).
__global__ void __launch_bounds__(256) inputs_kernel(int n, int ns, int nf, int fpad, const float *__restrict__ F,
                                                     int ldf, const float *__restrict__ mean,
                                                     const float *__restrict__ std, __nv_bfloat16 *__restrict__ X,
                                                     int ldx, __nv_bfloat16 *__restrict__ XT, int ldxt,
                                                     const float *__restrict__ m, double *__restrict__ msum) {
    __shared__ __nv_bfloat16 tile[64][66];
    const int s0 = blockIdx.x * 64, f0 = blockIdx.y * 64;
    for (int i = threadIdx.x; i < 64 * 64; i += blockDim.x) {
        const int s = s0 + i / 64, f = f0 + i % 64;
        float v = 0.0f;
        if (s < n && f < nf) v = __fdiv_rn(F[(size_t)s * ldf + f] - mean[f], std[f]);
        const __nv_bfloat16 b = __float2bfloat16(v);
        if (s < ns && f < fpad) X[(size_t)s * ldx + f] = b;
        tile[i / 64][i % 64] = b;
    }
    if (m && blockIdx.y == 0 && threadIdx.x < 32) {
        double w = 0.0;
        for (int s = s0 + threadIdx.x; s < min(n, s0 + 64); s += 32) w += m[s];
        for (int o = 16; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
        if (threadIdx.x == 0) atomicAdd(msum, w);
    }
    if (!XT) return;
    __syncthreads();
    for (int i = threadIdx.x; i < 64 * 64; i += blockDim.x) {
        const int f = f0 + i / 64, s = s0 + i % 64;
        if (s < ns && f < fpad) XT[(size_t)f * ldxt + s] = tile[i % 64][i / 64];
    }
}

// Output layer, forward and backward, over tiles of 64 samples (a thread per two units and half of the samples):
//   y = H W^T + b; with targets: loss, dY = 2 wout m (y - t) / sum(m) (BF16), db, dW = dY^T H,
//   dZ = (dY W) o (H > 0) row-major and transposed, dbz = column sums of dZ.
// With two outputs the products are a dot product and an outer product per sample, so the layer is bound by reading H
// and writing dZ twice; as tensor-core products padded to 64 and 128 columns with separate mask, loss and sum kernels it
// took 430 us for 65536 x 256 (B200), here 50 us.
constexpr int HEAD_S = 64, HEAD_NO = 2;

// NH: the number of units where it is known when compiling (the network's 256), else 0
template <int NH>
__global__ void __launch_bounds__(256) head_kernel(int ns, int n, int nh_, const __nv_bfloat16 *__restrict__ H, int ldh,
                                                   const __nv_bfloat16 *__restrict__ W, int ldw,
                                                   const float *__restrict__ b, const float *__restrict__ T,
                                                   const float *__restrict__ tscale, const float *__restrict__ m,
                                                   float wout0, float wout1, const double *__restrict__ msum,
                                                   float *__restrict__ Y, __nv_bfloat16 *__restrict__ dZ, int lddz,
                                                   __nv_bfloat16 *__restrict__ dZT, int lddzt, float *__restrict__ dW,
                                                   float *__restrict__ db, float *__restrict__ dbz,
                                                   double *__restrict__ loss) {
    extern __shared__ __align__(16) unsigned char head_sm[];
    const int nh = NH ? NH : nh_;
    const int pitch = nh + 8;  // 16 bytes more than a power of two: rows start in different banks
    __nv_bfloat16 *hs = reinterpret_cast<__nv_bfloat16 *>(head_sm);
    float *ws = reinterpret_cast<float *>(head_sm + sizeof(__nv_bfloat16) * HEAD_S * pitch);  // W as FP32
    __shared__ __align__(8) float ys[HEAD_S][HEAD_NO];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    for (int i = tid; i < HEAD_NO * nh; i += 256) ws[i] = __bfloat162float(W[(size_t)(i / nh) * ldw + i % nh]);
    float wl[HEAD_NO][8];  // this lane's eight units in the forward products
#pragma unroll
    for (int e = 0; e < 8; ++e)
#pragma unroll
        for (int o = 0; o < HEAD_NO; ++o)
            wl[o][e] = 8 * lane < nh ? __bfloat162float(W[(size_t)o * ldw + 8 * lane + e]) : 0.0f;
    const double wsum = T ? *msum : 1.0;
    const float inv_norm = (float)(1.0 / (wsum < 1e-30 ? 1e-30 : wsum));  // not a number if a weight is not
    float2 dw0 = make_float2(0.0f, 0.0f), dw1 = dw0, dbh = dw0;  // of units u0 and u0 + 1, for one half of each tile's samples
    const int u0 = 2 * (tid & 127), half = tid >> 7;
    float dbo = 0.0f;  // output tid % 2
    double l = 0.0;
    for (int s0 = blockIdx.x * HEAD_S; s0 < ns; s0 += gridDim.x * HEAD_S) {
        __syncthreads();  // ws is written; the last tile has been read
#pragma unroll 8
        for (int i = tid; i < HEAD_S * (nh / 8); i += 256) {
            const int s = i / (nh / 8), c = i % (nh / 8);
            uint4 v = make_uint4(0, 0, 0, 0);
            if (s0 + s < ns) v = *reinterpret_cast<const uint4 *>(H + (size_t)(s0 + s) * ldh + 8 * c);
            *reinterpret_cast<uint4 *>(hs + s * pitch + 8 * c) = v;
        }
        __syncthreads();
        // y: a warp per sample, eight units per lane
#pragma unroll 2
        for (int s = warp; s < HEAD_S; s += 8) {
            float a0 = 0.0f, a1 = 0.0f;
            if (8 * lane < nh) {
                const uint4 v = *reinterpret_cast<const uint4 *>(hs + s * pitch + 8 * lane);
                const uint32_t hv[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float2 h = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&hv[e]));
                    a0 = fmaf(h.x, wl[0][2 * e], fmaf(h.y, wl[0][2 * e + 1], a0));
                    a1 = fmaf(h.x, wl[1][2 * e], fmaf(h.y, wl[1][2 * e + 1], a1));
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                a0 += __shfl_xor_sync(0xffffffffu, a0, o);
                a1 += __shfl_xor_sync(0xffffffffu, a1, o);
            }
            if (lane < HEAD_NO) ys[s][lane] = (lane == 0 ? a0 : a1) + b[lane];
        }
        __syncthreads();
        if (Y)
            for (int i = tid; i < HEAD_S * HEAD_NO; i += blockDim.x)
                if (s0 + i / HEAD_NO < ns) Y[(size_t)s0 * HEAD_NO + i] = ys[i / HEAD_NO][i % HEAD_NO];
        if (!T) continue;
        // dY in place of y, rounded to BF16 as a tensor-core operand would be
        for (int i = tid; i < HEAD_S * HEAD_NO; i += blockDim.x) {
            const int s = s0 + i / HEAD_NO, o = i % HEAD_NO;
            float g = 0.0f;
            if (s < n) {
                const float d = ys[i / HEAD_NO][o] - __fmul_rn(T[(size_t)s * HEAD_NO + o], tscale[o]);
                const float w = (o ? wout1 : wout0) * m[s];
                l += (double)w * d * d * inv_norm;
                g = 2.0f * w * d * inv_norm;
                dbo += g;
            }
            ys[i / HEAD_NO][o] = __bfloat162float(__float2bfloat16(g));
        }
        __syncthreads();
        if (u0 < nh) {
            const float wx0 = ws[u0], wy0 = ws[u0 + 1], wx1 = ws[nh + u0], wy1 = ws[nh + u0 + 1];
            const int sb = half * (HEAD_S / 2);
#pragma unroll
            for (int sg = sb; sg < sb + HEAD_S / 2; sg += 8) {
                uint32_t zp[8];
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const int s = sg + k;
                    const float2 h = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(hs + s * pitch + u0));
                    const float2 d = *reinterpret_cast<const float2 *>(ys[s]);
                    float2 z;
                    z.x = h.x > 0.0f ? fmaf(d.y, wx1, d.x * wx0) : 0.0f;
                    z.y = h.y > 0.0f ? fmaf(d.y, wy1, d.x * wy0) : 0.0f;
                    dbh.x += z.x;
                    dbh.y += z.y;
                    dw0.x = fmaf(d.x, h.x, dw0.x);
                    dw0.y = fmaf(d.x, h.y, dw0.y);
                    dw1.x = fmaf(d.y, h.x, dw1.x);
                    dw1.y = fmaf(d.y, h.y, dw1.y);
                    const __nv_bfloat162 zb = __float22bfloat162_rn(z);
                    zp[k] = *reinterpret_cast<const uint32_t *>(&zb);
                    if (s0 + s < ns) *reinterpret_cast<uint32_t *>(dZ + (size_t)(s0 + s) * lddz + u0) = zp[k];
                }
#pragma unroll
                for (int e = 0; e < 2; ++e) {  // eight samples of units u0 and u0 + 1 along their rows of dZT
                    const unsigned sel = e ? 0x7632u : 0x5410u;
                    uint32_t w[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k) w[k] = __byte_perm(zp[2 * k], zp[2 * k + 1], sel);
                    __nv_bfloat16 *dst = dZT + (size_t)(u0 + e) * lddzt + s0 + sg;
                    if (s0 + sg + 8 <= ns && (reinterpret_cast<uintptr_t>(dst) & 15) == 0)
                        *reinterpret_cast<uint4 *>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
                    else
                        for (int k = 0; k < 8 && s0 + sg + k < ns; ++k)
                            reinterpret_cast<unsigned short *>(dst)[k] = (unsigned short)(w[k >> 1] >> (16 * (k & 1)));
                }
            }
        }
    }
    if (!T) return;
    if (u0 < nh) {
        atomicAdd(dW + u0, dw0.x);
        atomicAdd(dW + u0 + 1, dw0.y);
        atomicAdd(dW + nh + u0, dw1.x);
        atomicAdd(dW + nh + u0 + 1, dw1.y);
        atomicAdd(dbz + u0, dbh.x);
        atomicAdd(dbz + u0 + 1, dbh.y);
    }
    for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
    for (int o = 16; o > 1; o >>= 1) dbo += __shfl_xor_sync(0xffffffffu, dbo, o);
    if (lane == 0) atomicAdd(loss, l);
    if (lane < HEAD_NO) atomicAdd(db + lane, dbo);
}

}  // namespace

extern "C" {

int dftb_mlp_inputs(int n, int ns, int nf, int fpad, const float *F, int ldf, const float *mean, const float *std,
                    void *X, int ldx, void *XT, int ldxt, const float *m, double *msum, void *stream) {
    if (n < 0 || ns < n || ns <= 0 || nf <= 0 || fpad < nf || ldf < nf || ldx < fpad || (XT && ldxt < ns))
        return mlp_fail(DFTB_ERR_BAD_SIZE, "mlp_inputs: sizes");
    if ((n > 0 && !F) || !mean || !std || !X || (m && !msum)) return mlp_fail(DFTB_ERR_NULL, "mlp_inputs: null");
    inputs_kernel<<<dim3((ns + 63) / 64, (fpad + 63) / 64), 256, 0, S(stream)>>>(
        n, ns, nf, fpad, F, ldf, mean, std, reinterpret_cast<__nv_bfloat16 *>(X), ldx,
        reinterpret_cast<__nv_bfloat16 *>(XT), ldxt, m, msum);
    return mlp_check("inputs_kernel");
}

int dftb_mlp_head(int ns, int n, int nh, const void *H, int ldh, const void *W, int ldw, const float *b, const float *T,
                  const float *tscale, const float *m, float wout0, float wout1, const double *msum, float *Y, void *dZ,
                  int lddz, void *dZT, int lddzt, float *dW, float *db, float *dbz, double *loss, void *stream) {
    if (ns <= 0 || n < 0 || n > ns || nh <= 0 || nh > 256 || nh % 8 || ldh < nh || ldh % 8 || ldw < nh)
        return mlp_fail(DFTB_ERR_BAD_SIZE, "mlp_head: sizes (up to 256 units, a multiple of 8)");
    if (!H || !W || !b || (reinterpret_cast<uintptr_t>(H) & 15)) return mlp_fail(DFTB_ERR_NULL, "mlp_head: operands");
    if (T) {
        if (!tscale || !m || !msum || !dZ || !dZT || !dW || !db || !dbz || !loss)
            return mlp_fail(DFTB_ERR_NULL, "mlp_head: training outputs");
        if (lddz < nh || lddz % 2 || (reinterpret_cast<uintptr_t>(dZ) & 3) || lddzt < ns)
            return mlp_fail(DFTB_ERR_BAD_SIZE, "mlp_head: leading dimensions");
    } else if (!Y) {
        return mlp_fail(DFTB_ERR_NULL, "mlp_head: Y");
    }
    const int tiles = (ns + HEAD_S - 1) / HEAD_S;
    const size_t smem = sizeof(__nv_bfloat16) * HEAD_S * (nh + 8) + sizeof(float) * HEAD_NO * nh;
    const auto kernel = nh == 256 ? head_kernel<256> : head_kernel<0>;
    kernel<<<tiles < 148 * 4 ? tiles : 148 * 4, 256, smem, S(stream)>>>(
        ns, n, nh, reinterpret_cast<const __nv_bfloat16 *>(H), ldh, reinterpret_cast<const __nv_bfloat16 *>(W), ldw, b, T,
        tscale, m, wout0, wout1, msum, Y, reinterpret_cast<__nv_bfloat16 *>(dZ), lddz, reinterpret_cast<__nv_bfloat16 *>(dZT),
        lddzt, dW, db, dbz, loss);
    return mlp_check("head_kernel");
}

const char *dftb_mlp_last_error(void) { return g_mlp_err; }

int dftb_mlp_bias_relu(int ns, int nh, const float *Z, int ldz, const float *b, void *H, int ldh, void *HT, int ldht,
                       void *stream) {
    if (ns <= 0 || nh <= 0 || ldz < nh || ldh < nh || (HT && ldht < ns)) return mlp_fail(DFTB_ERR_BAD_SIZE, "mlp_bias_relu: sizes");
    if (!Z || !b || !H) return mlp_fail(DFTB_ERR_NULL, "mlp_bias_relu: null");
    dim3 grid((ns + TILE - 1) / TILE, (nh + TILE - 1) / TILE);
    bias_relu_kernel<<<grid, dim3(TILE, 8), 0, S(stream)>>>(ns, nh, Z, ldz, b, reinterpret_cast<__nv_bfloat16 *>(H),
                                                           ldh, reinterpret_cast<__nv_bfloat16 *>(HT), ldht);
    return mlp_check("bias_relu_kernel");
}

int dftb_mlp_relu_backward(int ns, int nh, const float *G, int ldg, const void *H, int ldh, void *dZ, int lddz,
                           void *dZT, int lddzt, float *db, void *stream) {
    if (ns <= 0 || nh <= 0 || ldg < nh || ldh < nh || (dZ && lddz < nh) || lddzt < ns)
        return mlp_fail(DFTB_ERR_BAD_SIZE, "mlp_relu_backward: sizes");
    if (!G || !H || !dZT || !db) return mlp_fail(DFTB_ERR_NULL, "mlp_relu_backward: null");
    dim3 grid((ns + TILE - 1) / TILE, (nh + TILE - 1) / TILE);
    relu_backward_kernel<<<grid, dim3(TILE, 8), 0, S(stream)>>>(
        ns, nh, G, ldg, reinterpret_cast<const __nv_bfloat16 *>(H), ldh, reinterpret_cast<__nv_bfloat16 *>(dZ), lddz,
        reinterpret_cast<__nv_bfloat16 *>(dZT), lddzt, db);
    return mlp_check("relu_backward_kernel");
}

int dftb_mlp_output(int ns, int no, const float *Z, int ldz, const float *b, const float *T, const float *m,
                    const float *wout, float inv_norm, float *Y, void *dYp, int lddy, void *dYT, int lddyt, float *db,
                    double *loss, void *stream) {
    if (ns <= 0 || no <= 0 || no > 8 || ldz < no) return mlp_fail(DFTB_ERR_BAD_SIZE, "mlp_output: sizes");
    if (!Z || !b || !Y) return mlp_fail(DFTB_ERR_NULL, "mlp_output: null");
    if (T && (!m || !wout || !dYp || !dYT || !db || !loss || lddy < no || lddyt < ns))
        return mlp_fail(DFTB_ERR_NULL, "mlp_output: training outputs");
    output_kernel<<<(ns + 255) / 256, 256, 0, S(stream)>>>(ns, no, Z, ldz, b, T, m, wout, inv_norm, Y,
                                                           reinterpret_cast<__nv_bfloat16 *>(dYp), lddy,
                                                           reinterpret_cast<__nv_bfloat16 *>(dYT), lddyt, db, loss);
    return mlp_check("output_kernel");
}

int dftb_mlp_adam(int rows, int cols, float *W, const float *G, float *m1, float *m2, float lr, float beta1,
                  float beta2, float eps, int step, float weight_decay, void *Wb, int ldwb, void *WbT, int ldwbt,
                  void *stream) {
    if (rows <= 0 || cols <= 0 || step < 1 || (Wb && ldwb < cols) || (WbT && ldwbt < rows))
        return mlp_fail(DFTB_ERR_BAD_SIZE, "mlp_adam: sizes");
    if (!W || !G || !m1 || !m2) return mlp_fail(DFTB_ERR_NULL, "mlp_adam: null");
    const float bc1 = 1.0f - powf(beta1, (float)step), bc2 = 1.0f - powf(beta2, (float)step);
    const long long n = (long long)rows * cols;
    const int blocks = (int)((n + 255) / 256 < 4096 ? (n + 255) / 256 : 4096);
    adam_kernel<<<blocks, 256, 0, S(stream)>>>(rows, cols, W, G, m1, m2, lr, beta1, beta2, eps, bc1, bc2, weight_decay,
                                               reinterpret_cast<__nv_bfloat16 *>(Wb), ldwb,
                                               reinterpret_cast<__nv_bfloat16 *>(WbT), ldwbt);
    return mlp_check("adam_kernel");
}

}  // extern "C"
