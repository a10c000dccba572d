// Eigen-decomposition of small symmetric FP64 matrices (n <= 128), one CTA per matrix and one launch per batch (no
// counterpart in DFTBaby, which calls LAPACK: DFTB2.py:1086, Solver.py:486, 772).
//
// The SCC of a molecule and the projected problems of the Davidson solver need one small decomposition per iteration.
// A library call is a chain of some 240 dependent launches at these sizes (tridiagonalisation, divide and conquer by
// level, two launches per reflector for the vectors), so it is bound by launch latency: 1.75 ms at n = 102 on B200.
// Here the whole decomposition stays on one SM:
//
//   1. Householder tridiagonalisation with the matrix in registers (thread (warp, lane): rows warp + WARPS r, columns
//      lane + 32 c); two barriers a reflector.
//   2. Divide and conquer (Cuppen 1981) from blocks of one, merging neighbours of width w at all positions at once.
//      Deflation as in Dongarra and Sorensen (1987); roots of the secular equation by the rational interpolation of
//      Li (1993), bracketed, four lanes a root; vectors from the recomputed z of Gu and Eisenstat (1994), which keeps
//      them orthogonal without extended precision; their product with the old vectors by FP64 tensor instructions, a
//      warp owning 8 rows, so that it is done in place.
//   3. The reflectors are applied to the columns, which four lanes each hold in registers; no barriers.
//
// Bound by the latency of its serial steps, not by a unit.  B200, host included, against torch.linalg.eigh: n = 20 0.26
// -> 0.11 ms, 42 0.70 -> 0.17, 64 0.94 -> 0.21, 102 1.75 -> 0.41, 128 2.11 -> 0.50; batches of 256 against cuSOLVER's
// batched call: n = 20 0.34 -> 0.12 ms, 64 1.08 -> 0.38, 128 3.30 -> 0.96.  Residuals and orthogonality as the library's.
#include <cuda_runtime.h>
#include <math.h>
#include <math_constants.h>
#include <stdint.h>
#include <stdio.h>

#include "dftbaby_b200.h"

namespace {

#include "dmma.cuh"

constexpr double EPS = 1.1102230246251565e-16;  // unit roundoff
constexpr int SECULAR_ITERATIONS = 80;          // the bracket alone converges in fewer

// Shared memory: Z (rows in blocks of 8, pitch 4 mod 16 doubles: conflict-free reads of the tensor instruction's A
// operand), U (pitch 8 mod 16: its B operand; 64 columns at a time), the vectors below.
struct Layout {
    int rows, zp, up;
    __host__ __device__ explicit Layout(int n)
        : rows((n + 7) / 8 * 8), zp((n + 15) / 16 * 16 + 4), up((n > 64 ? 64 : (n + 15) / 16 * 16) + 8) {}
    __host__ __device__ size_t z() const { return (size_t)rows * zp; }
    __host__ __device__ size_t u() const { return (size_t)rows * up; }
};

template <int NC> struct Vectors {
    static constexpr int N = 32 * NC;
    double d[N], e[N], tau[N], zs[N], ds[N], kd[N], kz[N], zh[N], x[N], scale[N];
    double rho[N / 2];
    double red[4 * NC];
    int ord[N], slot[N], org[N], typ[N], top[N], bot[N];
    int K[N / 2], ntop[N / 2], nbot[N / 2];
    int bad;
};

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Sums of M (a power of two up to 8) values over the 32 lanes: lane l returns the sum of value l / (32 / M).
template <int M> __device__ __forceinline__ double warp_sums(double (&v)[8]) {
    const int lane = threadIdx.x & 31;
    int o = 16;
#pragma unroll
    for (int half = M / 2; half > 0; half >>= 1, o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int q = 0; q < half; ++q) {
            const double send = up ? v[q] : v[q + half], keep = up ? v[q + half] : v[q];
            v[q] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    double s = v[0];
    for (; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

// sum / product over the four lanes that share a column or a root; they are always converged
__device__ __forceinline__ double quad_sum(double v) {
    const unsigned m = 0xfu << (threadIdx.x & 28);
    v += __shfl_xor_sync(m, v, 1);
    return v + __shfl_xor_sync(m, v, 2);
}

__device__ __forceinline__ double quad_product(double v) {
    const unsigned m = 0xfu << (threadIdx.x & 28);
    v *= __shfl_xor_sync(m, v, 1);
    return v * __shfl_xor_sync(m, v, 2);
}

// The root (a - s) / (2 c) of c t^2 - a t + b, s = sqrt(a^2 - 4 b c) (last: the root (a + s) / (2 c)), without
// cancellation.
__device__ __forceinline__ double quadratic(double c, double a, double b, bool last) {
    const double s = sqrt(fabs(a * a - 4.0 * b * c));
    if (last) return a >= 0.0 ? (a + s) / (2.0 * c) : 2.0 * b / (a - s);
    return a <= 0.0 ? (a - s) / (2.0 * c) : 2.0 * b / (a + s);
}

// Root j of 1/rho + sum_i z_i^2 / (d_i - lambda) (K poles d ascending, |z| = 1 at most) as lambda = d[origin] + x, the
// origin being the nearer pole, so that d_i - lambda is known to full relative precision for every i.  Called by the
// four lanes of a quad; lane q sums the terms q, q + 4, ...
__device__ void secular_root(int K, int j, const double *d, const double *z, double rho, int q, int *origin, double *xout) {
    const double ri = 1.0 / rho;
    if (K == 1) {
        *origin = 0;
        *xout = rho * z[0] * z[0];
        return;
    }
    const bool last = j == K - 1;
    const int jl = last ? K - 2 : j, jr = jl + 1;  // the two poles of the interpolation
    // psi sums the terms up to jl, phi those from jr on
    double lo, hi, x;
    int org;
    {
        // the value half way decides the origin; the terms of the two poles, exact, give the first x
        const double base = last ? d[K - 1] : d[j];
        const double len = last ? rho : d[j + 1] - d[j];
        const double mid = 0.5 * len;
        double rest = 0.0;
        for (int i = q; i < K; i += 4)
            if (i != jl && i != jr) rest += z[i] * z[i] / ((d[i] - base) - mid);
        const double c = ri + quad_sum(rest);
        const double zl = z[jl] * z[jl], zr = z[jr] * z[jr];
        const double w = c + zl / ((d[jl] - base) - mid) + zr / ((d[jr] - base) - mid);
        org = last ? K - 1 : (w >= 0.0 ? j : j + 1);
        const double dl = d[jl] - d[org], dr = d[jr] - d[org];
        if (last) {
            lo = w <= 0.0 ? mid : 0.0;
            hi = w <= 0.0 ? len * (1.0 + 64.0 * EPS) : mid;  // |z| = 1 up to roundoff
        } else {
            lo = w >= 0.0 ? 0.0 : -mid;
            hi = w >= 0.0 ? mid : 0.0;
        }
        x = quadratic(c, c * (dl + dr) + zl + zr, c * dl * dr + zl * dr + zr * dl, last);
        if (!(x > lo && x < hi)) x = 0.5 * (lo + hi);
    }
    const double o = d[org], dl = d[jl] - o, dr = d[jr] - o;
    for (int it = 0; it < SECULAR_ITERATIONS; ++it) {
        double psi = 0.0, dpsi = 0.0, phi = 0.0, dphi = 0.0;
        for (int i = q; i < K; i += 4) {
            const double t = z[i] / ((d[i] - o) - x);
            if (i <= jl) {
                psi += z[i] * t;
                dpsi += t * t;
            } else {
                phi += z[i] * t;
                dphi += t * t;
            }
        }
        psi = quad_sum(psi);
        phi = quad_sum(phi);
        dpsi = quad_sum(dpsi);
        dphi = quad_sum(dphi);
        const double w = ri + psi + phi, dw = dpsi + dphi;
        if (fabs(w) <= EPS * (ri + 8.0 * (fabs(psi) + fabs(phi)) + fabs(x) * dw)) break;
        if (w < 0.0)
            lo = x;
        else
            hi = x;
        const double tl = dl - x, tr = dr - x;
        double c = w - tl * dpsi - tr * dphi;
        if (last) c = fabs(c);
        double eta = quadratic(c, (tl + tr) * w - tl * tr * dw, tl * tr * w, last);
        if (!(w * eta < 0.0)) eta = -w / dw;
        double xn = x + eta;
        if (!(xn > lo && xn < hi)) xn = 0.5 * (lo + hi);
        if (xn == x || !(xn > lo && xn < hi)) break;  // the bracket has no number left inside
        x = xn;
    }
    *origin = org;
    *xout = x;
}

// Deflation of one merge (positions off .. off + s of the sorted d and z) by one warp: the kept poles to kd, kz, slot;
// equal ones are rotated together in the columns of Z.
template <int NC>
__device__ int deflate(Vectors<NC> &sv, double *Z, int zp, int off, int s, double rho, double tol) {
    const int lane = threadIdx.x & 31;
    int K = 0;
    for (int c = 0; c < s; c += 32) {
        const int p = off + c + lane;
        const bool keep = c + lane < s && rho * fabs(sv.zs[p]) > tol;
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        if (keep) {
            const int k = off + K + __popc(m & ((1u << lane) - 1));
            sv.kd[k] = sv.ds[p];
            sv.kz[k] = sv.zs[p];
            sv.slot[k] = sv.ord[p];
        }
        K += __popc(m);
    }
    __syncwarp();
    // two neighbours deflate when the rotation that zeroes one of their z leaves an element below tol
    auto close = [&](double d0, double z0, double d1, double z1) {
        return fabs((d1 - d0) * z0 * z1) <= tol * (z0 * z0 + z1 * z1);
    };
    bool any = false;
    for (int i = lane; i < K - 1; i += 32)
        any |= close(sv.kd[off + i], sv.kz[off + i], sv.kd[off + i + 1], sv.kz[off + i + 1]);
    if (__any_sync(0xffffffffu, any)) {
        double pd = sv.kd[off], pz = sv.kz[off];
        int ps = sv.slot[off], out = 0;
        for (int i = 1; i < K; ++i) {
            const double d = sv.kd[off + i], z = sv.kz[off + i];
            const int sl = sv.slot[off + i];
            __syncwarp();
            if (close(pd, pz, d, z)) {
                const double t = sqrt(z * z + pz * pz), c = z / t, sn = pz / t;
                for (int r = off + lane; r < off + s; r += 32) {
                    const double a = Z[r * zp + ps], b = Z[r * zp + sl];
                    Z[r * zp + ps] = c * a - sn * b;
                    Z[r * zp + sl] = c * b + sn * a;
                }
                if (lane == 0) {
                    sv.d[ps] = pd * c * c + d * sn * sn;
                    const int ty = sv.typ[ps] | sv.typ[sl];
                    sv.typ[ps] = sv.typ[sl] = ty;
                }
                pd = pd * sn * sn + d * c * c;
                pz = t;
            } else {
                if (lane == 0) {
                    sv.kd[off + out] = pd;
                    sv.kz[off + out] = pz;
                    sv.slot[off + out] = ps;
                }
                ++out;
                pd = d;
                pz = z;
            }
            ps = sl;
        }
        if (lane == 0) {
            sv.kd[off + out] = pd;
            sv.kz[off + out] = pz;
            sv.slot[off + out] = ps;
        }
        K = out + 1;
    }
    __syncwarp();
    return K;
}

// the kept columns of one merge with elements in its upper (bit 1) or lower (bit 2) rows, as lists
template <int NC> __device__ int column_list(const Vectors<NC> &sv, int *list, int off, int K, int bit) {
    const int lane = threadIdx.x & 31;
    int n = 0;
    for (int c = 0; c < K; c += 32) {
        const bool in = c + lane < K && (sv.typ[sv.slot[off + c + lane]] & bit);
        const unsigned m = __ballot_sync(0xffffffffu, in);
        if (in) list[off + n + __popc(m & ((1u << lane) - 1))] = c + lane;
        n += __popc(m);
    }
    return n;
}

// n <= 32 NC.  A: lower triangle of batch matrices, element (i, j) at A[b * sb + i * si + j * sj].  W: ascending
// eigenvalues (batch x n).  V: vector j of matrix b at V[(b n + j) n ..].  info[b]: 0, or 1 for a matrix that is not finite.
// V may be A when si = n, sj = 1, sb = n n: it is written after A has been read.
template <int NC>
__global__ void __launch_bounds__(128 * NC, 1)
    small_eigh_kernel(int n, const double *A, long long sb, long long si, long long sj, double *W, double *V, int *info) {
    constexpr int N = 32 * NC, WARPS = 4 * NC, THREADS = 32 * WARPS, NR = 8;
    extern __shared__ __align__(16) double smem[];
    const Layout lay(n);
    const int zp = lay.zp, up = lay.up;
    double *Z = smem, *U = Z + lay.z();
    Vectors<NC> &sv = *reinterpret_cast<Vectors<NC> *>(U + lay.u());
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    A += blockIdx.x * sb;
    W += (size_t)blockIdx.x * n;
    V += (size_t)blockIdx.x * n * n;

    // ---------------- 1. tridiagonalisation
    double a[NR][NC];
    double amax = 0.0;
    bool finite = true;
#pragma unroll
    for (int r = 0; r < NR; ++r)
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const int i = warp + WARPS * r, j = lane + 32 * c;
            double v = 0.0;
            if (i < n && j < n) v = i >= j ? A[i * si + j * sj] : A[j * si + i * sj];
            a[r][c] = v;
            amax = fmax(amax, fabs(v));
            finite = finite && isfinite(v);
        }
    if (tid == 0) sv.bad = 0;
    __syncthreads();
    if (!finite) sv.bad = 1;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmax(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    if (lane == 0) sv.red[warp] = amax;
    __syncthreads();
    if (sv.bad) {
        if (tid == 0) info[blockIdx.x] = 1;
        for (int i = tid; i < n; i += THREADS) W[i] = CUDART_NAN;
        for (int i = tid; i < n * n; i += THREADS) V[i] = CUDART_NAN;
        return;
    }
    for (int w = 0; w < WARPS; ++w) amax = fmax(amax, sv.red[w]);
    // a power of two that brings the largest element near one: no sum of squares over- or underflows
    int ex = 0;
    if (amax > 0.0) frexp(amax, &ex);
    ex = max(-1000, min(1000, ex));
    const double down = ldexp(1.0, -ex), back = ldexp(1.0, ex);
#pragma unroll
    for (int r = 0; r < NR; ++r)
#pragma unroll
        for (int c = 0; c < NC; ++c) a[r][c] *= down;

    double *hv = U, *hp = U + 2 * N;  // reflector and A v, two buffers each
#pragma unroll
    for (int r = 0; r < NR; ++r) {
        for (int t = 0; t < WARPS; ++t) {
            const int k = WARPS * r + t;
            if (k >= n - 2) break;
            double *v = hv + (k & 1) * N, *p = hp + (k & 1) * N;
            if (warp == t) {
                double dk = 0.0, alpha = 0.0, sigma = 0.0;
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    const int j = lane + 32 * c;
                    const double dd = __shfl_sync(0xffffffffu, a[r][c], k & 31);
                    const double aa = __shfl_sync(0xffffffffu, a[r][c], (k + 1) & 31);
                    if (c == k / 32) dk = dd;
                    if (c == (k + 1) / 32) alpha = aa;
                    if (j > k + 1) sigma += a[r][c] * a[r][c];
                }
                sigma = warp_sum(sigma);
                double beta = alpha, tau = 0.0, scale = 0.0;
                if (sigma > 0.0) {
                    beta = -copysign(sqrt(alpha * alpha + sigma), alpha);
                    tau = (beta - alpha) / beta;
                    scale = 1.0 / (alpha - beta);
                }
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    const int j = lane + 32 * c;
                    const double x = j > k + 1 ? a[r][c] * scale : (j == k + 1 ? 1.0 : 0.0);
                    v[j] = x;
                    if (j > k && j < n) V[(size_t)k * n + j] = x;  // kept for step 3
                }
                if (lane == 0) {
                    sv.d[k] = dk;
                    sv.e[k] = beta;
                    sv.tau[k] = tau;
                }
            }
            __syncthreads();
            const double tau = sv.tau[k];
            if (tau == 0.0) continue;
            double vj[NC], s[8];
#pragma unroll
            for (int c = 0; c < NC; ++c) vj[c] = v[lane + 32 * c];
            // rows before WARPS r are done: NR - r values a lane
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                s[q] = 0.0;
                if (r + q < NR)
#pragma unroll
                    for (int c = 0; c < NC; ++c) s[q] += a[r + q < NR ? r + q : 0][c] * vj[c];
            }
            const int left = NR - r;
            if (left > 4) {
                const double x = warp_sums<8>(s);
                const int q = lane >> 2;
                if ((lane & 3) == 0 && q < left) p[warp + WARPS * (r + q)] = x;
            } else if (left > 2) {
                const double x = warp_sums<4>(s);
                const int q = lane >> 3;
                if ((lane & 7) == 0 && q < left) p[warp + WARPS * (r + q)] = x;
            } else {
                const double x = warp_sums<2>(s);
                const int q = lane >> 4;
                if ((lane & 15) == 0 && q < left) p[warp + WARPS * (r + q)] = x;
            }
            __syncthreads();
            // A -= v w^T + w v^T, w = tau p - (tau^2 v.p / 2) v
            double wj[NC], vp = 0.0;
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                const int j = lane + 32 * c;
                wj[c] = j > k ? p[j] : 0.0;
                vp += vj[c] * wj[c];
            }
            const double half = 0.5 * tau * tau * warp_sum(vp);
#pragma unroll
            for (int c = 0; c < NC; ++c) wj[c] = tau * wj[c] - half * vj[c];
#pragma unroll
            for (int q = 0; q < NR; ++q) {
                if (r + q >= NR) continue;
                const int i = warp + WARPS * (r + q);
                const double vi = v[i], wi = i > k ? tau * p[i] - half * vi : 0.0;
#pragma unroll
                for (int c = 0; c < NC; ++c) a[r + q < NR ? r + q : 0][c] -= vi * wj[c] + wi * vj[c];
            }
        }
    }
#pragma unroll
    for (int r = 0; r < NR; ++r)
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const int i = warp + WARPS * r, j = lane + 32 * c;
            if (i == j && i < n && i >= n - 2) sv.d[i] = a[r][c];
            if (i == n - 1 && j == n - 2) sv.e[j] = a[r][c];
        }
    __syncthreads();

    // ---------------- 2. divide and conquer, from blocks of one: every coupling is taken out of both its neighbours
    for (int i = tid; i < lay.rows * zp; i += THREADS) Z[i] = 0.0;
    double dleaf = 0.0;
    if (tid < n) {
        dleaf = sv.d[tid];
        if (tid > 0) dleaf -= fabs(sv.e[tid - 1]);
        if (tid < n - 1) dleaf -= fabs(sv.e[tid]);
    }
    __syncthreads();
    if (tid < n) {
        sv.d[tid] = dleaf;
        Z[tid * zp + tid] = 1.0;
    }
    __syncthreads();
    const int pos = tid >> 2, q4 = tid & 3;  // column, pole or root of this quad
    for (int w = 1; w < n; w *= 2) {
        const int off = pos / (2 * w) * (2 * w), mid = off + w, end = min(off + 2 * w, n);
        const int m = pos / (2 * w), jj = pos - off;
        const bool merging = pos < n && mid < n;
        // z, and d and z in ascending order
        if (merging) {
            const double e = sv.e[mid - 1];
            const double zi = (pos < mid ? Z[(mid - 1) * zp + pos] : copysign(1.0, e) * Z[mid * zp + pos]) * 0.70710678118654752440;
            const double di = sv.d[pos];
            int rank = 0;
            for (int i = off + q4; i < end; i += 4) {
                const double x = sv.d[i];
                rank += x < di || (x == di && i < pos);
            }
            const unsigned qm = 0xfu << (lane & 28);
            rank += __shfl_xor_sync(qm, rank, 1);
            rank += __shfl_xor_sync(qm, rank, 2);
            if (q4 == 0) {
                sv.ds[off + rank] = di;
                sv.zs[off + rank] = zi;
                sv.ord[off + rank] = pos;
                sv.typ[pos] = pos < mid ? 1 : 2;
            }
        }
        __syncthreads();
        for (int mm = warp; mm * 2 * w + w < n; mm += WARPS) {
            const int o = mm * 2 * w, s = min(2 * w, n - o);
            double zmax = 0.0, dmax = 0.0;
            for (int i = lane; i < s; i += 32) {
                zmax = fmax(zmax, fabs(sv.zs[o + i]));
                dmax = fmax(dmax, fabs(sv.ds[o + i]));
            }
#pragma unroll
            for (int x = 16; x > 0; x >>= 1) {
                zmax = fmax(zmax, __shfl_xor_sync(0xffffffffu, zmax, x));
                dmax = fmax(dmax, __shfl_xor_sync(0xffffffffu, dmax, x));
            }
            const double rho = 2.0 * fabs(sv.e[o + w - 1]), tol = 8.0 * EPS * fmax(dmax, zmax);
            const int K = deflate<NC>(sv, Z, zp, o, s, rho, tol);
            const int nt = column_list<NC>(sv, sv.top, o, K, 1), nb = column_list<NC>(sv, sv.bot, o, K, 2);
            if (lane == 0) {
                sv.K[mm] = K;
                sv.ntop[mm] = nt;
                sv.nbot[mm] = nb;
                sv.rho[mm] = rho;
            }
        }
        __syncthreads();
        const int K = merging ? sv.K[m] : 0;
        const double *kd = sv.kd + off, *kz = sv.kz + off;
        if (jj < K) {
            int org;
            double x;
            secular_root(K, jj, kd, kz, sv.rho[m], q4, &org, &x);
            if (q4 == 0) {
                sv.org[pos] = org;
                sv.x[pos] = x;
            }
        }
        __syncthreads();
        // the z for which these roots are exact: z_i^2 = prod_j (lambda_j - d_i) / prod_(j != i) (d_j - d_i), up to a factor
        if (jj < K) {
            const double di = kd[jj];
            double pr = 1.0;
            for (int j = q4; j < K; j += 4) {
                const double num = (kd[sv.org[off + j]] - di) + sv.x[off + j];
                const double den = j < jj ? kd[j] - di : (j < K - 1 ? kd[j + 1] - di : 1.0);
                pr *= num / den;
            }
            pr = quad_product(pr);
            if (q4 == 0) sv.zh[pos] = copysign(sqrt(fabs(pr)), kz[jj]);
        }
        __syncthreads();
        // vectors of the merged problem, 64 columns at a time, and their product with the old ones
        constexpr int CHUNKS = NC > 2 ? 2 : 1;
        const double lam = jj < K ? kd[sv.org[pos]] + sv.x[pos] : 0.0;
        auto vectors = [&](int ch) {
            if (jj < K && jj / 64 == ch) {
                const double o = kd[sv.org[pos]], x = sv.x[pos];
                double ss = 0.0;
                for (int i = q4; i < K; i += 4) {
                    const double u = sv.zh[off + i] / ((kd[i] - o) - x);
                    U[(off + i) * up + jj - 64 * ch] = u;
                    ss += u * u;
                }
                ss = quad_sum(ss);
                if (q4 == 0) sv.scale[pos] = 1.0 / sqrt(ss);
            }
        };
        if (2 * w >= 8) {
            // warp: rows 8 warp .. + 7, inside one merge
            const int r0 = 8 * warp, ro = r0 / (2 * w) * (2 * w), rm = r0 / (2 * w);
            const bool live = r0 < n && ro + w < n;
            const int RK = live ? sv.K[rm] : 0;
            const bool upper = r0 < ro + w, lower = r0 + 7 >= ro + w;
            const int cnt = upper && lower ? RK : (upper ? (live ? sv.ntop[rm] : 0) : (live ? sv.nbot[rm] : 0));
            const int *list = upper ? sv.top + ro : sv.bot + ro;
            double acc[CHUNKS][8][2];
#pragma unroll
            for (int ch = 0; ch < CHUNKS; ++ch) {
                if (ch > 0) __syncthreads();  // the first 64 columns have been used
                if (ch == 0 || 2 * w > 64) vectors(ch);
                __syncthreads();
#pragma unroll
                for (int t = 0; t < 8; ++t) acc[ch][t][0] = acc[ch][t][1] = 0.0;
                const int cols = RK - 64 * ch;
                if (cols > 0)
                    for (int k0 = 0; k0 < cnt; k0 += 4) {
                        const int kq = k0 + (lane & 3), kc = min(kq, cnt - 1);
                        const int ki = upper && lower ? kc : list[kc];
                        const double av = kq < cnt ? Z[(r0 + (lane >> 2)) * zp + sv.slot[ro + ki]] : 0.0;
                        const double *ur = U + (ro + ki) * up + (lane >> 2);
#pragma unroll
                        for (int t = 0; t < 8; ++t)
                            if (8 * t < cols) dmma884(acc[ch][t][0], acc[ch][t][1], av, ur[8 * t]);
                    }
            }
            __syncwarp();
            const int r = r0 + (lane >> 2);
#pragma unroll
            for (int ch = 0; ch < CHUNKS; ++ch)
#pragma unroll
                for (int t = 0; t < 8; ++t)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int j = 64 * ch + 8 * t + 2 * (lane & 3) + h;
                        if (r < n && j < RK) Z[r * zp + sv.slot[ro + j]] = acc[ch][t][h] * sv.scale[ro + j];
                    }
        } else {
            // blocks of two and four: an element a thread (row pos, column q4)
            vectors(0);
            __syncthreads();
            double v = 0.0;
            const bool mine = merging && q4 < K;
            if (mine) {
                for (int i = 0; i < K; ++i) v += Z[pos * zp + sv.slot[off + i]] * U[(off + i) * up + q4];
                v *= sv.scale[off + q4];
            }
            __syncthreads();
            if (mine) Z[pos * zp + sv.slot[off + q4]] = v;
        }
        if (jj < K && q4 == 0) sv.d[sv.slot[pos]] = lam;
        __syncthreads();
    }

    // ---------------- 3. reflectors, in the order n - 3 .. 0, on this quad's column; ascending order
    // reflector k from element base(k) + k + 1 on; base(k) is even, so that pairs of rows come in 16-byte reads
    auto base = [&](int k) {
        // rows of n - k + 1 elements, rounded up to even, minus the k leading ones that are not stored (even part)
        const int kk = k / 2;  // reflectors 2 kk and 2 kk + 1 both start at row 2 kk
        const int len = (n + 1) & ~1;
        return (k & 1 ? (len - 2 * kk) : 0) + 2 * (kk * len - kk * (kk - 1)) - 2 * kk;
    };
    for (int k = warp; k < n - 2; k += WARPS) {
        double *dst = U + base(k);
        for (int j = (k & ~1) + lane; j < ((n + 1) & ~1); j += 32) dst[j] = j > k && j < n ? V[(size_t)k * n + j] : 0.0;
    }
    const double ev = pos < n ? sv.d[pos] : 0.0;
    int rank = 0;
    for (int i = q4; i < n; i += 4) {
        const double x = sv.d[i];
        rank += x < ev || (x == ev && i < pos);
    }
    rank += __shfl_xor_sync(0xffffffffu, rank, 1);
    rank += __shfl_xor_sync(0xffffffffu, rank, 2);
    __syncthreads();  // V has been read
    double y[N / 8][2];  // rows 8 t + 2 q4, + 1
#pragma unroll
    for (int t = 0; t < N / 8; ++t)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int i = 8 * t + 2 * q4 + h;
            y[t][h] = i < n && pos < n ? Z[i * zp + pos] : 0.0;
        }
    for (int k = n - 3; k >= 0; --k) {
        const double tau = sv.tau[k];
        if (tau == 0.0) continue;
        const double *v = U + base(k) + 2 * q4;
        const int t0 = k / 8;  // earlier blocks of rows are zero in v
        double s0 = 0.0, s1 = 0.0;
#pragma unroll
        for (int t = 0; t < N / 8; ++t)
            if (t >= t0 && 8 * t + 2 * q4 < n && 8 * t + 2 * q4 >= (k & ~1)) {
                const double2 x = *reinterpret_cast<const double2 *>(v + 8 * t);
                s0 += x.x * y[t][0];
                s1 += x.y * y[t][1];
            }
        const double f = tau * quad_sum(s0 + s1);
#pragma unroll
        for (int t = 0; t < N / 8; ++t)
            if (t >= t0 && 8 * t + 2 * q4 < n && 8 * t + 2 * q4 >= (k & ~1)) {
                const double2 x = *reinterpret_cast<const double2 *>(v + 8 * t);
                y[t][0] -= f * x.x;
                y[t][1] -= f * x.y;
            }
    }
    if (pos < n) {
        if (q4 == 0) W[rank] = ev * back;
#pragma unroll
        for (int t = 0; t < N / 8; ++t)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int i = 8 * t + 2 * q4 + h;
                if (i < n) V[(size_t)rank * n + i] = y[t][h];
            }
    }
    if (tid == 0) info[blockIdx.x] = 0;
}

template <int NC>
cudaError_t launch_eigh(int n, int batch, const double *A, long long sb, long long si, long long sj, double *W, double *V,
                        int *info, cudaStream_t st) {
    const Layout lay(n);
    const size_t bytes = (lay.z() + lay.u()) * sizeof(double) + sizeof(Vectors<NC>);
    cudaError_t e = cudaFuncSetAttribute(small_eigh_kernel<NC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return e;
    small_eigh_kernel<NC><<<batch, 128 * NC, bytes, st>>>(n, A, sb, si, sj, W, V, info);
    return cudaGetLastError();
}

}  // namespace

extern "C" int dftb_small_eigh(int n, int batch, const double *A, long long batch_stride, long long row_stride,
                               long long col_stride, double *W, double *V, int *info, void *stream) {
    if (n <= 0 || n > DFTB_SMALL_EIGH_MAX || batch <= 0) return DFTB_ERR_BAD_SIZE;
    if (!A || !W || !V || !info) return DFTB_ERR_NULL;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    cudaError_t e = n <= 32   ? launch_eigh<1>(n, batch, A, batch_stride, row_stride, col_stride, W, V, info, st)
                    : n <= 64 ? launch_eigh<2>(n, batch, A, batch_stride, row_stride, col_stride, W, V, info, st)
                    : n <= 96 ? launch_eigh<3>(n, batch, A, batch_stride, row_stride, col_stride, W, V, info, st)
                              : launch_eigh<4>(n, batch, A, batch_stride, row_stride, col_stride, W, V, info, st);
    return e == cudaSuccess ? DFTB_OK : DFTB_ERR_CUDA;
}
