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
//   3. The reflectors are applied in blocks of eight by FP64 tensor instructions, a warp owning 8 columns; no barriers.
//
// Bound by its serial steps and by instruction issue on one SM (n = 102: tridiagonalisation 266k cycles, divide and
// conquer 249k, reflectors 42k; applying these one at a time from columns in registers took 184k).  B200, host
// included, against torch.linalg.eigh: n = 20 0.26 -> 0.11 ms, 42 0.70 -> 0.15, 64 0.94 -> 0.19, 102 1.75 -> 0.34, 128
// 2.11 -> 0.39; batches of 256 against cuSOLVER's batched call: n = 20 0.34 -> 0.12 ms, 64 1.08 -> 0.33, 128 3.28 ->
// 0.75.  Residuals and orthogonality as the library's.
#include <cuda_runtime.h>
#include <math.h>
#include <math_constants.h>
#include <stdint.h>
#include <stdio.h>

#include "dftbaby_b200.h"

namespace {

#include "dmma.cuh"

constexpr double EPS = 1.1102230246251565e-16;  // unit roundoff
// The bracket alone converges in fewer: it is at most 4 wide, and deflation keeps a root at least 1e-33 from its pole, so
// about 110 halvings reach the root's magnitude and 53 more its last bit.  (6 to 45 steps on tridiagonals of small
// integers, Clement, Wilkinson and glued matrices.)
constexpr int SECULAR_ITERATIONS = 192;

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
    double d[N], tau[N];
    double e[N], zs[N], ds[N], kd[N], kz[N], zh[N], x[N], scale[N];  // step 3: 8 x 8 matrices of the reflector blocks
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

// sum / product over the four lanes that share a column or a root; called by whole warps
__device__ __forceinline__ double quad_sum(double v) {
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    return v + __shfl_xor_sync(0xffffffffu, v, 2);
}

__device__ __forceinline__ double quad_product(double v) {
    v *= __shfl_xor_sync(0xffffffffu, v, 1);
    return v * __shfl_xor_sync(0xffffffffu, v, 2);
}

// The root (a - s) / (2 c) of c t^2 - a t + b, s = sqrt(a^2 - 4 b c) (last: the root (a + s) / (2 c)), without
// cancellation.
__device__ __forceinline__ double quadratic(double c, double a, double b, bool last) {
    const double s = sqrt(fabs(a * a - 4.0 * b * c));
    if (last) return a >= 0.0 ? (a + s) / (2.0 * c) : 2.0 * b / (a - s);
    return a <= 0.0 ? (a - s) / (2.0 * c) : 2.0 * b / (a + s);
}

// Root j of 1/rho + sum_i z_i^2 / (d_i - lambda) (K poles d ascending, |z| = 1 at most) as lambda = d[origin] + x, the
// origin being the nearer pole, so that d_i - lambda is known to full relative precision for every i.  A quad of lanes a
// root, lane q summing the terms q, q + 4, ...; the warp's eight quads (of up to Kw poles each) iterate in step.  live: this
// quad has a root.  Returns whether this quad's root converged.
__device__ bool secular_roots(bool live, int K, int Kw, int j, const double *d, const double *z, double rho, int q,
                              int *origin, double *xout) {
    const double ri = 1.0 / rho;
    const bool single = K < 2;
    const bool last = j == K - 1;
    const int jl = single ? 0 : (last ? K - 2 : j), jr = single ? 0 : jl + 1;  // the two poles of the interpolation
    const double o0 = d[j], len = last ? rho : d[jr] - o0, mid = 0.5 * len;
    // the value half way decides the origin; the terms of the two poles, exact, give the first x
    double c = 0.0;
    for (int i0 = 0; i0 < Kw; i0 += 8) {  // two terms share a division
        const int i = min(i0 + q, K - 1), i2 = min(i0 + q + 4, K - 1);
        const double z1 = i0 + q < K && i != jl && i != jr ? z[i] : 0.0, z2 = i0 + q + 4 < K && i2 != jl && i2 != jr ? z[i2] : 0.0;
        const double a = (d[i] - o0) - mid, b = (d[i2] - o0) - mid, r = 1.0 / (a * b);
        c += z1 * z1 * (b * r) + z2 * z2 * (a * r);
    }
    c = ri + quad_sum(c);
    const double zl = z[jl] * z[jl], zr = z[jr] * z[jr];
    const double wm = c + zl / ((d[jl] - o0) - mid) + zr / ((d[jr] - o0) - mid);
    const int org = last ? j : (wm >= 0.0 ? j : jr);
    const double o = d[org], dl = d[jl] - o, dr = d[jr] - o;
    double lo, hi;
    if (last) {
        lo = wm <= 0.0 ? mid : 0.0;
        hi = wm <= 0.0 ? len * (1.0 + 64.0 * EPS) : mid;  // |z| = 1 up to roundoff
    } else {
        lo = wm >= 0.0 ? 0.0 : -mid;
        hi = wm >= 0.0 ? mid : 0.0;
    }
    double x = quadratic(c, c * (dl + dr) + zl + zr, c * dl * dr + zl * dr + zr * dl, last);
    if (!(x > lo && x < hi)) x = 0.5 * (lo + hi);
    if (single) x = rho * z[0] * z[0];
    // The middle is an end of the bracket but no pole, and a root may lie on it (matrices of small integers, symmetric
    // chains): it is tried as a value when a step first leads there.
    const double end = last || wm >= 0.0 ? mid : -mid;
    bool untried = true;
    bool done = !live || single;
    for (int it = 0; it < SECULAR_ITERATIONS; ++it) {
        if (__all_sync(0xffffffffu, done)) break;
        double psi = 0.0, dpsi = 0.0, all = 0.0, dw = 0.0;  // the terms up to jl, and all of them
        for (int i0 = 0; i0 < Kw; i0 += 8) {
            const int i = min(i0 + q, K - 1), i2 = min(i0 + q + 4, K - 1);
            const double z1 = i0 + q < K ? z[i] : 0.0, z2 = i0 + q + 4 < K ? z[i2] : 0.0;
            const double a = (d[i] - o) - x, b = (d[i2] - o) - x, r = 1.0 / (a * b);
            const double t1 = z1 * (b * r), t2 = z2 * (a * r);
            const double l1 = i <= jl ? t1 : 0.0, l2 = i2 <= jl ? t2 : 0.0;
            all += z1 * t1 + z2 * t2;
            dw += t1 * t1 + t2 * t2;
            psi += z1 * l1 + z2 * l2;
            dpsi += l1 * l1 + l2 * l2;
        }
        psi = quad_sum(psi);
        all = quad_sum(all);
        dpsi = quad_sum(dpsi);
        dw = quad_sum(dw);
        const double phi = all - psi, dphi = fmax(dw - dpsi, 0.0), w = ri + all;
        done = done || fabs(w) <= EPS * (ri + 8.0 * (fabs(psi) + fabs(phi)) + fabs(x) * dw);
        lo = w < 0.0 ? x : lo;
        hi = w < 0.0 ? hi : x;
        const double tl = dl - x, tr = dr - x;
        const double cc = w - tl * dpsi - tr * dphi;
        double eta = quadratic(last ? fabs(cc) : cc, (tl + tr) * w - tl * tr * dw, tl * tr * w, last);
        if (!(w * eta < 0.0)) eta = -w / dw;
        double xn = x + eta;
        // a step this short against the distances to the poles is the last, if it is taken: its error is of second order
        // in them
        bool last_step = fabs(eta) <= 1e-9 * fmin(fabs(tl), fabs(tr)), full = xn == x;
        if (!full && !(xn > lo && xn < hi)) {
            const bool try_end = untried && (w < 0.0 ? hi : lo) == end;
            xn = try_end ? end : 0.5 * (lo + hi);
            untried = untried && !try_end;
            full = !try_end && !(xn > lo && xn < hi);  // the bracket has no number left inside
            last_step = false;
        }
        if (!done && !full) x = xn;
        done = done || full || last_step;
    }
    *origin = org;
    *xout = x;
    return done;
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

// the kept columns of one merge with elements in its upper (bit 1) or lower (bit 2) rows (bits 3: all), as lists of
// pole | slot << 8
template <int NC> __device__ int column_list(const Vectors<NC> &sv, int *list, int off, int K, int bit) {
    const int lane = threadIdx.x & 31;
    int n = 0;
    for (int c = 0; c < K; c += 32) {
        const bool in = c + lane < K && (sv.typ[sv.slot[off + c + lane]] & bit);
        const unsigned m = __ballot_sync(0xffffffffu, in);
        if (in) list[off + n + __popc(m & ((1u << lane) - 1))] = (c + lane) | sv.slot[off + c + lane] << 8;
        n += __popc(m);
    }
    return n;
}

// n <= 32 NC.  A: lower triangle of batch matrices, element (i, j) at A[b * sb + i * si + j * sj].  W: ascending
// eigenvalues (batch x n).  V: vector j of matrix b at V[(b n + j) n ..].  info[b]: 0, 1 for a matrix that is not finite, or 2
// for a root that did not converge.
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
    // reflector k, H = 1 - tau v v^T, from row k of the reduced matrix (held by one warp): v = x - beta e_(k+1)
    auto publish = [&](const double (&row)[NC], int k) {
        double dk = 0.0, alpha = 0.0, sigma = 0.0;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const double dd = __shfl_sync(0xffffffffu, row[c], k & 31);
            const double aa = __shfl_sync(0xffffffffu, row[c], (k + 1) & 31);
            if (c == k / 32) dk = dd;
            if (c == (k + 1) / 32) alpha = aa;
            if (lane + 32 * c > k + 1) sigma += row[c] * row[c];
        }
        sigma = warp_sum(sigma);
        // elements below 1e-140 of the largest one are dropped: their squares underflow
        const bool flat = !(sigma > 1e-280);
        const double beta = flat ? alpha : -copysign(sqrt(alpha * alpha + sigma), alpha);
        double *v = hv + (k & 1) * N;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const int j = lane + 32 * c;
            const double x = flat || j <= k ? 0.0 : (j == k + 1 ? alpha - beta : row[c]);
            v[j] = x;
            if (j > k && j < n) V[(size_t)k * n + j] = x;  // kept for step 3
        }
        if (lane == 0) {
            sv.d[k] = dk;
            sv.e[k] = beta;
            sv.tau[k] = flat ? 0.0 : 1.0 / (beta * (beta - alpha));
        }
    };
    if (n > 2 && warp == 0) publish(a[0], 0);
#pragma unroll
    for (int r = 0; r < NR; ++r) {
        const int C0 = WARPS * r / 32;  // columns 32 C0 and earlier rows are done
        for (int t = 0; t < WARPS; ++t) {
            const int k = WARPS * r + t;
            if (k >= n - 2) break;
            const double *v = hv + (k & 1) * N;
            double *p = hp + (k & 1) * N;
            const bool next = k + 1 < n - 2 && warp == (t + 1) % WARPS;  // this warp holds row k + 1
            __syncthreads();
            const double tau = sv.tau[k];
            if (tau == 0.0) {
                if (next && t + 1 < WARPS) publish(a[r], k + 1);
                if (next && t + 1 == WARPS) publish(a[r + 1 < NR ? r + 1 : r], k + 1);
                continue;
            }
            double vj[NC], s[8];
#pragma unroll
            for (int c = C0; c < NC; ++c) vj[c] = v[lane + 32 * c];
            // rows before WARPS r are done: NR - r values a lane
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                s[q] = 0.0;
                if (r + q < NR)
#pragma unroll
                    for (int c = C0; c < NC; ++c) s[q] += a[r + q < NR ? r + q : 0][c] * vj[c];
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
            for (int c = C0; c < NC; ++c) {
                const int j = lane + 32 * c;
                wj[c] = j > k ? p[j] : 0.0;
                vp += vj[c] * wj[c];
            }
            const double half = 0.5 * tau * (tau * warp_sum(vp));
#pragma unroll
            for (int c = C0; c < NC; ++c) wj[c] = tau * wj[c] - half * vj[c];
            auto update = [&](double (&row)[NC], int i) {
                const double vi = v[i], wi = i > k ? tau * p[i] - half * vi : 0.0;
#pragma unroll
                for (int c = C0; c < NC; ++c) row[c] -= vi * wj[c] + wi * vj[c];
            };
            // row k + 1 first: the next reflector is a serial chain that the other warps' updates hide
            int done = -1;
            if (next) {
                if (t + 1 < WARPS) {
                    update(a[r], warp + WARPS * r);
                    publish(a[r], k + 1);
                    done = 0;
                } else {
                    update(a[r + 1 < NR ? r + 1 : r], warp + WARPS * (r + 1));
                    publish(a[r + 1 < NR ? r + 1 : r], k + 1);
                    done = 1;
                }
            }
#pragma unroll
            for (int q = 0; q < NR; ++q)
                if (r + q < NR && q != done) update(a[r + q < NR ? r + q : 0], warp + WARPS * (r + q));
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
            // a block of 8 rows holds both halves of a merge of 4 + 4
            const int nt = column_list<NC>(sv, sv.top, o, K, w < 8 ? 3 : 1), nb = column_list<NC>(sv, sv.bot, o, K, 2);
            if (lane == 0) {
                sv.K[mm] = K;
                sv.ntop[mm] = nt;
                sv.nbot[mm] = nb;
                sv.rho[mm] = rho;
            }
        }
        __syncthreads();
        const int K = merging ? sv.K[m] : 0;
        const int Kw = __reduce_max_sync(0xffffffffu, K), Kc = max(K, 1);
        const bool live = jj < K;
        const int jc = live ? jj : 0;
        const double *kd = sv.kd + (merging ? off : 0), *kz = sv.kz + (merging ? off : 0);
        int org = 0;
        double x = 0.0;
        if (Kw > 0 && !secular_roots(live, Kc, Kw, jc, kd, kz, merging ? sv.rho[m] : 1.0, q4, &org, &x)) sv.bad = 2;
        if (live && q4 == 0) {
            sv.org[pos] = org;
            sv.x[pos] = x;
        }
        __syncthreads();
        // the z for which these roots are exact: z_i^2 = prod_j (lambda_j - d_i) / prod_(j != i) (d_j - d_i), up to a factor
        const int base = merging ? off : 0;
        {
            const double di = kd[jc];
            double pr = 1.0;
            for (int j0 = q4; j0 < Kw; j0 += 16) {  // four ratios share a division
                double num = 1.0, den = 1.0;
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int j = j0 + 4 * u, jm = min(j, Kc - 1);
                    const double a = (kd[live ? sv.org[base + jm] : 0] - di) + sv.x[base + jm];
                    const double b = kd[jm < jj ? jm : min(jm + 1, Kc - 1)] - di;
                    num *= j < K ? a : 1.0;
                    den *= j < K && !(j >= jj && j == K - 1) ? b : 1.0;
                }
                pr *= num / den;
            }
            __syncwarp();
            pr = quad_product(pr);
            if (live && q4 == 0) sv.zh[pos] = copysign(sqrt(fabs(pr)), kz[jc]);
        }
        __syncthreads();
        // vectors of the merged problem, 64 columns at a time, and their product with the old ones
        constexpr int CHUNKS = NC > 2 ? 2 : 1;
        const double o = kd[org], lam = o + x;
        auto vectors = [&](int ch) {
            const bool mine = live && jj / 64 == ch;
            if (__any_sync(0xffffffffu, mine)) {
                double ss = 0.0;
                double *col = U + base * up + jj - 64 * ch;
                for (int i0 = 0; i0 < Kw; i0 += 8) {  // two elements share a division
                    const int i = min(i0 + q4, Kc - 1), i2 = min(i0 + q4 + 4, Kc - 1);
                    const double a = (kd[i] - o) - x, b = (kd[i2] - o) - x, r = 1.0 / (a * b);
                    const double u1 = sv.zh[base + i] * (b * r), u2 = sv.zh[base + i2] * (a * r);
                    if (mine && i0 + q4 < K) {
                        col[i * up] = u1;
                        ss += u1 * u1;
                    }
                    if (mine && i0 + q4 + 4 < K) {
                        col[i2 * up] = u2;
                        ss += u2 * u2;
                    }
                }
                ss = quad_sum(ss);
                if (mine && q4 == 0) sv.scale[pos] = 1.0 / sqrt(ss);
            }
        };
        if (2 * w >= 8) {
            // warp: rows 8 warp .. + 7, inside one merge
            const int r0 = 8 * warp, ro = r0 / (2 * w) * (2 * w), rm = r0 / (2 * w);
            const bool rows = r0 < n && ro + w < n;
            const int RK = rows ? sv.K[rm] : 0;
            const bool upper = r0 < ro + w;
            const int cnt = rows ? (upper ? sv.ntop[rm] : sv.nbot[rm]) : 0;
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
                if (cols > 0 && cnt > 0) {
                    int next = list[min(lane & 3, cnt - 1)];
                    for (int k0 = 0; k0 < cnt; k0 += 4) {
                        const int cur = next;
                        next = list[min(k0 + 4 + (lane & 3), cnt - 1)];
                        const double av = k0 + (lane & 3) < cnt ? Z[(r0 + (lane >> 2)) * zp + (cur >> 8)] : 0.0;
                        const double *ur = U + (ro + (cur & 255)) * up + (lane >> 2);
#pragma unroll
                        for (int t = 0; t < 8; ++t)
                            if (8 * t < cols) dmma884(acc[ch][t][0], acc[ch][t][1], av, ur[8 * t]);
                    }
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
        if (live && q4 == 0) sv.d[sv.slot[pos]] = lam;
        __syncthreads();
    }

    // ---------------- 3. reflectors, blocks of eight from the last to the first, on the warp's eight columns:
    // H_k ... H_(k+7) = 1 - R T R^T with the reflectors as the columns of R and a triangular T
    // block b: eight rows (reflectors) of the elements from 8 b on, pitch 4 mod 8 doubles
    auto block = [&](int b) { return U + 8 * (b * (lay.rows + 4) - 4 * b * (b - 1)); };
    const int blocks = n > 2 ? (n - 2 + 7) / 8 : 0;
    for (int k = warp; k < 8 * blocks; k += WARPS) {
        const int b = k / 8, len = lay.rows - 8 * b;
        double *dst = block(b) + (k & 7) * (len + 4);
        for (int i = lane; i < len; i += 32) {
            const int j = 8 * b + i;
            dst[i] = k < n - 2 && j > k && j < n ? V[(size_t)k * n + j] : 0.0;
        }
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
    if (pos < n && q4 == 0) {
        W[rank] = ev * back;
        sv.ord[pos] = rank;
    }
    const int fr = lane >> 2, fc = lane & 3;  // fragment row (A) or column (B), and the other index
    double *tm = sv.e;                        // T of block b at 64 b
    if (warp < blocks) {
        const int len = lay.rows - 8 * warp, pitch = len + 4;
        const double *R = block(warp);
        double g0 = 0.0, g1 = 0.0;
        for (int i = 0; i < len; i += 4) {
            const double x = R[fr * pitch + i + fc];
            dmma884(g0, g1, x, x);
        }
        double *T = tm + 64 * warp;
        T[fr * 8 + 2 * fc] = g0;
        T[fr * 8 + 2 * fc + 1] = g1;
        __syncwarp();
        // row l of T: T_lj = -T_jj sum_(m < j) T_lm (R^T R)_mj
        double row[8];
        const int l = lane & 7;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const double tj = 8 * warp + j < n - 2 ? sv.tau[8 * warp + j] : 0.0;
            double x = 0.0;
#pragma unroll
            for (int m = 0; m < j; ++m) x += row[m] * T[m * 8 + j];
            row[j] = j < l ? 0.0 : (j == l ? tj : -tj * x);
        }
        __syncwarp();
        if (lane < 8)
#pragma unroll
            for (int j = 0; j < 8; ++j) T[l * 8 + j] = row[j];
    }
    __syncthreads();
    const int c0 = 8 * warp;
    if (c0 < n) {
        // accumulator layout (row fr, columns 2 fc, + 1) to B operand (row 4 s + fc, column fr)
        auto operand = [&](double d0, double d1, int s) {
            const int src = (4 * s + fc) * 4 + (fr >> 1);
            const double x0 = __shfl_sync(0xffffffffu, d0, src), x1 = __shfl_sync(0xffffffffu, d1, src);
            return fr & 1 ? x1 : x0;
        };
        for (int b = blocks - 1; b >= 0; --b) {
            const int len = lay.rows - 8 * b, pitch = len + 4;
            const double *R = block(b), *T = tm + 64 * b;
            double *Zb = Z + 8 * b * zp + c0;
            double w0 = 0.0, w1 = 0.0, u0 = 0.0, u1 = 0.0;
#pragma unroll 4
            for (int i = 0; i < len; i += 8) {
                dmma884(w0, w1, R[fr * pitch + i + fc], Zb[(i + fc) * zp + fr]);
                dmma884(u0, u1, R[fr * pitch + i + 4 + fc], Zb[(i + 4 + fc) * zp + fr]);
            }
            w0 += u0;
            w1 += u1;
            double x0 = 0.0, x1 = 0.0;
            dmma884(x0, x1, T[fr * 8 + fc], operand(w0, w1, 0));
            dmma884(x0, x1, T[fr * 8 + 4 + fc], operand(w0, w1, 1));
            const double b0 = -operand(x0, x1, 0), b1 = -operand(x0, x1, 1);
            __syncwarp();
#pragma unroll 4
            for (int i = 0; i < len; i += 8) {
                double2 *z = reinterpret_cast<double2 *>(Zb + (i + fr) * zp + 2 * fc);
                double2 x = *z;
                dmma884(x.x, x.y, R[fc * pitch + i + fr], b0);
                dmma884(x.x, x.y, R[(4 + fc) * pitch + i + fr], b1);
                *z = x;
            }
            __syncwarp();
        }
        for (int c = c0; c < min(c0 + 8, n); ++c) {
            double *dst = V + (size_t)sv.ord[c] * n;
            for (int i = lane; i < n; i += 32) dst[i] = Z[i * zp + c];
        }
    }
    if (tid == 0) info[blockIdx.x] = sv.bad;
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
