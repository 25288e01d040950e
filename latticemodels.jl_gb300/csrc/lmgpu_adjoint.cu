// Adjoint of the Chebyshev evolution: gradients of a density loss with respect to the
// on-site potentials and the field amplitudes.
//
// Forward step n:  psi_{n+1} = U_n psi_n,  U_n = e^{-ib dt} sum_k c_k T_k(H~_n),  H~ = (H - b)/a
// with a, b, K fixed (frozen spectral bounds), so U_n is an exact polynomial in H_n and its
// discrete adjoint is exact.  With the co-state lambda_{n+1} = dL/dpsi*_{n+1} (L real):
//
//   lambda_n = U_n^dagger lambda_{n+1}           (the propagator with conjugate coefficients)
//   dL/dtheta += Re e^{-ib dt} sum_{k>=1} < beta_k , s_k >,   s_1 = D~ T_0,  s_k = 2 D~ T_{k-1}
//
// where D~ = (dH/dtheta)/a and beta is the adjoint of the three-term recurrence,
//   beta_k = conj(c_k) lambda + 2 H~ beta_{k+1} - beta_{k+2},  beta_{K+1} = beta_{K+2} = 0.
// For an on-site potential V_i, < beta, D~ T > = conj(beta_i) T_i / a summed over kets; for a
// field amplitude A, dH[s, s+e]/dA = -2 pi i LI_e(A = 1) H[s, s+e] on every bond.
//
// lm_adjoint_step recomputes T_0 .. T_{K-1} from psi_n, then runs the beta recurrence and the gradient
// sums (FP64 results; c32 sums in double-float): ComplexF32 kets that fit on chip take one lattice-resident
// launch per recurrence and one kernel for the sums over all orders, the others one launch per order,
// beta and its sums in one pass.  The caller applies U^dagger to lambda with a solver updated for -dt
// (the same polynomial with conjugate coefficients).
#include <cuda_runtime.h>
#include <math.h>

#include <algorithm>
#include <new>
#include <vector>

#include "lmgpu_internal.cuh"
#include "lmgpu_order.cuh"
#include "lmgpu_resident.cuh"

namespace lmgpu {

// out = alpha * (2H~) tp - tpp + w * lam   (tables hold 2H/a and 2(V-b)/a; tpp, lam optional)
// w = conj(c_k): (s, 0) for even k, (0, s) for odd k (conj(-i s) = i s).
// With y non-null, also y += cy * out (the real-coefficient Chebyshev series of lm_cheb_apply).
// XR: every x-hop is real, so the x-neighbour terms take 2 FMAs instead of 4.
template <typename R, bool XR>
__global__ void __launch_bounds__(256) adj_recur_kernel(Geom g, const typename CT<R>::V* __restrict__ hop2,
                                                        const R* __restrict__ diag2,
                                                        const typename CT<R>::V* __restrict__ tp,
                                                        const typename CT<R>::V* __restrict__ tpp,
                                                        const typename CT<R>::V* __restrict__ lam,
                                                        typename CT<R>::V* __restrict__ out, int64_t ld, int64_t M,
                                                        R alpha, R w_re, R w_im, typename CT<R>::V* __restrict__ y,
                                                        R cy) {
    typedef typename CT<R>::V V;
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= g.N) return;
    const Nbr nb = neighbours(g, s);
    const V z = CT<R>::make(0, 0);
    const V hxp = nb.hxp ? hop2[s] : z, hyp = nb.hyp ? hop2[g.N + s] : z;
    V t = nb.hxm ? hop2[nb.xm] : z;
    const V hxm = CT<R>::make(t.x, -t.y);
    t = nb.hym ? hop2[g.N + nb.ym] : z;
    const V hym = CT<R>::make(t.x, -t.y);
    const R d = diag2[s];
    for (int64_t m = blockIdx.y; m < M; m += gridDim.y) {
        const int64_t o = m * ld;
        V acc = z;
        if (tp) {
            const V v0 = tp[o + s], vxp = tp[o + nb.xp], vxm = tp[o + nb.xm], vyp = tp[o + nb.yp], vym = tp[o + nb.ym];
            if (XR) {
                acc.x = fma(hxp.x, vxp.x, acc.x);
                acc.y = fma(hxp.x, vxp.y, acc.y);
                acc.x = fma(hxm.x, vxm.x, acc.x);
                acc.y = fma(hxm.x, vxm.y, acc.y);
            } else {
                acc.x = fma(hxp.x, vxp.x, acc.x); acc.x = fma(-hxp.y, vxp.y, acc.x);
                acc.y = fma(hxp.x, vxp.y, acc.y); acc.y = fma(hxp.y, vxp.x, acc.y);
                acc.x = fma(hxm.x, vxm.x, acc.x); acc.x = fma(-hxm.y, vxm.y, acc.x);
                acc.y = fma(hxm.x, vxm.y, acc.y); acc.y = fma(hxm.y, vxm.x, acc.y);
            }
            acc.x = fma(hyp.x, vyp.x, acc.x); acc.x = fma(-hyp.y, vyp.y, acc.x);
            acc.y = fma(hyp.x, vyp.y, acc.y); acc.y = fma(hyp.y, vyp.x, acc.y);
            acc.x = fma(hym.x, vym.x, acc.x); acc.x = fma(-hym.y, vym.y, acc.x);
            acc.y = fma(hym.x, vym.y, acc.y); acc.y = fma(hym.y, vym.x, acc.y);
            acc.x = fma(d, v0.x, acc.x);
            acc.y = fma(d, v0.y, acc.y);
            acc.x *= alpha;
            acc.y *= alpha;
        }
        if (tpp) {
            const V q = tpp[o + s];
            acc.x -= q.x;
            acc.y -= q.y;
        }
        if (lam) {
            const V l = lam[o + s];
            acc.x = fma(w_re, l.x, fma(-w_im, l.y, acc.x));
            acc.y = fma(w_re, l.y, fma(w_im, l.x, acc.y));
        }
        out[o + s] = acc;
        if (y) {
            V t = y[o + s];
            t.x = fma(cy, acc.x, t.x);
            t.y = fma(cy, acc.y, t.y);
            y[o + s] = t;
        }
    }
}

// out = alpha (2H~) tp - tpp + w lam over an n x M block (the three-term Chebyshev recurrence
// and its adjoint; KPM uses it for the moments).  out may alias tpp.
cudaError_t launch_stencil_recur(lm_ctx* ctx, const Geom& g, int precision, const void* hop2, const void* diag2,
                                 const void* tp, const void* tpp, const void* lam, void* out, int64_t ld, int64_t M,
                                 double alpha, double wre, double wim, void* y, double cy, bool xreal) {
    if (M <= 0 || g.N <= 0) return cudaSuccess;
    const dim3 grid((unsigned)((g.N + 255) / 256), (unsigned)(M < 65535 ? M : 65535));
#define LM_RECUR(R, V, XRV)                                                                                   \
    adj_recur_kernel<R, XRV><<<grid, 256, 0, ctx->stream>>>(g, (const V*)hop2, (const R*)diag2, (const V*)tp, \
                                                           (const V*)tpp, (const V*)lam, (V*)out, ld, M,        \
                                                           (R)alpha, (R)wre, (R)wim, (V*)y, (R)cy)
    if (precision == LM_C64) {
        if (xreal) LM_RECUR(double, double2, true);
        else LM_RECUR(double, double2, false);
    } else {
        if (xreal) LM_RECUR(float, float2, true);
        else LM_RECUR(float, float2, false);
    }
#undef LM_RECUR
    ctx->launches++;
    return cudaGetLastError();
}

// The on-site and field terms of one order at a site from its sums v, before the factor f; the field
// term is f times the real part.
__device__ __forceinline__ double grad_site_V(const double (&v)[10], double ph_re, double ph_im) {
    return ph_re * v[0] - ph_im * v[1];
}

__device__ __forceinline__ double grad_site_A(const Geom& g, const Nbr& nb, int64_t s, const double (&v)[10],
                                              const double2* dhop, double ph_re, double ph_im, double f) {
    const double2 zz = make_double2(0.0, 0.0);
    const double2 D[4] = {nb.hxp ? dhop[s] : zz, nb.hyp ? dhop[g.N + s] : zz, nb.hxm ? dhop[nb.xm] : zz,
                          nb.hym ? dhop[g.N + nb.ym] : zz};
    double zr = 0.0, zi = 0.0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const double sr = v[2 + 2 * q], si = v[3 + 2 * q];
        if (q < 2) {  // D S
            zr += D[q].x * sr - D[q].y * si;
            zi += D[q].x * si + D[q].y * sr;
        } else {      // conj(D) S
            zr += D[q].x * sr + D[q].y * si;
            zi += D[q].x * si - D[q].y * sr;
        }
    }
    return f * (ph_re * zr - ph_im * zi);
}

// A block's gradient contributions of one order from its sums v: gV_part of its 32 sites and gA_part of
// the block, one writer per entry and launch (one warp calls this).
__device__ __forceinline__ void grad_block_out(const Geom& g, const Nbr& nb, int64_t s, int lane, const double (&v)[10],
                                               const double2* dhop, double ph_re, double ph_im, double f,
                                               double* gV_part, double* gA_part) {
    double ga = 0.0;
    if (s < g.N) {
        double* gv = gV_part + (int64_t)blockIdx.y * g.N + s;
        *gv = fma(f, grad_site_V(v, ph_re, ph_im), *gv);
        if (dhop) ga = grad_site_A(g, nb, s, v, dhop, ph_re, ph_im, f);
    }
    if (gA_part) {
        for (int o = 16; o > 0; o >>= 1) ga += __shfl_down_sync(0xffffffffu, ga, o);
        if (lane == 0) gA_part[(int64_t)blockIdx.y * gridDim.x + blockIdx.x] += ga;
    }
}

// One order k of the adjoint, fused: the beta recurrence and the gradient sums in one pass.
//   beta_k = conj(c_k) lambda + (2H~) beta_{k+1} - beta_{k+2}         (written to bk)
//   gV[s] += f Re( ph * sum_m conj(beta_k,sm) T_sm )
//   gA    += f Re( ph * sum_s [ D[s,s+x] S1x + D[s,s+y] S1y + conj(D[s-x,s]) S2x + conj(D[s-y,s]) S2y ] )
//            S1e = sum_m conj(beta_k,sm) T_{s+e,m},  S2e = sum_m conj(beta_k,sm) T_{s-e,m}
// with T = T_{k-1}, ph = e^{-ib dt}, f = 1/a (k = 1) or 2/a (k >= 2), D = dH/dA per bond (owned
// by its source site).  Every bond enters twice -- conj(b_s) D T_j at its source s and
// conj(b_j) conj(D) T_s at its destination j -- so a thread needs only its own beta_k and
// read-only neighbours of T.  A block owns 32 sites and one chunk of the kets (blockIdx.y);
// its 8 warps split the chunk and their partial sums are added in warp order.  gV_part and
// gA_part have one writer per entry per launch and lm_adjoint_gradients adds them in chunk
// and block order, so the gradients are bit-reproducible.  c32 sums are double-float.
template <typename R>
__global__ void __launch_bounds__(256, sizeof(R) == sizeof(float) ? 3 : 2) adj_beta_grad_kernel(
    Geom g, const typename CT<R>::V* __restrict__ hop2, const R* __restrict__ diag2,
    const typename CT<R>::V* __restrict__ b1, const typename CT<R>::V* __restrict__ b2,
    const typename CT<R>::V* __restrict__ lam, typename CT<R>::V* __restrict__ bk, R w_re, R w_im,
    const double2* __restrict__ dhop, const typename CT<R>::V* __restrict__ T, int64_t ld, int64_t M, int64_t mchunk,
    double ph_re, double ph_im, double f, double* __restrict__ gV_part, double* __restrict__ gA_part) {
    typedef typename CT<R>::V V;
    __shared__ double red[8][10][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t s = (int64_t)blockIdx.x * 32 + lane;
    const int64_t m0 = (int64_t)blockIdx.y * mchunk, m1 = min(M, m0 + mchunk);
    Acc<R> a[10];  // conj(b)T_s (re, im); S1x; S1y; S2x; S2y
    Nbr nb;
    if (s < g.N) {
        nb = neighbours(g, s);
        const V z = CT<R>::make(0, 0);
        const V hxp = nb.hxp ? hop2[s] : z, hyp = nb.hyp ? hop2[g.N + s] : z;
        V t = nb.hxm ? hop2[nb.xm] : z;
        const V hxm = CT<R>::make(t.x, -t.y);
        t = nb.hym ? hop2[g.N + nb.ym] : z;
        const V hym = CT<R>::make(t.x, -t.y);
        const R d = diag2[s];
        for (int64_t m = m0 + warp; m < m1; m += 8) {
            const int64_t o = m * ld;
            V acc = z;
            if (b1) {
                const V v0 = b1[o + s], vxp = b1[o + nb.xp], vxm = b1[o + nb.xm], vyp = b1[o + nb.yp], vym = b1[o + nb.ym];
                acc.x = fma(hxp.x, vxp.x, acc.x); acc.x = fma(-hxp.y, vxp.y, acc.x);
                acc.y = fma(hxp.x, vxp.y, acc.y); acc.y = fma(hxp.y, vxp.x, acc.y);
                acc.x = fma(hxm.x, vxm.x, acc.x); acc.x = fma(-hxm.y, vxm.y, acc.x);
                acc.y = fma(hxm.x, vxm.y, acc.y); acc.y = fma(hxm.y, vxm.x, acc.y);
                acc.x = fma(hyp.x, vyp.x, acc.x); acc.x = fma(-hyp.y, vyp.y, acc.x);
                acc.y = fma(hyp.x, vyp.y, acc.y); acc.y = fma(hyp.y, vyp.x, acc.y);
                acc.x = fma(hym.x, vym.x, acc.x); acc.x = fma(-hym.y, vym.y, acc.x);
                acc.y = fma(hym.x, vym.y, acc.y); acc.y = fma(hym.y, vym.x, acc.y);
                acc.x = fma(d, v0.x, acc.x);
                acc.y = fma(d, v0.y, acc.y);
            }
            if (b2) {
                const V q = b2[o + s];
                acc.x -= q.x;
                acc.y -= q.y;
            }
            const V l = lam[o + s];
            acc.x = fma(w_re, l.x, fma(-w_im, l.y, acc.x));
            acc.y = fma(w_re, l.y, fma(w_im, l.x, acc.y));
            bk[o + s] = acc;
            const V b = acc, ts = T[o + s];
            a[0].add_prod(b.x, ts.x);
            a[0].add_prod(b.y, ts.y);
            a[1].add_prod(b.x, ts.y);
            a[1].add_prod(-b.y, ts.x);
            if (dhop) {
                const V tn[4] = {T[o + nb.xp], T[o + nb.yp], T[o + nb.xm], T[o + nb.ym]};
#pragma unroll
                for (int q = 0; q < 4; ++q) {  // conj(b) T_n
                    a[2 + 2 * q].add_prod(b.x, tn[q].x);
                    a[2 + 2 * q].add_prod(b.y, tn[q].y);
                    a[3 + 2 * q].add_prod(b.x, tn[q].y);
                    a[3 + 2 * q].add_prod(-b.y, tn[q].x);
                }
            }
        }
    }
#pragma unroll
    for (int q = 0; q < 10; ++q) red[warp][q][lane] = a[q].get();
    __syncthreads();
    if (warp != 0) return;
    double v[10];
#pragma unroll
    for (int q = 0; q < 10; ++q) {
        double t = 0.0;
        for (int w = 0; w < 8; ++w) t += red[w][q][lane];
        v[q] = t;
    }
    grad_block_out(g, nb, s, lane, v, dhop, ph_re, ph_im, f, gV_part, gA_part);
}

// The gradient sums of a whole step from all its T_{k-1} and beta_k (which the lattice-resident kernels
// wrote to HBM): order by order the sums of adj_beta_grad_kernel<float>, term for term, so that both forms
// give the same bits.
//
// What bounds it: the FP32 pipe, 20 double-float products (10 operations each) per site, ket and order, as
// packed pairs (re, im): 140 us at that pipe's rate on 64 x 64 sites with 1024 kets and K = 6, and at a
// block's end the FP64 pipe's latency (a warp-wide DADD holds a partition for 64 clocks), so each of the
// 8 warps adds one sum's partials and the pairs become doubles by integer operations.  An order is a block of
// its own (6144 blocks; all orders in turn made 1024, whose last wave was a quarter full) and
// adj_fold_kernel adds them.  The step took 5 recurrence launches of 41 us and 6 fused passes of 102 us; now
// T_k and beta_k take 61 + 66 us on chip (each writes 200 MB) and the sums 214 + 5 us (293 us with the
// orders in turn and scalar products; 227 to 253 us with the loads by cp.async; 272 us with 2 blocks per SM).
struct GradOrders {
    const float2* T[kResMaxK];      // T_0 .. T_{K-1}
    const float2* b[kResMaxK + 1];  // beta_1 .. beta_K
};

__global__ void __launch_bounds__(256, 3) adj_sums_kernel(Geom g, const __grid_constant__ GradOrders ord,
                                                          const double2* __restrict__ dhop, int64_t ld, int64_t M,
                                                          int64_t mchunk, double ph_re, double ph_im, double inv_a,
                                                          double* __restrict__ sums_V, double* __restrict__ sums_A) {
    __shared__ double red[8][10][32];
    __shared__ double tot[10][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int k = (int)blockIdx.z + 1;
    const int64_t s = (int64_t)blockIdx.x * 32 + lane;
    const int64_t m0 = (int64_t)blockIdx.y * mchunk, m1 = min(M, m0 + mchunk);
    const bool on = s < g.N;
    Nbr nb;
    Acc2 a[5];  // (re, im) of conj(b)T_s; S1x; S1y; S2x; S2y
    if (on) {
        nb = neighbours(g, s);
        const int xp = (int)(nb.xp - s), yp = (int)(nb.yp - s), xm = (int)(nb.xm - s), ym = (int)(nb.ym - s);
        // beta, T and T's neighbours of the next ket are loaded while this one is summed
        int n = m0 + warp < m1 ? (int)((m1 - m0 - warp + 7) / 8) : 0;
        const float2* T = ord.T[k - 1] + (m0 + warp) * ld + s;
        const float2* bk = ord.b[k] + (m0 + warp) * ld + s;
        auto load = [&](float2 (&d)[6]) {
            d[0] = __ldg(bk);
            d[1] = __ldg(T);
            if (dhop) {
                d[2] = __ldg(T + xp);
                d[3] = __ldg(T + yp);
                d[4] = __ldg(T + xm);
                d[5] = __ldg(T + ym);
            }
            T += 8 * ld;
            bk += 8 * ld;
        };
        auto sum = [&](const float2 (&d)[6]) {
            const float2 b = d[0];
            const float2 b1 = make_float2(b.x, b.x), n1 = make_float2(-b.x, -b.x);
            const float2 b2 = make_float2(b.y, -b.y), n2 = make_float2(-b.y, b.y);
#pragma unroll
            for (int q = 0; q < 5; ++q) {  // conj(b) T at the site and its neighbours
                if (q > 0 && !dhop) break;
                const float2 t = d[1 + q];
                a[q].add_prod(b1, n1, t);
                a[q].add_prod(b2, n2, make_float2(t.y, t.x));
            }
        };
        float2 v[6], w[6];
        if (n > 0) load(v);
        while (n > 0) {
            if (n > 1) load(w);
            sum(v);
            if (--n == 0) break;
            if (n > 1) load(v);
            sum(w);
            --n;
        }
    }
#pragma unroll
    for (int q = 0; q < 5; ++q) {
        red[warp][2 * q][lane] = widen(a[q].hi.x) + widen(a[q].lo.x);
        red[warp][2 * q + 1][lane] = widen(a[q].hi.y) + widen(a[q].lo.y);
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 2; ++r) {  // sum q of the block, warps in order
        const int q = warp + 8 * r;
        if (q < 10 && (q < 2 || dhop)) {
            double t = red[0][q][lane];
#pragma unroll
            for (int u = 1; u < 8; ++u) t += red[u][q][lane];
            tot[q][lane] = t;
        }
    }
    __syncthreads();
    if (warp != 0) return;
    double t[10], ga = 0.0;
#pragma unroll
    for (int q = 0; q < 10; ++q) t[q] = q < 2 || dhop ? tot[q][lane] : 0.0;
    const int64_t row = (int64_t)(k - 1) * gridDim.y + blockIdx.y;
    if (on) {
        sums_V[row * g.N + s] = grad_site_V(t, ph_re, ph_im);
        if (dhop) ga = grad_site_A(g, nb, s, t, dhop, ph_re, ph_im, k == 1 ? inv_a : 2.0 * inv_a);
    }
    if (dhop) {
        for (int o = 16; o > 0; o >>= 1) ga += __shfl_down_sync(0xffffffffu, ga, o);
        if (lane == 0) sums_A[row * gridDim.x + blockIdx.x] = ga;
    }
}

// Adds the orders' terms to the gradients' parts, K first, as the per-order kernels do: nV entries of gV_part
// and nA of gA_part (null without a field derivative).
__global__ void adj_fold_kernel(int K, int64_t nV, int64_t nA, double inv_a, const double* __restrict__ sums_V,
                                const double* __restrict__ sums_A, double* __restrict__ gV_part,
                                double* __restrict__ gA_part) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < nV) {
        double t = gV_part[i];
        for (int k = K; k >= 1; --k) t = fma(k == 1 ? inv_a : 2.0 * inv_a, sums_V[(int64_t)(k - 1) * nV + i], t);
        gV_part[i] = t;
    }
    if (gA_part && i < nA) {
        double t = gA_part[i];
        for (int k = K; k >= 1; --k) t += sums_A[(int64_t)(k - 1) * nA + i];
        gA_part[i] = t;
    }
}

// rho_s = sum_m |psi_sm|^2; loss = sum_s (rho_s - target_s)^2; lambda = 4 (rho_s - target_s) psi.
// A block owns 32 sites (8 warps split the kets); loss_part[block] receives its partial loss.
template <typename R>
__global__ void __launch_bounds__(256) adj_seed_kernel(int64_t N, const typename CT<R>::V* __restrict__ psi,
                                                       typename CT<R>::V* __restrict__ lam, int64_t ld, int64_t M,
                                                       const double* __restrict__ target,
                                                       double* __restrict__ loss_part) {
    typedef typename CT<R>::V V;
    __shared__ double red[8][32];
    __shared__ double diff_s[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t s = (int64_t)blockIdx.x * 32 + lane;
    Acc<R> acc;
    if (s < N)
        for (int64_t m = warp; m < M; m += 8) {
            const V v = psi[m * ld + s];
            acc.add_prod(v.x, v.x);
            acc.add_prod(v.y, v.y);
        }
    red[warp][lane] = acc.get();
    __syncthreads();
    if (warp == 0) {
        double rho = 0.0;
        for (int w = 0; w < 8; ++w) rho += red[w][lane];
        const double diff = s < N ? rho - target[s] : 0.0;
        diff_s[lane] = diff;
        double l = diff * diff;
        for (int o = 16; o > 0; o >>= 1) l += __shfl_down_sync(0xffffffffu, l, o);
        if (lane == 0) loss_part[blockIdx.x] = l;
    }
    __syncthreads();
    if (s < N) {
        const R fct = (R)(4.0 * diff_s[lane]);
        for (int64_t m = warp; m < M; m += 8) {
            const V v = psi[m * ld + s];
            lam[m * ld + s] = CT<R>::make(fct * v.x, fct * v.y);
        }
    }
}

// dH[s, s+e]/dA_c = -2 pi i LI_c(A_c = 1) H[s, s+e] for field component c.
__global__ void flux_derivative_kernel(Geom g, FieldSet f, int comp, const double2* __restrict__ hop,
                                       double2* __restrict__ dhop) {
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= g.N) return;
    FieldSet one = f;
    one.n = 1;
    one.c[0] = f.c[comp];
    one.amp[0] = 1.0;
    const int64_t xi = s / g.Ly, yi = s - xi * g.Ly;
    const double x1 = (double)(xi + 1), y1 = (double)(yi + 1);
    const int dir = blockIdx.y;  // a direction per thread, as in the assembly
    const double x2 = dir == 0 ? x1 + 1.0 : x1, y2 = dir == 0 ? y1 : y1 + 1.0;
    const double li = field_line_integral(g, one, x1, y1, x2, y2);
    const double2 h = hop[dir * g.N + s];
    const double w = -2.0 * M_PI * li;  // d/dA e^{-2 pi i A li} = -2 pi i li (...)
    dhop[dir * g.N + s] = make_double2(-w * h.y, w * h.x);  // (i w) h
}

}  // namespace lmgpu

using namespace lmgpu;

struct lm_adjoint {
    lm_ctx* ctx = nullptr;
    int64_t n = 0, m = 0;
    int precision = LM_C64;
    size_t elem = 16;
    int K = 0;
    int lean_K = 1 << 30;  // from this order on the blocks of the lattice-resident form did not fit
    std::vector<void*> T;  // T_0 .. T_{K-1} (T_0 aliases psi during a step)
    std::vector<void*> B;  // beta_k by order (lattice-resident form) or three rotating blocks
    double* d_gV = nullptr;     // per ket chunk, one partial per site (nchunk x n)
    double* d_gA = nullptr;     // per gradient slot, one partial per (chunk, 32-site block)
    int nslots = 0;
    int64_t nblk = 0;           // 32-site blocks of the gradient and seed kernels
    int64_t nchunk = 1, mchunk = 1;  // ket chunks of the gradient kernel (grid y) and their size
    double* d_loss = nullptr;   // one partial per 32-site block (nblk)
    double* d_target = nullptr;
    double2* d_dhop = nullptr;
    double* d_sums = nullptr;   // lattice-resident form: the orders' terms of gV and gA before they are added
};

static void adj_free_stack(lm_adjoint* a) {
    for (size_t i = 1; i < a->T.size(); ++i)
        dev_free(a->ctx, a->T[i]);
    a->T.clear();
    for (auto& b : a->B)
        dev_free(a->ctx, b);
    a->B.clear();
    dev_free(a->ctx, a->d_sums);
    a->d_sums = nullptr;
    a->K = 0;
}

static int adj_alloc(lm_ctx* ctx, void** p, size_t bytes) {
    if (dev_alloc(ctx, p, bytes) != cudaSuccess) {
        *p = nullptr;
        cudaGetLastError();
        return set_err(ctx, LM_ERR_OOM, "lm_adjoint: device allocation failed");
    }
    return LM_OK;
}

static int adj_ensure_stack(lm_adjoint* a, int K, bool all_beta) {
    const size_t nb = all_beta ? (size_t)K + 1 : 3;
    if (a->K == K && !a->T.empty() && a->B.size() == nb) return LM_OK;
    adj_free_stack(a);
    const size_t bytes = a->elem * (size_t)a->n * (size_t)a->m;
    a->T.assign((size_t)K, nullptr);
    for (int k = 1; k < K; ++k) {
        int rc = adj_alloc(a->ctx, &a->T[(size_t)k], bytes);
        if (rc != LM_OK) return rc;
    }
    a->B.assign(nb, nullptr);
    for (size_t k = all_beta ? 1 : 0; k < nb; ++k) {
        int rc = adj_alloc(a->ctx, &a->B[k], bytes);
        if (rc != LM_OK) return rc;
    }
    if (all_beta) {
        int rc = adj_alloc(a->ctx, (void**)&a->d_sums, sizeof(double) * (size_t)K * (size_t)a->nchunk * (size_t)(a->n + a->nblk));
        if (rc != LM_OK) return rc;
        // the other form takes K - 3 blocks less: what a program still allocates (the scratch of its states,
        // a checkpoint) must not fail for them
        size_t free_b = 0, total = 0;
        if (cudaMemGetInfo(&free_b, &total) == cudaSuccess && free_b < 4 * bytes)
            return set_err(a->ctx, LM_ERR_OOM, "lm_adjoint: no room beside the blocks of all orders");
    }
    a->K = K;
    return LM_OK;
}

extern "C" {

int lm_adjoint_create(lm_ctx* ctx, int64_t n, int64_t m, int precision, int nslots, lm_adjoint** out) {
    if (!ctx) return LM_ERR_ARG;
    if (!out) return set_err(ctx, LM_ERR_ARG, "lm_adjoint_create: null output");
    *out = nullptr;
    if (n < 1 || m < 1 || nslots < 0) return set_err(ctx, LM_ERR_ARG, "lm_adjoint_create: bad sizes");
    if (precision != LM_C64 && precision != LM_C32) return set_err(ctx, LM_ERR_ARG, "lm_adjoint_create: unknown precision");
    lm_adjoint* a = new (std::nothrow) lm_adjoint();
    if (!a) return set_err(ctx, LM_ERR_OOM, "host allocation");
    a->ctx = ctx;
    a->n = n;
    a->m = m;
    a->precision = precision;
    a->elem = precision == LM_C64 ? 16 : 8;
    a->nslots = nslots;
    a->nblk = (n + 31) / 32;
    // enough (block, chunk) pairs for ~6 blocks per SM, chunks of at least 64 kets
    const int64_t want = ((int64_t)6 * std::max(ctx->sm_count, 1) + a->nblk - 1) / a->nblk;
    a->nchunk = std::max<int64_t>(1, std::min<int64_t>(want, (m + 63) / 64));
    a->mchunk = (m + a->nchunk - 1) / a->nchunk;
    a->nchunk = (m + a->mchunk - 1) / a->mchunk;
    cudaSetDevice(ctx->device);
    const size_t gA_len = (size_t)(nslots > 0 ? nslots : 1) * (size_t)a->nblk * (size_t)a->nchunk;
    const size_t gV_len = (size_t)n * (size_t)a->nchunk;
    int rc = adj_alloc(ctx, (void**)&a->d_gV, sizeof(double) * gV_len);
    if (rc == LM_OK) rc = adj_alloc(ctx, (void**)&a->d_gA, sizeof(double) * gA_len);
    if (rc == LM_OK) rc = adj_alloc(ctx, (void**)&a->d_loss, sizeof(double) * (size_t)a->nblk);
    if (rc == LM_OK) rc = adj_alloc(ctx, (void**)&a->d_target, sizeof(double) * (size_t)n);
    if (rc == LM_OK) rc = adj_alloc(ctx, (void**)&a->d_dhop, sizeof(double2) * 2 * (size_t)n);
    if (rc != LM_OK) {
        dev_free(ctx, a->d_gV);
        dev_free(ctx, a->d_gA);
        dev_free(ctx, a->d_loss);
        dev_free(ctx, a->d_target);
        dev_free(ctx, a->d_dhop);
        delete a;
        return rc;
    }
    cudaMemsetAsync(a->d_gV, 0, sizeof(double) * gV_len, ctx->stream);
    cudaMemsetAsync(a->d_gA, 0, sizeof(double) * gA_len, ctx->stream);
    *out = a;
    return LM_OK;
}

int lm_adjoint_destroy(lm_adjoint* a) {
    if (!a) return LM_OK;
    cudaSetDevice(a->ctx->device);
    cudaStreamSynchronize(a->ctx->stream);
    adj_free_stack(a);
    dev_free(a->ctx, a->d_gV);
    dev_free(a->ctx, a->d_gA);
    dev_free(a->ctx, a->d_loss);
    dev_free(a->ctx, a->d_target);
    dev_free(a->ctx, a->d_dhop);
    delete a;
    return LM_OK;
}

int lm_adjoint_reset(lm_adjoint* a) {
    if (!a) return LM_ERR_ARG;
    lm_ctx* ctx = a->ctx;
    cudaSetDevice(ctx->device);
    CUDA_TRY(ctx, cudaMemsetAsync(a->d_gV, 0, sizeof(double) * (size_t)a->n * (size_t)a->nchunk, ctx->stream), "memset");
    CUDA_TRY(ctx, cudaMemsetAsync(a->d_gA, 0,
                                  sizeof(double) * (size_t)(a->nslots > 0 ? a->nslots : 1) * (size_t)a->nblk *
                                      (size_t)a->nchunk,
                                  ctx->stream),
             "memset");
    return LM_OK;
}

int lm_adjoint_seed(lm_adjoint* a, lm_state* psi, const double* target, lm_state* lam, double* loss) {
    if (!a) return LM_ERR_ARG;
    lm_ctx* ctx = a->ctx;
    if (!psi || !lam || !target || !loss) return set_err(ctx, LM_ERR_ARG, "lm_adjoint_seed: null argument");
    if (psi->n != a->n || psi->m != a->m || lam->n != a->n || lam->m != a->m || psi->precision != a->precision ||
        lam->precision != a->precision || psi->kind != LM_KETS || lam->kind != LM_KETS)
        return set_err(ctx, LM_ERR_ARG, "lm_adjoint_seed: state shapes differ from the adjoint");
    cudaSetDevice(ctx->device);
    CUDA_TRY(ctx, cudaMemcpyAsync(a->d_target, target, sizeof(double) * (size_t)a->n, cudaMemcpyHostToDevice, ctx->stream),
             "upload target");
    const unsigned blocks = (unsigned)a->nblk;
    if (a->precision == LM_C64)
        adj_seed_kernel<double><<<blocks, 256, 0, ctx->stream>>>(a->n, (const double2*)psi->d_data, (double2*)lam->d_data,
                                                                 psi->ld, a->m, a->d_target, a->d_loss);
    else
        adj_seed_kernel<float><<<blocks, 256, 0, ctx->stream>>>(a->n, (const float2*)psi->d_data, (float2*)lam->d_data,
                                                                psi->ld, a->m, a->d_target, a->d_loss);
    ctx->launches++;
    CUDA_TRY(ctx, cudaGetLastError(), "seed kernel");
    std::vector<double> part((size_t)a->nblk);
    CUDA_TRY(ctx, cudaMemcpyAsync(part.data(), a->d_loss, sizeof(double) * part.size(), cudaMemcpyDeviceToHost,
                                  ctx->stream),
             "download loss");
    CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream), "sync");
    double tot = 0.0;
    for (double v : part) tot += v;  // block order
    *loss = tot;
    return wait_status(ctx);
}

int lm_adjoint_step(lm_adjoint* a, lm_solver* s, lm_ham* h, int component, int slot, lm_state* psi, lm_state* lam) {
    if (!a || !s) return LM_ERR_ARG;
    lm_ctx* ctx = a->ctx;
    if (!h || !psi || !lam) return set_err(ctx, LM_ERR_ARG, "lm_adjoint_step: null argument");
    if (!s->valid || s->ham != h) return set_err(ctx, LM_ERR_STATE, "lm_adjoint_step: update the solver with this Hamiltonian first");
    if (psi->n != a->n || psi->m != a->m || lam->n != a->n || lam->m != a->m || psi->precision != a->precision ||
        lam->precision != a->precision)
        return set_err(ctx, LM_ERR_ARG, "lm_adjoint_step: state shapes differ from the adjoint");
    if (component >= h->fields.n || (component >= 0 && (slot < 0 || slot >= a->nslots)))
        return set_err(ctx, LM_ERR_ARG, "lm_adjoint_step: bad field component or gradient slot");
    cudaSetDevice(ctx->device);
    const Geom& g = h->lat->g;
    const int K = s->K;
    const bool f64 = a->precision == LM_C64;
    // ComplexF32 kets that fit on chip: T_k and beta_k of all orders in one launch each, then the sums
    // over all of them.  The recurrences' operation order is that of the per-order kernels.
    ResidentInst ri{};
    int cl = 0;
    bool resident = !f64 && ctx->fused && K >= 3 && K < a->lean_K && psi->ld == lam->ld &&
                    resident_single_plan(ctx, g, K, a->m, psi->ld, psi->d_data, lam->d_data, ri, &cl);
    int rc = adj_ensure_stack(a, K, resident);
    if (rc == LM_ERR_OOM && resident) {  // K + 2 blocks instead of 2K - 1, and the same bits
        a->lean_K = K;
        resident = false;
        rc = adj_ensure_stack(a, K, false);
    }
    if (rc != LM_OK) return rc;
    const void* hop2 = f64 ? (const void*)s->d_hop2 : (const void*)s->d_hop2f;
    const void* diag2 = f64 ? (const void*)s->d_diag2 : (const void*)s->d_diag2f;
    const int64_t ld = psi->ld, M = a->m;
    auto recur = [&](const void* tp, const void* tpp, const void* lamp, void* out, double alpha, double wre,
                     double wim) -> cudaError_t {
        return launch_stencil_recur(ctx, g, a->precision, hop2, diag2, tp, tpp, lamp, out, ld, M, alpha, wre, wim,
                                    nullptr, 0.0);
    };
    // T_0 = psi_n (aliased), T_1 = H~ T_0, T_k = 2 H~ T_{k-1} - T_{k-2}  (k < K)
    a->T[0] = psi->d_data;
    if (resident) {
        ri.hop2 = s->d_hop2f;
        ri.diag2 = s->d_diag2f;
        resident_fill_coef(ri, K, s->coef.data(), s->phase_re, s->phase_im);
        ResidentOrders ot{}, ob{};
        for (int k = 1; k < K; ++k) ot.p[k] = (float2*)a->T[(size_t)k];
        for (int k = 1; k <= K; ++k) ob.p[k] = (float2*)a->B[(size_t)k];
        rc = resident_single(ctx, K, false, cl, 1, ri, ot);
        ri.x = (const float2*)lam->d_data;
        if (rc == LM_OK) rc = resident_single(ctx, K, false, cl, 2, ri, ob);
        if (rc != LM_OK) return rc;
    }
    for (int k = 1; k < K && !resident; ++k) {
        CUDA_TRY(ctx, recur(a->T[(size_t)k - 1], k >= 2 ? a->T[(size_t)k - 2] : nullptr, nullptr, a->T[(size_t)k],
                            k == 1 ? 0.5 : 1.0, 0.0, 0.0),
                 "adjoint forward recurrence");
    }
    // field derivative table
    const double2* dhop = nullptr;
    if (component >= 0) {
        flux_derivative_kernel<<<dim3((unsigned)((g.N + 127) / 128), 2), 128, 0, ctx->stream>>>(
            g, h->fields, component, h->d_hop, a->d_dhop);
        ctx->launches++;
        CUDA_TRY(ctx, cudaGetLastError(), "flux derivative kernel");
        dhop = a->d_dhop;
    }
    // beta_K .. beta_1 with gradient terms; B[k % 3] rotates
    const dim3 ggrid((unsigned)a->nblk, (unsigned)a->nchunk);
    double* gA = component >= 0 ? a->d_gA + (size_t)slot * (size_t)a->nblk * (size_t)a->nchunk : nullptr;
    if (resident) {
        GradOrders go{};
        for (int k = 1; k <= K; ++k) {
            go.T[k - 1] = (const float2*)a->T[(size_t)k - 1];
            go.b[k] = (const float2*)a->B[(size_t)k];
        }
        const int64_t nV = a->n * a->nchunk, nA = a->nblk * a->nchunk;
        double* sums_V = a->d_sums;
        double* sums_A = a->d_sums + nV * K;
        adj_sums_kernel<<<dim3(ggrid.x, ggrid.y, (unsigned)K), 256, 0, ctx->stream>>>(
            g, go, dhop, ld, M, a->mchunk, s->phase_re, s->phase_im, 1.0 / s->a, sums_V, sums_A);
        ctx->launches++;
        CUDA_TRY(ctx, cudaGetLastError(), "adjoint gradient sums");
        adj_fold_kernel<<<(unsigned)((nV + 255) / 256), 256, 0, ctx->stream>>>(K, nV, nA, 1.0 / s->a, sums_V, sums_A,
                                                                               a->d_gV, gA);
        ctx->launches++;
        CUDA_TRY(ctx, cudaGetLastError(), "adjoint gradient fold");
        return LM_OK;
    }
    for (int k = K; k >= 1; --k) {
        const ChebCoef c = s->coef[(size_t)k];
        const double wre = c.odd ? 0.0 : c.s, wim = c.odd ? c.s : 0.0;  // conj(c_k)
        void* bk = a->B[k % 3];
        const void* b1 = k + 1 <= K ? a->B[(k + 1) % 3] : nullptr;
        const void* b2 = k + 2 <= K ? a->B[(k + 2) % 3] : nullptr;
        const double f = (k == 1 ? 1.0 : 2.0) / s->a;
        if (f64)
            adj_beta_grad_kernel<double><<<ggrid, 256, 0, ctx->stream>>>(
                g, (const double2*)hop2, (const double*)diag2, (const double2*)b1, (const double2*)b2,
                (const double2*)lam->d_data, (double2*)bk, wre, wim, dhop, (const double2*)a->T[(size_t)k - 1], ld, M,
                a->mchunk, s->phase_re, s->phase_im, f, a->d_gV, gA);
        else
            adj_beta_grad_kernel<float><<<ggrid, 256, 0, ctx->stream>>>(
                g, (const float2*)hop2, (const float*)diag2, (const float2*)b1, (const float2*)b2,
                (const float2*)lam->d_data, (float2*)bk, (float)wre, (float)wim, dhop,
                (const float2*)a->T[(size_t)k - 1], ld, M, a->mchunk, s->phase_re, s->phase_im, f, a->d_gV, gA);
        ctx->launches++;
        CUDA_TRY(ctx, cudaGetLastError(), "adjoint beta/gradient kernel");
    }
    return LM_OK;
}

int lm_adjoint_gradients(lm_adjoint* a, double* gV, double* gA) {
    if (!a) return LM_ERR_ARG;
    lm_ctx* ctx = a->ctx;
    cudaSetDevice(ctx->device);
    const size_t nc = (size_t)a->nchunk, nb = (size_t)a->nblk;
    std::vector<double> pv, pa;
    if (gV) {
        pv.resize((size_t)a->n * nc);
        CUDA_TRY(ctx, cudaMemcpyAsync(pv.data(), a->d_gV, sizeof(double) * pv.size(), cudaMemcpyDeviceToHost, ctx->stream),
                 "download gV");
    }
    if (gA && a->nslots > 0) {
        pa.resize((size_t)a->nslots * nb * nc);
        CUDA_TRY(ctx, cudaMemcpyAsync(pa.data(), a->d_gA, sizeof(double) * pa.size(), cudaMemcpyDeviceToHost, ctx->stream),
                 "download gA");
    }
    CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream), "sync");
    if (gV)
        for (int64_t i = 0; i < a->n; ++i) {
            double tot = 0.0;
            for (size_t c = 0; c < nc; ++c) tot += pv[c * (size_t)a->n + (size_t)i];  // chunk order
            gV[i] = tot;
        }
    for (int j = 0; gA && j < a->nslots; ++j) {
        double tot = 0.0;
        const double* p = pa.data() + (size_t)j * nb * nc;
        for (size_t q = 0; q < nb * nc; ++q) tot += p[q];  // chunk-major block order
        gA[j] = tot;
    }
    return wait_status(ctx);
}

int lm_solver_set_bounds(lm_solver* s, double emin, double emax) {
    if (!s) return LM_ERR_ARG;
    if (!(emin == 0.0 && emax == 0.0) && !(isfinite(emin) && isfinite(emax) && emax > emin))
        return set_err(s->ctx, LM_ERR_ARG, "lm_solver_set_bounds: need emin < emax (or 0, 0 for automatic)");
    s->fixed_bounds = !(emin == 0.0 && emax == 0.0);
    s->fix_emin = emin;
    s->fix_emax = emax;
    s->valid = 0;
    return LM_OK;
}

}  // extern "C"
