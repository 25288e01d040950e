// Chebyshev series sum_k c_k T_k(H~) with a whole ket on chip for all orders: the ComplexF64
// propagator step of kets and density matrices (the step! of src/evolution.jl:69-78) and the
// double-float real series of lm_cheb_apply, on square lattices that fit in shared memory.
//
// A CTA takes KT kets at a time.  Their T_{k-1} and T_{k-2} lie in two shared buffers (T_k
// overwrites T_{k-2}), the sum in registers; a thread owns one row y over a run of `cols` columns,
// so the x-neighbours come from a register window and three shared loads serve a site.  One block
// barrier per order, one read and one write of the ket per launch.
//
// The stencil runs in a gauge in which every x-hop is the real t1: H = G H' G^dagger with
// g(x + 1, y) = g(x, y) conj(h_x) / t1.  Any field on a lattice with an open x axis has one (and a
// Landau field without an x twist is in it, g = 1).  A site and order then takes 16 real
// multiply-adds instead of 20, for 8 more per ket and launch at the load and the store.
//
// What bounds it: the arithmetic.  FP64 runs at 2 lane operations per clock and SM (1.84 reached; its pipe is
// 79 % busy with one CTA per SM), so the 16 of a site and order are all that counts; a double-float product and sum takes 12 FP32
// operations (error-free product, TwoSum, one compensation word that is folded in once per site)
// instead of 18 with a normalised sum, on packed pairs (re, im).  Measured: a dense 10 x 10 step 21 us
// against 18 launches of 3 us and their host time (67 us), a dense 47 x 31 step 1.31 ms as with a launch per
// order, the Fermi operator of a 48 x 48 lattice (470 terms) 16.9 ms (19.4 ms with scalar operations)
// against 54 ms with a launch per term.
#include <cuda_runtime.h>

#include <algorithm>

#include "lmgpu_order.cuh"
#include "lmgpu_series.cuh"

namespace lmgpu {

namespace {

constexpr int kThreads = 384;
constexpr size_t kMaxSmem = 226 * 1024;

__device__ __forceinline__ double2 dmul(double2 a, double2 b) {
    return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ double2 dconj(double2 a) { return make_double2(a.x, -a.y); }
__device__ __forceinline__ float2 dsplit(double v) {
    const float h = (float)v;
    return make_float2(h, (float)(v - (double)h));
}

// Arithmetic on one complex value: FP64 ...
struct ArithF64 {
    typedef double2 Elem;
    typedef double2 CCoef;
    typedef double Coef;
    struct Acc {
        double re, im;
    };
    __device__ static Elem from(double2 v) { return v; }
    __device__ static double2 to(const Acc& a) { return make_double2(a.re, a.im); }
    __device__ static Coef coef(double v) { return v; }
    __device__ static void clear(Acc& a) { a.re = a.im = 0.0; }
    __device__ static void neg(Acc& a, Elem v) {
        a.re = -v.x;
        a.im = -v.y;
    }
    __device__ static void add(Acc& a, Coef c, Elem v) {
        a.re = fma(c, v.x, a.re);
        a.im = fma(c, v.y, a.im);
    }
    __device__ static void add2(Acc& a, Coef c, Elem u, Elem v) {
        add(a, c, u);
        add(a, c, v);
    }
    __device__ static void addc(Acc& a, CCoef h, Elem v) {
        a.re = fma(-h.y, v.y, fma(h.x, v.x, a.re));
        a.im = fma(h.y, v.x, fma(h.x, v.y, a.im));
    }
    __device__ static void addy(Acc& a, Coef c, Elem v) { add(a, c, v); }
    __device__ static CCoef conj(CCoef h) { return dconj(h); }
    __device__ static CCoef czero() { return make_double2(0.0, 0.0); }
    __device__ static Elem finish(const Acc& a) { return make_double2(a.re, a.im); }
    __device__ static Elem half(Elem v) { return make_double2(0.5 * v.x, 0.5 * v.y); }
    __device__ static Elem mul_mi(Elem v) { return make_double2(v.y, -v.x); }  // -i v
    __device__ static Elem zero() { return make_double2(0.0, 0.0); }
};

// ... and double-float, real and imaginary part side by side.  An accumulator is an unnormalised pair:
// products enter h by TwoSum, every error term l.  All operations round to nearest, and the compiler
// neither contracts nor reorders them.
struct ArithDF {
    typedef float4 Elem;   // {re.hi, im.hi, re.lo, im.lo}
    typedef float4 CCoef;  // {re.hi, re.lo, im.hi, im.lo}
    typedef float2 Coef;
    typedef DF2 Acc;
    __device__ static Elem from(double2 v) {
        const float2 r = dsplit(v.x), i = dsplit(v.y);
        return make_float4(r.x, i.x, r.y, i.y);
    }
    __device__ static double2 to(const Acc& a) {
        return make_double2((double)a.h.x + (double)a.l.x, (double)a.h.y + (double)a.l.y);
    }
    __device__ static Coef coef(double v) { return dsplit(v); }
    __device__ static void clear(Acc& a) { a = DF2(); }
    __device__ static void neg(Acc& a, Elem v) { a = DF2(make_float4(-v.x, -v.y, -v.z, -v.w)); }
    __device__ static void add(Acc& a, Coef c, Elem v) { a.madd(c, DF2(v)); }
    __device__ static void add2(Acc& a, Coef c, Elem u, Elem v) {  // the sum first: one product for two neighbours
        a.madd(c, df2_sum(DF2(u), DF2(v)));
    }
    __device__ static void addc(Acc& a, CCoef h, Elem v) { a.maddc(h, DF2(v)); }
    // the sum over the orders: hundreds of terms, so the pair is normalised after each (left as it is,
    // the compensation word grows and the series ends 4 times as far off, 1.7e-13 at 48 x 48)
    __device__ static void addy(Acc& a, Coef c, Elem v) {
        add(a, c, v);
        a.normalise();
    }
    __device__ static CCoef conj(CCoef h) { return make_float4(h.x, h.y, -h.z, -h.w); }
    __device__ static CCoef czero() { return make_float4(0.f, 0.f, 0.f, 0.f); }
    __device__ static Elem finish(Acc a) {
        a.normalise();
        return a.word();
    }
    __device__ static Elem half(Elem v) { return make_float4(0.5f * v.x, 0.5f * v.y, 0.5f * v.z, 0.5f * v.w); }
    __device__ static Elem mul_mi(Elem v) { return make_float4(v.y, -v.x, v.w, -v.z); }
    __device__ static Elem zero() { return make_float4(0.f, 0.f, 0.f, 0.f); }
};

// KT kets per CTA, at most S columns per thread.  PROP: c_k = (-i)^k-alternating (propagator, cf),
// else real (cd).
template <class A, int KT, int S, bool PROP>
__global__ void __launch_bounds__(kThreads, 1) series_resident_kernel(const __grid_constant__ SeriesArgs a) {
    typedef typename A::Elem Elem;
    extern __shared__ float4 smem4[];
    const int Lx = a.Lx, Ly = a.Ly, N = Lx * Ly;
    const int strip = (Lx + 2) * Ly;  // a ket with a zero column on either side
    Elem* buf = reinterpret_cast<Elem*>(smem4);
    typename A::CCoef* hy = reinterpret_cast<typename A::CCoef*>(buf + (size_t)2 * KT * strip);
    typename A::Coef* dg = reinterpret_cast<typename A::Coef*>(hy + N);
    const int t = threadIdx.x, nt = blockDim.x;
    for (int i = t; i < N; i += nt) {
        hy[i] = reinterpret_cast<const typename A::CCoef*>(a.hy)[i];
        dg[i] = reinterpret_cast<const typename A::Coef*>(a.diag)[i];
    }
    for (int i = t; i < 2 * KT * Ly; i += nt) {  // the zero columns
        Elem* b = buf + (size_t)(i / Ly) * strip + i % Ly;
        b[0] = A::zero();
        b[(size_t)(Lx + 1) * Ly] = A::zero();
    }
    const int seg = t / Ly, y = t - seg * Ly;
    const int xa = seg * a.cols, xb = seg < a.nseg ? min(Lx, xa + a.cols) : xa;
    const int dyp = y + 1 < Ly ? 1 : (a.per_y ? 1 - Ly : 0);
    const int dym = y > 0 ? -1 : (a.per_y ? Ly - 1 : 0);
    const bool down = y > 0 || a.per_y;  // an absent upward bond has hop 0 in the table
    const typename A::Coef alpha = A::coef(a.alpha);
    const int64_t items = (a.M + KT - 1) / KT;
    for (int64_t item = blockIdx.x; item < items; item += gridDim.x) {
        typename A::Acc sum[KT][S];
        __syncthreads();
#pragma unroll
        for (int i = 0; i < S; ++i) {
            const int x = xa + i;
            if (x >= xb) break;
            const int s = x * Ly + y;
            double2 f = PROP ? a.phase : make_double2(1.0, 0.0);
            if (a.gauge && a.in) f = dmul(f, dconj(a.gauge[s]));
#pragma unroll
            for (int q = 0; q < KT; ++q) {
                const int64_t m = item * KT + q;
                double2 v = make_double2(0.0, 0.0);
                if (m < a.M) {
                    if (!a.in) v.x = m == s ? 1.0 : 0.0;
                    else v = (PROP || a.gauge) ? dmul(f, a.in[m * a.ld_in + s]) : a.in[m * a.ld_in + s];
                }
                const Elem e = A::from(v);
                buf[(size_t)q * strip + s + Ly] = e;
                A::clear(sum[q][i]);
                if constexpr (PROP) A::add(sum[q][i], A::coef(a.cf[0]), e);
                else A::add(sum[q][i], a.cd[0], e);
            }
        }
        __syncthreads();
        for (int k = 1; k <= a.K; ++k) {
            const Elem* src = buf + (size_t)((k - 1) & 1) * KT * strip + Ly;  // T_{k-1}, column 0
            Elem* dst = buf + (size_t)(k & 1) * KT * strip + Ly;              // T_{k-2}, then T_k
            typename A::Coef ck;
            if constexpr (PROP) ck = A::coef(a.cf[k]);
            else ck = a.cd[k];
            Elem tm[KT], tc[KT];
            const int xm = xa > 0 ? xa - 1 : (a.per_x ? Lx - 1 : -1);
            if (xa < xb) {
#pragma unroll
                for (int q = 0; q < KT; ++q) {
                    tm[q] = src[(size_t)q * strip + xm * Ly + y];
                    tc[q] = src[(size_t)q * strip + xa * Ly + y];
                }
            }
#pragma unroll
            for (int i = 0; i < S; ++i) {
                const int x = xa + i;
                if (x >= xb) break;
                const int s = x * Ly + y;
                const int xp = x + 1 < Lx ? x + 1 : (a.per_x ? 0 : Lx);
                const typename A::CCoef hu = hy[s];
                const typename A::CCoef hd = down ? A::conj(hy[s + dym]) : A::czero();
                const typename A::Coef d = dg[s];
#pragma unroll
                for (int q = 0; q < KT; ++q) {
                    const Elem* sq = src + (size_t)q * strip;
                    const Elem tp = sq[xp * Ly + y];
                    typename A::Acc acc;
                    if (k == 1) A::clear(acc);
                    else A::neg(acc, dst[(size_t)q * strip + s]);
                    A::add2(acc, alpha, tm[q], tp);
                    A::addc(acc, hu, sq[s + dyp]);
                    A::addc(acc, hd, sq[s + dym]);
                    A::add(acc, d, tc[q]);
                    Elem tk = A::finish(acc);
                    if (k == 1) tk = A::half(tk);
                    if (k < a.K) dst[(size_t)q * strip + s] = tk;
                    A::addy(sum[q][i], ck, PROP && (k & 1) ? A::mul_mi(tk) : tk);
                    tm[q] = tc[q];
                    tc[q] = tp;
                }
            }
            __syncthreads();
        }
#pragma unroll
        for (int i = 0; i < S; ++i) {
            const int x = xa + i;
            if (x >= xb) break;
            const int s = x * Ly + y;
            const double2 g = a.gauge ? a.gauge[s] : make_double2(1.0, 0.0);
#pragma unroll
            for (int q = 0; q < KT; ++q) {
                const int64_t m = item * KT + q;
                if (m >= a.M) continue;
                double2 v = A::to(sum[q][i]);
                if (a.gauge) {
                    v = dmul(v, g);
                    if (!a.in) v = dmul(v, dconj(a.gauge[m]));
                }
                const int64_t o = a.transpose ? (int64_t)s * a.ld_out + m : m * a.ld_out + s;
                if (a.transpose) v.y = -v.y;
                if (a.out) a.out[o] = v;
                else a.out32[o] = make_float2((float)v.x, (float)v.y);
            }
        }
    }
}

// A warp per row y: g along the row by a product scan over 32 sites at a time (of this row and of the
// next, so that hy' needs no second launch), each kept at modulus 1.
__global__ void __launch_bounds__(32) gauge_tables_kernel(Geom g, const double2* __restrict__ hop,
                                                          const double* __restrict__ onsite, double inv_t, double b,
                                                          double sc, int natural, double2* __restrict__ gauge,
                                                          double2* __restrict__ hy, double* __restrict__ diag,
                                                          float4* __restrict__ hyd, float2* __restrict__ diagd) {
    const int y = blockIdx.x, lane = threadIdx.x;
    const int Lx = (int)g.Lx, Ly = (int)g.Ly;
    const int yn = y + 1 < Ly ? y + 1 : 0;
    double2 run[2] = {make_double2(1.0, 0.0), make_double2(1.0, 0.0)};  // g at the first site of the chunk
    for (int x0 = 0; x0 < Lx; x0 += 32) {
        const int x = x0 + lane;
        double2 gv[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            gv[r] = make_double2(1.0, 0.0);
            if (natural) continue;
            double2 u = make_double2(1.0, 0.0);  // g(x + 1) / g(x)
            if (x + 1 < Lx) {
                const double2 h = hop[(int64_t)x * Ly + (r ? yn : y)];
                if (inv_t != 0.0) u = make_double2(h.x * inv_t, -h.y * inv_t);
            }
#pragma unroll
            for (int w = 1; w < 32; w *= 2) {  // inclusive scan
                const double2 v = make_double2(__shfl_up_sync(0xffffffffu, u.x, w), __shfl_up_sync(0xffffffffu, u.y, w));
                if (lane >= w) u = dmul(u, v);
            }
            double2 ex = make_double2(__shfl_up_sync(0xffffffffu, u.x, 1), __shfl_up_sync(0xffffffffu, u.y, 1));
            if (lane == 0) ex = make_double2(1.0, 0.0);
            ex = dmul(run[r], ex);
            u = dmul(run[r], u);
            const double f = 0.5 * (3.0 - fma(ex.x, ex.x, ex.y * ex.y));
            gv[r] = make_double2(f * ex.x, f * ex.y);
            const double fu = 0.5 * (3.0 - fma(u.x, u.x, u.y * u.y));
            run[r] = make_double2(__shfl_sync(0xffffffffu, fu * u.x, 31), __shfl_sync(0xffffffffu, fu * u.y, 31));
        }
        if (x >= Lx) continue;
        const int64_t s = (int64_t)x * Ly + y;
        double2 h = hop[g.N + s];
        if (!natural) h = dmul(dmul(dconj(gv[0]), h), gv[1]);
        h = make_double2(h.x * sc, h.y * sc);
        const double d = ((onsite ? onsite[s] : 0.0) - b) * sc;
        if (gauge) gauge[s] = gv[0];
        if (hy) hy[s] = h;
        if (diag) diag[s] = d;
        if (hyd) {
            const float2 r = dsplit(h.x), i = dsplit(h.y);
            hyd[s] = make_float4(r.x, r.y, i.x, i.y);
        }
        if (diagd) diagd[s] = dsplit(d);
    }
}

// CTAs of this block and shared size that fit an SM, remembered for the last ones.
template <class A, int KT, int S, bool PROP>
cudaError_t fit_t(lm_ctx* ctx, int variant, int threads, size_t smem, int* fit) {
    auto& f = ctx->series_fit[variant];
    if (f.threads != threads || f.smem != smem) {
        cudaError_t e = cudaFuncSetAttribute(series_resident_kernel<A, KT, S, PROP>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem);
        int n = 1;
        if (e == cudaSuccess)
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, series_resident_kernel<A, KT, S, PROP>, threads, smem);
        if (e != cudaSuccess) return e;
        f.threads = threads;
        f.smem = smem;
        f.fit = std::max(n, 1);
    }
    *fit = f.fit;
    return cudaSuccess;
}

// Several CTAs of a small lattice share an SM, each taking an equal share of the items.
struct Share {
    int64_t waves, grid;
};
Share share(int64_t items, int fit, int sm_count) {
    const int64_t slots = (int64_t)fit * sm_count, waves = (items + slots - 1) / slots;
    return {waves, (items + waves - 1) / waves};
}

int block_threads(int Ly, int nseg) { return (Ly * nseg + 31) / 32 * 32; }

template <class A, int KT, int S, bool PROP>
cudaError_t launch_t(lm_ctx* ctx, const SeriesPlan& p, const SeriesArgs& a, int variant) {
    const int threads = block_threads(a.Ly, a.nseg);
    int fit = 1;
    const cudaError_t e = fit_t<A, KT, S, PROP>(ctx, variant, threads, p.smem, &fit);
    if (e != cudaSuccess) return e;
    const Share sh = share((a.M + KT - 1) / KT, fit, ctx->sm_count);
    series_resident_kernel<A, KT, S, PROP><<<(unsigned)sh.grid, threads, p.smem, ctx->stream>>>(a);
    ctx->launches++;
    return cudaGetLastError();
}

// CTAs per SM of a plan's FP64 kernel (0 on an error).
int fit_f64(lm_ctx* ctx, const SeriesPlan& p, int threads) {
    int fit = 0;
    const cudaError_t e = p.cols <= 2   ? fit_t<ArithF64, 1, 2, true>(ctx, 0, threads, p.smem, &fit)
                          : p.cols <= 4 ? fit_t<ArithF64, 1, 4, true>(ctx, 1, threads, p.smem, &fit)
                          : p.cols <= 8 ? fit_t<ArithF64, 1, 8, true>(ctx, 2, threads, p.smem, &fit)
                                        : fit_t<ArithF64, 1, 12, true>(ctx, 3, threads, p.smem, &fit);
    if (e == cudaSuccess) return fit;
    cudaGetLastError();
    return 0;
}

}  // namespace

SeriesPlan series_plan(lm_ctx* ctx, const Geom& g, bool x_real, int64_t M, bool df) {
    SeriesPlan p;
    // a periodic x axis has no such gauge in general; there the FP64 form stays with the per-order
    // kernels also where the x-hops are real, so that both kinds of field round alike
    if ((g.per_x && (!x_real || !df)) || g.Ly > kThreads || g.N > 8192) return p;
    const size_t ket = 2 * 16 * (size_t)((g.Lx + 2) * g.Ly), tables = 24 * (size_t)g.N;
    // FP64: half the threads where two CTAs fit an SM, so that one computes while the other waits at
    // an order's barrier (6 warps each keep the FP64 pipe full)
    int threads = kThreads;
    if (!df && 2 * (ket + tables) <= kMaxSmem && g.Ly * ((g.Lx + 7) / 8) <= kThreads / 2) threads = kThreads / 2;
    p.nseg = (int)std::min<int64_t>(g.Lx, threads / g.Ly);
    p.cols = (int)((g.Lx + p.nseg - 1) / p.nseg);
    p.nseg = (int)((g.Lx + p.cols - 1) / p.cols);
    if (p.cols > 12) return p;
    // two kets share the table loads of the double-float form while there are enough of them
    const int kt = df && p.cols <= 6 && M >= 2 * ctx->sm_count && 2 * ket + tables <= kMaxSmem ? 2 : 1;
    p.smem = kt * ket + tables;
    if (p.smem > kMaxSmem) return p;
    // Against one launch per order.
    const double sites = (double)g.N, mhz = 2000.0;
    double here, there;
    if (df) {
        // An order takes the longest SM's share of the kets at 1.9 clocks a site, a launch per order about 5 us
        // and its memory traffic (48 x 48: 34 against 111 us an order).
        const int64_t per_sm = (M + (int64_t)kt * ctx->sm_count - 1) / ((int64_t)kt * ctx->sm_count) * kt;
        here = 0.5 + (double)per_sm * sites * 1.9 / mhz;
        there = 5.0 + (double)M * sites * 2.0e-5;
    } else {
        // A launch per order takes 4.25 us and the block's 16 or 20 DFMAs a site at 1.84 a clock and SM.  Here the
        // kets of the SM with the most of them count, in whole CTAs and waves, at 9.4 or 10.1 clocks for a
        // thread's column, idle lanes included.  Fitted to 330 steps of 13 lattices from 6 x 6 to 64 x 62 with 1 to
        // 1500 kets and dense (here within 20 %, there within 10 %).  Complex x-hops, K = 9, here / there: dense
        // 10 x 10 25 / 74 us, 24 x 24 229 / 296 us, 40 x 33 1476 / 1207 us; 32 x 27 with 304 kets 96 / 126 us, with 330,
        // whose third CTA makes it four kets an SM, 187 / 133 us; 31 x 47 with 700 436 / 367 us.
        const int threads = block_threads((int)g.Ly, p.nseg), fit = fit_f64(ctx, p, threads);
        if (!fit) return p;
        const Share sh = share(M, fit, ctx->sm_count);
        const int64_t kets = (sh.grid + ctx->sm_count - 1) / ctx->sm_count * sh.waves;
        here = 0.55 + 0.2 * (double)sh.waves + (double)kets * threads * p.cols * (x_real ? 9.4 : 10.1) / mhz;
        there = 4.25 + (double)M * sites * (x_real ? 16.0 : 20.0) / 1.84 / mhz / ctx->sm_count;
    }
    if (here < there) p.kt = kt;
    return p;
}

cudaError_t launch_gauge_tables(lm_ctx* ctx, const Geom& g, const double2* hop, const double* onsite, double t1, double a,
                                double b, bool x_real, double2* gauge, double2* hy, double* diag, float4* hyd,
                                float2* diagd) {
    gauge_tables_kernel<<<(unsigned)g.Ly, 32, 0, ctx->stream>>>(g, hop, onsite, t1 != 0.0 ? 1.0 / t1 : 0.0, b, 2.0 / a,
                                                                x_real ? 1 : 0, gauge, hy, diag, hyd, diagd);
    ctx->launches++;
    return cudaGetLastError();
}

cudaError_t launch_series_f64(lm_ctx* ctx, const SeriesPlan& p, SeriesArgs a) {
    a.nseg = p.nseg;
    a.cols = p.cols;
    if (p.cols <= 2) return launch_t<ArithF64, 1, 2, true>(ctx, p, a, 0);
    if (p.cols <= 4) return launch_t<ArithF64, 1, 4, true>(ctx, p, a, 1);
    if (p.cols <= 8) return launch_t<ArithF64, 1, 8, true>(ctx, p, a, 2);
    return launch_t<ArithF64, 1, 12, true>(ctx, p, a, 3);
}

cudaError_t launch_series_df(lm_ctx* ctx, const SeriesPlan& p, SeriesArgs a) {
    a.nseg = p.nseg;
    a.cols = p.cols;
    if (p.kt == 2) return p.cols <= 2 ? launch_t<ArithDF, 2, 2, false>(ctx, p, a, 4) : launch_t<ArithDF, 2, 6, false>(ctx, p, a, 5);
    if (p.cols <= 2) return launch_t<ArithDF, 1, 2, false>(ctx, p, a, 6);
    if (p.cols <= 6) return launch_t<ArithDF, 1, 6, false>(ctx, p, a, 7);
    return launch_t<ArithDF, 1, 12, false>(ctx, p, a, 8);
}

}  // namespace lmgpu
