// Kernel polynomial method: Chebyshev moments of the tight-binding Hamiltonian on the device,
// for the density of states and the local density of states without a full eigensystem (the
// reference computes dos / ldos from an Eigensystem or a GreenFunction, src/greenfunction.jl:
// 306-339).  The moments of a block of starting vectors v are
//   mu_n = sum_v <v| T_n(H~) |v>,   H~ = (H - b)/a,
// from the recurrence T_{n+1} = 2 H~ T_n - T_{n-1} on the block and the doubling relations
//   mu_2n = 2 <T_n v|T_n v> - mu_0,   mu_2n+1 = 2 <T_n+1 v|T_n v> - mu_1,
// so nmom moments take about nmom / 2 stencil passes.  With the N unit vectors as the block
// the sum is the exact trace and column j gives the local moments of site j.
//
// lm_cheb_apply evaluates a real Chebyshev series sum_n c_n T_n(H~) on a block (the identity
// gives the matrix function f(H) itself): the Fermi operator of densitymatrix at T > 0
// (src/spectrum.jl:226-257) without an eigensystem.
#include <cuda_runtime.h>
#include <math.h>

#include <algorithm>

#include <new>
#include <utility>
#include <vector>

#include "lmgpu_internal.cuh"
#include "lmgpu_order.cuh"
#include "lmgpu_series.cuh"

namespace lmgpu {

// A = identity (n x n, leading dimension ld).
__global__ void set_identity_kernel(double2* __restrict__ a, int64_t n, int64_t ld) {
    for (int64_t col = blockIdx.y; col < n; col += gridDim.y)
        for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
            a[col * ld + i] = make_double2(i == col ? 1.0 : 0.0, 0.0);
}

// out[col] = Re sum_i conj(A[i, col]) B[i, col], one block per column (fixed-order reduction).
__global__ void __launch_bounds__(256) column_dots_kernel(const double2* __restrict__ A, const double2* __restrict__ B,
                                                          int64_t n, int64_t ld, int64_t M, double* __restrict__ out) {
    __shared__ double red[8];
    for (int64_t col = blockIdx.x; col < M; col += gridDim.x) {
        const double2* a = A + col * ld;
        const double2* b = B + col * ld;
        double acc = 0.0;
        for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
            const double2 x = a[i], y = b[i];
            acc = fma(x.x, y.x, fma(x.y, y.y, acc));
        }
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
        __syncthreads();
        if (threadIdx.x == 0) {
            double t = 0.0;
            for (int w = 0; w < 8; ++w) t += red[w];
            out[col] = t;
        }
        __syncthreads();
    }
}

// y = y + c x (real c), n complex entries
__global__ void axpy_kernel(double2* __restrict__ y, const double2* __restrict__ x, double c, int64_t n) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        double2 v = y[i];
        const double2 u = x[i];
        v.x = fma(c, u.x, v.x);
        v.y = fma(c, u.y, v.y);
        y[i] = v;
    }
}

// y = c x (real c)
__global__ void scaled_copy_kernel(double2* __restrict__ y, const double2* __restrict__ x, double c, int64_t n) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        y[i] = make_double2(c * x[i].x, c * x[i].y);
}

// Lanczos start vector: entries of modulus 1/sqrt(n) with pseudo-random phases (splitmix64 of
// (seed, i)), so every eigenvector has a component in it almost surely.
__global__ void start_vector_kernel(double2* __restrict__ v, int64_t n, unsigned long long seed) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        unsigned long long z = seed + 0x9E3779B97F4A7C15ull * (unsigned long long)(i + 1);
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        z ^= z >> 31;
        const double phi = 6.283185307179586 * (double)(z >> 11) * (1.0 / 9007199254740992.0);
        double sn, cs;
        sincos(phi, &sn, &cs);
        const double r = rsqrt((double)n);
        v[i] = make_double2(r * cs, r * sn);
    }
}


// ------------------------------------------------------------------------------------------
// Double-float ("df") form of the moment recurrence (LM_OPT_KPM = 1, the default).  A real number is an
// unevaluated sum hi + lo of two FP32 values (about 48 significant bits), so the recurrence
// runs on the FP32 pipe instead of GB300's 1/64-rate FP64 pipe.  A complex df value is a float4
// {re.hi, im.hi, re.lo, im.lo}, the size of a double2, so the FP64 buffers are reused in place.
// Products take the exact FMA error term (p + e = a*b exactly); sums use the double-word
// addition of Dekker and of Knuth's TwoSum.  Every step is an explicit round-to-nearest
// intrinsic, which nvcc never contracts into an FMA or reorders, so the error-free
// transformations stay exact.  An exact emulation of this arithmetic keeps the moments within
// about 1e-14 of FP64 after 1024 passes.
// ------------------------------------------------------------------------------------------
struct DF {
    float h, l;
};
__device__ __forceinline__ DF df_fast_two_sum(float a, float b) {
    const float s = __fadd_rn(a, b);
    return DF{s, __fsub_rn(b, __fsub_rn(s, a))};
}
__device__ __forceinline__ DF df_add(DF x, DF y) {
    const float s = __fadd_rn(x.h, y.h);
    const float bb = __fsub_rn(s, x.h);
    float e = __fadd_rn(__fsub_rn(x.h, __fsub_rn(s, bb)), __fsub_rn(y.h, bb));
    e = __fadd_rn(e, __fadd_rn(x.l, y.l));
    return df_fast_two_sum(s, e);
}
__device__ __forceinline__ DF df_mul(DF x, DF y) {
    const float p = __fmul_rn(x.h, y.h);
    float e = __fmaf_rn(x.h, y.h, -p);
    e = __fmaf_rn(x.h, y.l, e);
    e = __fmaf_rn(x.l, y.h, e);
    return df_fast_two_sum(p, e);
}
__device__ __forceinline__ DF df_re(float4 v) { return DF{v.x, v.z}; }
__device__ __forceinline__ DF df_im(float4 v) { return DF{v.y, v.w}; }
__device__ __forceinline__ DF df_from(double x) {
    const float h = (float)x;
    return DF{h, (float)(x - (double)h)};
}
__device__ __forceinline__ double df_value(DF x) { return (double)x.h + (double)x.l; }

// hi + lo of a double: hi the nearest FP32 number, lo the remaining 28 bits rounded to FP32, by
// integer operations (conversions run on the FP64 pipe, at its rate: a block of
// 268 MB took 240 us with them, 95 us without).  What is or leaves an FP32 subnormal, and what overflows FP32
// (infinities and NaN included), goes through the conversion; below 2^-150 that gives 0.
__device__ __forceinline__ DF df_split(double v) {
    const int hw = __double2hiint(v);
    const unsigned lw = (unsigned)__double2loint(v);
    const int ex = (hw >> 20) & 0x7ff;
    if (ex >= 1150) return DF{(float)v, 0.f};
    if (ex <= 896 + 53) return ex < 1023 - 150 ? DF{0.f, 0.f} : DF{(float)v, (float)(v - (double)(float)v)};
    const int sign = hw & 0x80000000;
    int low = (int)(lw & 0x1fffffffu);
    const int up = low >> 28;  // round to nearest: the next FP32 number and a negative remainder
    low -= up << 29;
    const float h = __int_as_float(sign | ((((hw & 0x7fffffff) - (896 << 20)) << 3 | (int)(lw >> 29)) + up));
    const float l = __int2float_rn(low) * __int_as_float((ex - 896 - 52) << 23);
    return DF{h, sign ? -l : l};
}

// out = in as df values, column by column (ld_in may differ from ld_out; in null: the identity).
__global__ void to_df_kernel(const double2* __restrict__ in, int64_t ld_in, int64_t n, int64_t M, float4* __restrict__ out,
                             int64_t ld_out) {
    for (int64_t m = blockIdx.y; m < M; m += gridDim.y)
        for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
            if (!in) {
                out[m * ld_out + i] = make_float4(i == m ? 1.f : 0.f, 0.f, 0.f, 0.f);
                continue;
            }
            const double2 v = in[m * ld_in + i];
            const DF r = df_split(v.x), q = df_split(v.y);
            out[m * ld_out + i] = make_float4(r.h, q.h, r.l, q.l);
        }
}

// The stencil tables in df form: hop (2N double2) -> 2N float4, diag (N double) -> N float2.
__global__ void df_tables_kernel(const double2* __restrict__ hop2, const double* __restrict__ diag2, int64_t N,
                                 float4* __restrict__ hopd, float2* __restrict__ diagd) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < 2 * N; i += (int64_t)gridDim.x * blockDim.x) {
        const DF r = df_from(hop2[i].x), m = df_from(hop2[i].y);
        hopd[i] = make_float4(r.h, r.l, m.h, m.l);
        if (i < N) {
            const DF d = df_from(diag2[i]);
            diagd[i] = make_float2(d.h, d.l);
        }
    }
}

// n x M df values -> ComplexF64 (out) or ComplexF32 (out32), leading dimension ld_out.
__global__ void from_df_kernel(const float4* __restrict__ in, int64_t ld_in, int64_t n, int64_t M,
                               double2* __restrict__ out, float2* __restrict__ out32, int64_t ld_out) {
    for (int64_t m = blockIdx.y; m < M; m += gridDim.y)
        for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
            const float4 v = in[m * ld_in + i];
            if (out) out[m * ld_out + i] = make_double2(df_value(df_re(v)), df_value(df_im(v)));
            else out32[m * ld_out + i] = make_float2(v.x, v.y);
        }
}

// One recurrence pass over an N x M block in df arithmetic: out = (2H~) tp - tpp (FIRST: out = H~ tp),
// out may alias tpp.  A thread owns one row y of KT kets and walks along x: the three columns of tp
// that a site needs lie in registers, so tp is read once per site from L2 (plus two shared-line reads
// of the y-neighbours), and the tables once per KT kets.  With DOT the pass also forms
// Re <tpp, tpp> and Re <tp, tpp> of every ket from the values it holds; with YACC, y += c out.
// Products enter an unnormalised pair (s, c) by TwoSum, every error term c: 12 FP32 operations per
// real product and sum; XR (x-hops all equal to the real alpha) adds the two x-neighbours first.
//
// What bounds it: the FP32 pipe (about 215 operations per element) and HBM (three block passes: read tp and
// tpp, write out), which do not overlap fully at 14 warps per SM: 119 us of traffic and 135 us without
// any memory access for 256 x 256 sites and 256 kets, measured 176 us (209 us with the loads of a column
// issued when it is used), the dots included.  One thread per site with normalised sums took 258 us, and 113 us
// more for the dots as a kernel of their own.
struct MarchArgs {
    Geom g;
    const float4* hop;   // 2N: x-hops, then y-hops (2H/a)
    const float2* diag;  // 2(V - b)/a
    const float4* tp;
    const float4* tpp;   // T_{n-1}; FIRST: unused
    float4* out;
    int64_t ld, M;
    int kt;                // kets per thread
    int rows, segs, cols;  // rows and x-segments per block, columns per segment
    float2 alpha;
    float4* y;
    float2 c;
    float2 c0;       // FIRST with YACC: y = c0 tp + c out
    double* part;    // DOT: partial sums [block][2][pstride]
    int64_t pstride;
};

template <bool XR, bool FIRST, bool DOT, bool YACC, int KT>
__global__ void __launch_bounds__(256, 2) df_march_kernel(const __grid_constant__ MarchArgs a) {
    const Geom& g = a.g;
    const int Ly = (int)g.Ly, Lx = (int)g.Lx;
    const int t = threadIdx.x, seg = t / a.rows, yl = t - seg * a.rows;
    const int chunks = (Ly + a.rows - 1) / a.rows;
    const int chunk = (int)(blockIdx.x % chunks);
    const int y = chunk * a.rows + yl;
    const int64_t xa = ((int64_t)(blockIdx.x / chunks) * a.segs + seg) * a.cols;
    const bool on = seg < a.segs && y < Ly && xa < Lx;
    const int xb = on ? (int)(xa + a.cols < Lx ? xa + a.cols : Lx) : 0;
    const int yp = y + 1 < Ly ? 1 : (g.per_y ? 1 - Ly : 0);
    const int ym = y > 0 ? -1 : (g.per_y ? Ly - 1 : 0);
    const bool down = y > 0 || g.per_y;
    const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
    const int64_t m0 = (int64_t)blockIdx.y * KT;
    int64_t off[KT];
    bool have[KT];
#pragma unroll
    for (int q = 0; q < KT; ++q) {
        have[q] = m0 + q < a.M;
        off[q] = (have[q] ? m0 + q : m0) * a.ld;
    }
    DF2 aa[KT], ba[KT];  // the real and imaginary products side by side
    if (on) {
        float4 tm[KT], tc[KT];
        const int x0 = (int)xa;
        const int xm = x0 > 0 ? x0 - 1 : (g.per_x ? Lx - 1 : -1);
        float4 hxm = z4;
        if (!XR && xm >= 0) hxm = a.hop[(int64_t)xm * Ly + y];
#pragma unroll
        for (int q = 0; q < KT; ++q) {
            tm[q] = xm >= 0 ? __ldg(a.tp + off[q] + (int64_t)xm * Ly + y) : z4;
            tc[q] = __ldg(a.tp + off[q] + (int64_t)x0 * Ly + y);
        }
        // the next column and the old value come from L2 or HBM: they are loaded one step ahead
        float4 tn[KT], t2[KT];
        const int xn = x0 + 1 < Lx ? x0 + 1 : (g.per_x ? 0 : -1);
#pragma unroll
        for (int q = 0; q < KT; ++q) {
            tn[q] = xn >= 0 ? __ldg(a.tp + off[q] + (int64_t)xn * Ly + y) : z4;
            t2[q] = FIRST ? z4 : a.tpp[off[q] + (int64_t)x0 * Ly + y];
        }
        for (int x = x0; x < xb; ++x) {
            const int64_t s = (int64_t)x * Ly + y;
            const int xp = x + 2 < Lx ? x + 2 : (g.per_x ? x + 2 - Lx : -1);
            float4 up[KT], dn[KT], tn1[KT], t21[KT];
#pragma unroll
            for (int q = 0; q < KT; ++q) {
                tn1[q] = xp >= 0 && x + 1 < xb ? __ldg(a.tp + off[q] + (int64_t)xp * Ly + y) : z4;
                t21[q] = !FIRST && x + 1 < xb ? a.tpp[off[q] + s + Ly] : z4;
                up[q] = __ldg(a.tp + off[q] + s + yp);
                dn[q] = __ldg(a.tp + off[q] + s + ym);
            }
            const float4 hu = __ldg(a.hop + g.N + s);
            float4 hd = down ? __ldg(a.hop + g.N + s + ym) : z4;
            hd.z = -hd.z;
            hd.w = -hd.w;
            const float2 d = __ldg(a.diag + s);
            float4 hxp = z4;
            if (!XR) hxp = a.hop[s];
#pragma unroll
            for (int q = 0; q < KT; ++q) {
                const DF2 u2(t2[q]), uc(tc[q]);
                DF2 r;
                if (!FIRST) r = DF2(make_float4(-t2[q].x, -t2[q].y, -t2[q].z, -t2[q].w));
                if (XR) {
                    r.madd(a.alpha, df2_sum(DF2(tm[q]), DF2(tn[q])));
                } else {
                    r.maddc(hxp, DF2(tn[q]));
                    r.maddc(make_float4(hxm.x, hxm.y, -hxm.z, -hxm.w), DF2(tm[q]));
                }
                r.maddc(hu, DF2(up[q]));
                r.maddc(hd, DF2(dn[q]));
                r.madd(d, uc);
                r.normalise();
                if (FIRST) {
                    r.h = make_float2(0.5f * r.h.x, 0.5f * r.h.y);
                    r.l = make_float2(0.5f * r.l.x, 0.5f * r.l.y);
                }
                if (DOT) {
                    const float2 nh = make_float2(-u2.h.x, -u2.h.y), nl = make_float2(-u2.l.x, -u2.l.y);
                    aa[q].madd(u2.h, nh, nl, u2.h, u2.l);
                    ba[q].madd(u2.h, nh, nl, uc.h, uc.l);
                    aa[q].normalise();  // long sums: keep the pairs normalised
                    ba[q].normalise();
                }
                if (have[q]) {
                    a.out[off[q] + s] = r.word();
                    if (YACC) {
                        DF2 yv;
                        if (FIRST) yv.madd(a.c0, uc);
                        else yv = DF2(a.y[off[q] + s]);
                        yv.madd(a.c, r);
                        yv.normalise();
                        a.y[off[q] + s] = yv.word();
                    }
                }
                tm[q] = tc[q];
                tc[q] = tn[q];
                tn[q] = tn1[q];
                t2[q] = t21[q];
            }
            if (!XR) hxm = hxp;
        }
    }
    if (DOT) {  // df over the warp, FP64 over the block's warps in order
        __shared__ double red[8][2 * KT];
#pragma unroll
        for (int q = 0; q < 2 * KT; ++q) {
            const DF2 w = q < KT ? aa[q < KT ? q : 0] : ba[q < KT ? 0 : q - KT];
            DF v = df_add(DF{w.h.x, w.l.x}, DF{w.h.y, w.l.y});
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
                v = df_add(v, DF{__shfl_xor_sync(0xffffffffu, v.h, o), __shfl_xor_sync(0xffffffffu, v.l, o)});
            if ((t & 31) == 0) red[t >> 5][q] = df_value(v);
        }
        __syncthreads();
        if (t < 2 * KT && m0 + t % KT < a.M) {
            double v = 0.0;
            for (int w = 0; w < (int)(blockDim.x + 31) / 32; ++w) v += red[w][t];
            a.part[((int64_t)blockIdx.x * 2 + t / KT) * a.pstride + m0 + t % KT] = v;
        }
    }
}

// out[pass][q][m] = sum of the blocks' partials [pass][block][2][M], in block order.
__global__ void sum_parts_kernel(const double* __restrict__ part, int nblk, int64_t M, double* __restrict__ out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 2 * M) return;
    const double* p = part + (int64_t)blockIdx.y * nblk * 2 * M + i;
    double v = 0.0;
    for (int b = 0; b < nblk; ++b) v += p[(int64_t)b * 2 * M];
    out[(int64_t)blockIdx.y * 2 * M + i] = v;
}

// out[col] = Re <A, A>, out[M + col] = Re <B, A> per column, in df per thread and then the
// fixed-order FP64 block reduction of column_dots_kernel.
__global__ void __launch_bounds__(256) column_dots2_df_kernel(const float4* __restrict__ A,
                                                              const float4* __restrict__ B, int64_t n, int64_t ld,
                                                              int64_t M, double* __restrict__ out) {
    __shared__ double red[2][8];
    for (int64_t col = blockIdx.x; col < M; col += gridDim.x) {
        const float4* a = A + col * ld;
        const float4* b = B + col * ld;
        DF aa = DF{0.f, 0.f}, ba = DF{0.f, 0.f};
        for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
            const float4 x = a[i], y = b[i];
            aa = df_add(aa, df_mul(df_re(x), df_re(x)));
            aa = df_add(aa, df_mul(df_im(x), df_im(x)));
            ba = df_add(ba, df_mul(df_re(y), df_re(x)));
            ba = df_add(ba, df_mul(df_im(y), df_im(x)));
        }
        double v[2] = {df_value(aa), df_value(ba)};
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_down_sync(0xffffffffu, v[q], o);
            if ((threadIdx.x & 31) == 0) red[q][threadIdx.x >> 5] = v[q];
        }
        __syncthreads();
        if (threadIdx.x < 2) {
            double t = 0.0;
            for (int w = 0; w < 8; ++w) t += red[threadIdx.x][w];
            out[threadIdx.x * M + col] = t;
        }
        __syncthreads();
    }
}

}  // namespace lmgpu

using namespace lmgpu;

// Number of eigenvalues of the symmetric tridiagonal (a, b) below x (Sturm sequence count).
static int sturm_count(const std::vector<double>& a, const std::vector<double>& b, double x) {
    int cnt = 0;
    double q = 1.0;
    for (size_t i = 0; i < a.size(); ++i) {
        const double bb = i ? b[i - 1] * b[i - 1] : 0.0;
        q = (a[i] - x) - (i ? bb / q : 0.0);
        if (q == 0.0) q = -1e-300;
        if (q < 0.0) ++cnt;
    }
    return cnt;
}

// Last component of the unit eigenvector of the tridiagonal (a, b) for eigenvalue theta, by
// inverse iteration with a slightly shifted theta and Gaussian elimination with partial
// pivoting (the factor of a tridiagonal gains one extra superdiagonal).
static double tridiag_last_component(const std::vector<double>& a, const std::vector<double>& b, double theta) {
    const size_t m = a.size();
    if (m == 1) return 1.0;
    const double shift = theta + 1e-10 * (fabs(theta) + 1.0);
    std::vector<double> x(m, 1.0);
    for (int it = 0; it < 3; ++it) {
        // rows: lower l[i] (below diag), diag d[i], upper u1[i], u2[i] (second superdiagonal)
        std::vector<double> d(m), u1(m, 0.0), u2(m, 0.0), rhs(x);
        std::vector<double> l(m, 0.0);
        for (size_t i = 0; i < m; ++i) {
            d[i] = a[i] - shift;
            if (i + 1 < m) u1[i] = b[i];
            if (i > 0) l[i] = b[i - 1];
        }
        for (size_t i = 0; i + 1 < m; ++i) {
            // eliminate l[i+1] (row i+1, column i) with the larger of rows i, i+1 as pivot
            if (fabs(l[i + 1]) > fabs(d[i])) {
                std::swap(d[i], l[i + 1]);
                std::swap(u1[i], d[i + 1]);
                std::swap(u2[i], u1[i + 1]);
                std::swap(rhs[i], rhs[i + 1]);
            }
            const double piv = d[i] != 0.0 ? d[i] : 1e-300;
            const double f = l[i + 1] / piv;
            d[i + 1] -= f * u1[i];
            u1[i + 1] -= f * u2[i];
            rhs[i + 1] -= f * rhs[i];
            l[i + 1] = 0.0;
        }
        for (size_t ii = m; ii-- > 0;) {
            double v = rhs[ii];
            if (ii + 1 < m) v -= u1[ii] * x[ii + 1];
            if (ii + 2 < m) v -= u2[ii] * x[ii + 2];
            x[ii] = v / (d[ii] != 0.0 ? d[ii] : 1e-300);
        }
        double nrm = 0.0;
        for (double v : x) nrm += v * v;
        nrm = sqrt(nrm);
        if (!(nrm > 0.0) || !isfinite(nrm)) return 1.0;  // fall back to the crude bound
        for (double& v : x) v /= nrm;
    }
    return x[m - 1];
}

// The k-th smallest eigenvalue (k = 0 .. m-1) of the tridiagonal by bisection.
static double tridiag_eig(const std::vector<double>& a, const std::vector<double>& b, int k, double lo, double hi) {
    for (int it = 0; it < 200 && hi - lo > 1e-14 * (fabs(lo) + fabs(hi) + 1e-300); ++it) {
        const double mid = 0.5 * (lo + hi);
        if (sturm_count(a, b, mid) > k) hi = mid;
        else lo = mid;
    }
    return 0.5 * (lo + hi);
}

constexpr int64_t kPartPasses = 16;  // passes whose partial dots are summed by one launch

// Kets per thread, rows and segments of a block, columns per segment: the split with the shortest waves of two
// blocks of up to 256 threads per SM, counting 1.5 columns for a segment's two shared edges and half a
// row for those of a chunk of rows (96 rows in one chunk leave a quarter of a block's threads out: 1.97 ms a
// pass of 9216 x 9216 against 1.66 ms in chunks of 32).  Two kets share the table loads, so one alone costs
// 0.8 of two; where a thread has three columns or less, its chain of loads and sums is what counts, and one ket
// costs 0.6 (64 x 64 sites, complex x-hops, a series of 64 terms on one / two / eight kets: 295 us each, the
// launches' pace; with two kets and at least four columns per thread 471 / 554 / 562 us).  Half a wave, one block
// per SM, costs 0.7 of one, 0.6 with the dots, whose sums at a block's end then come once per SM (256 x 256
// sites, four kets, 64 moments 464 us, in a whole wave of half the columns 502 us).
static void march_plan(const lm_ctx* ctx, const Geom& g, int64_t M, bool dots, MarchArgs& a) {
    const int64_t slots = 2ll * ctx->sm_count, chunks0 = (g.Ly + 255) / 256;
    double best = 1e300;
    for (int kt = 2; kt >= 1; --kt) {
        const int64_t groups = (M + kt - 1) / kt;
        for (int64_t c = chunks0; c <= std::max<int64_t>(chunks0, g.Ly / 32); ++c) {
            const int64_t rows = (g.Ly + c - 1) / c, segs = std::max<int64_t>(1, 256 / rows), chunks = (g.Ly + rows - 1) / rows;
            // the fewest columns whose blocks make w waves, for the first w that hold them all and on, as long as
            // w waves without an idle block could still be shorter
            const double edge = 1.0 + (c > 1 ? 0.5 / (double)rows : 0.0);
            const double work = (double)g.Lx * (double)(chunks * groups) / (double)(slots * segs);
            const int64_t w0 = (chunks * groups + slots - 1) / slots;
            auto take = [&](int64_t room, double waves) {  // `room` blocks, which cost so many waves
                const int64_t nseg = room / (chunks * groups) * segs, cols = (g.Lx + nseg - 1) / nseg;
                const double t = waves * ((double)cols + 1.5) * edge * (kt == 2 ? 1.0 : cols <= 3 ? 0.6 : 0.8);
                if (t < best) {
                    best = t;
                    a.kt = kt;
                    a.rows = (int)rows;
                    a.segs = (int)segs;
                    a.cols = (int)cols;
                }
                return cols;
            };
            if (chunks * groups <= slots / 2) take(slots / 2, dots ? 0.6 : 0.7);
            for (int64_t w = w0; w <= std::max<int64_t>(w0, 64); ++w) {
                if ((work + 1.5 * (double)w) * edge * (kt == 2 ? 1.0 : 0.6) >= best) break;
                if (take(w * slots, (double)w) <= 1) break;
            }
        }
    }
}

static int64_t march_blocks(const MarchArgs& a) {
    const int64_t chunks = (a.g.Ly + a.rows - 1) / a.rows, n = (a.g.Lx + a.cols - 1) / a.cols;
    return chunks * ((n + a.segs - 1) / a.segs);
}

template <bool XR, int KT>
static cudaError_t launch_march(lm_ctx* ctx, const MarchArgs& a, bool first) {
    const int threads = (a.rows * a.segs + 31) / 32 * 32;
    for (int64_t m = 0; m < a.M; m += 65535ll * KT) {  // the grid's y extent is 65535
        MarchArgs b = a;
        b.M = std::min<int64_t>(a.M - m, 65535ll * KT);
        b.tp += m * a.ld;
        if (b.tpp) b.tpp += m * a.ld;
        b.out += m * a.ld;
        if (b.y) b.y += m * a.ld;
        if (b.part) b.part += m;
        const dim3 grid((unsigned)march_blocks(a), (unsigned)((b.M + KT - 1) / KT));
        if (first && a.y) df_march_kernel<XR, true, false, true, KT><<<grid, threads, 0, ctx->stream>>>(b);
        else if (first) df_march_kernel<XR, true, false, false, KT><<<grid, threads, 0, ctx->stream>>>(b);
        else if (a.part) df_march_kernel<XR, false, true, false, KT><<<grid, threads, 0, ctx->stream>>>(b);
        else df_march_kernel<XR, false, false, true, KT><<<grid, threads, 0, ctx->stream>>>(b);
        ctx->launches++;
    }
    return cudaGetLastError();
}

static cudaError_t march(lm_ctx* ctx, const MarchArgs& a, bool xr, bool first = false) {
    if (a.kt == 2) return xr ? launch_march<true, 2>(ctx, a, first) : launch_march<false, 2>(ctx, a, first);
    return xr ? launch_march<true, 1>(ctx, a, first) : launch_march<false, 1>(ctx, a, first);
}

// lm_cheb_apply with every column on chip through the whole series (lmgpu_series.cu): no recurrence
// buffers and one read and one write of the block.
static int cheb_apply_resident(lm_ham* h, const SeriesPlan& plan, double a, double b, const double* coef, int ncoef,
                               const double2* in, int64_t ld_in, lm_state* out) {
    lm_ctx* ctx = h->ctx;
    const Geom& g = h->lat->g;
    const size_t N = (size_t)g.N;
    const bool xr = ham_x_real(h);
    char* buf = nullptr;  // hops, gauge, diagonal, coefficients
    const size_t o_g = sizeof(float4) * N, o_d = o_g + (xr ? 0 : sizeof(double2) * N), o_c = o_d + sizeof(float2) * N;
    cudaError_t e = dev_alloc(ctx, (void**)&buf, o_c + sizeof(float2) * (size_t)ncoef);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return check_cuda(ctx, e, "lm_cheb_apply: allocation");
    }
    std::vector<float2> cd((size_t)ncoef);
    for (int k = 0; k < ncoef; ++k) {
        const float c = (float)coef[k];
        cd[(size_t)k] = make_float2(c, (float)(coef[k] - (double)c));
    }
    double2* gauge = xr ? nullptr : (double2*)(buf + o_g);
    e = cudaMemcpyAsync(buf + o_c, cd.data(), sizeof(float2) * (size_t)ncoef, cudaMemcpyHostToDevice, ctx->stream);
    if (e == cudaSuccess)
        e = launch_gauge_tables(ctx, g, h->d_hop, h->d_onsite, h->t1, a, b, xr, gauge, nullptr, nullptr, (float4*)buf,
                                (float2*)(buf + o_d));
    if (e == cudaSuccess) {
        SeriesArgs r;
        r.Lx = (int)g.Lx;
        r.Ly = (int)g.Ly;
        r.per_x = g.per_x;
        r.per_y = g.per_y;
        r.K = ncoef - 1;
        r.M = out->m;
        r.in = in;
        r.ld_in = ld_in;
        r.ld_out = out->ld;
        if (out->precision == LM_C64) r.out = (double2*)out->d_data;
        else r.out32 = (float2*)out->d_data;
        r.gauge = gauge;
        r.hy = buf;
        r.diag = buf + o_d;
        r.alpha = 2.0 * h->t1 / a;
        r.cd = (const float2*)(buf + o_c);
        e = launch_series_df(ctx, plan, r);
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    const int rc = e == cudaSuccess ? LM_OK : check_cuda(ctx, e, "lm_cheb_apply: on-chip series");
    dev_free(ctx, buf);
    return rc;
}

extern "C" {

int lm_kpm_moments(lm_ham* h, double emin, double emax, int nmom, const lm_state* vecs, int per_column,
                   double* out) {
    if (!h) return LM_ERR_ARG;
    lm_ctx* ctx = h->ctx;
    CHECK_ARG(ctx, out != nullptr, "lm_kpm_moments: null output");
    CHECK_ARG(ctx, nmom >= 1, "lm_kpm_moments: need at least one moment");
    CHECK_ARG(ctx, isfinite(emin) && isfinite(emax) && emax > emin, "lm_kpm_moments: need emin < emax");
    if (!h->assembled) return set_err(ctx, LM_ERR_STATE, "lm_kpm_moments: Hamiltonian not assembled");
    const Geom& g = h->lat->g;
    const int64_t N = g.N;
    if (vecs) {
        CHECK_ARG(ctx, vecs->ctx == ctx && vecs->n == N, "lm_kpm_moments: vectors do not match the lattice");
        CHECK_ARG(ctx, vecs->kind == LM_KETS && vecs->precision == LM_C64,
                  "lm_kpm_moments: vectors must be a ComplexF64 ket block");
    }
    const int64_t M = vecs ? vecs->m : N;
    const int64_t ld = vecs ? vecs->ld : N;
    const double a = 0.5 * (emax - emin), b = 0.5 * (emax + emin);
    const int64_t nsteps = (nmom + 1) / 2;  // recurrence passes: T_0 .. T_nsteps
    cudaSetDevice(ctx->device);

    double2* hop2 = nullptr;
    double* diag2 = nullptr;
    float2* hop2f = nullptr;
    float* diag2f = nullptr;
    double2* TA = nullptr;
    double2* TB = nullptr;
    double* dots = nullptr;
    float4* hopd = nullptr;  // double-float tables (LM_OPT_KPM, default on)
    float2* diagd = nullptr;
    const bool use_df = ctx->kpm_df != 0;
    const size_t blk = sizeof(double2) * (size_t)ld * (size_t)M;
    const size_t ndots = (size_t)(nsteps + 1) * 2 * (size_t)M;
    const bool xr = ham_x_real(h);
    MarchArgs ma{};
    ma.g = g;
    ma.ld = ld;
    ma.M = ma.pstride = M;
    march_plan(ctx, g, M, true, ma);
    const int64_t nblk = march_blocks(ma);
    double* part = nullptr;  // partial dots of kPartPasses passes
    auto release = [&]() {
        for (void* p : {(void*)hop2, (void*)diag2, (void*)hop2f, (void*)diag2f, (void*)TA, (void*)TB, (void*)dots, (void*)hopd,
                        (void*)diagd, (void*)part})
            dev_free(ctx, p);
    };
    cudaError_t e = dev_alloc(ctx, (void**)&hop2, sizeof(double2) * 2 * (size_t)N);
    if (e == cudaSuccess) e = dev_alloc(ctx, (void**)&diag2, sizeof(double) * (size_t)N);
    if (e == cudaSuccess) e = dev_alloc(ctx, (void**)&hop2f, sizeof(float2) * 2 * (size_t)N);
    if (e == cudaSuccess) e = dev_alloc(ctx, (void**)&diag2f, sizeof(float) * (size_t)N);
    if (e == cudaSuccess) e = dev_alloc(ctx, (void**)&TA, blk);
    if (e == cudaSuccess) e = dev_alloc(ctx, (void**)&TB, blk);
    if (e == cudaSuccess) e = dev_alloc(ctx, (void**)&dots, sizeof(double) * ndots);
    if (e == cudaSuccess && use_df) e = dev_alloc(ctx, (void**)&hopd, sizeof(float4) * 2 * (size_t)N);
    if (e == cudaSuccess && use_df) e = dev_alloc(ctx, (void**)&diagd, sizeof(float2) * (size_t)N);
    if (e == cudaSuccess && use_df)
        e = dev_alloc(ctx, (void**)&part, sizeof(double) * (size_t)(kPartPasses * nblk * 2 * M));
    if (e != cudaSuccess) {
        cudaGetLastError();
        release();
        return check_cuda(ctx, e, "lm_kpm_moments: allocation");
    }
    auto fail = [&](cudaError_t err, const char* what) {
        const int rc = check_cuda(ctx, err, what);
        release();
        return rc;
    };
    e = launch_normalise(ctx, g, h->d_hop, h->d_onsite, a, b, hop2, diag2, hop2f, diag2f);
    if (e != cudaSuccess) return fail(e, "lm_kpm_moments: tables");
    const unsigned dgrid = (unsigned)(M < 65535 ? M : 65535);
    if (use_df) {
        df_tables_kernel<<<(unsigned)std::min<int64_t>((2 * N + 255) / 256, 65535), 256, 0, ctx->stream>>>(
            hop2, diag2, N, hopd, diagd);
        to_df_kernel<<<dim3((unsigned)std::min<int64_t>((N + 255) / 256, 65535), dgrid), 256, 0, ctx->stream>>>(
            vecs ? (const double2*)vecs->d_data : nullptr, ld, N, M, (float4*)TA, ld);
        ctx->launches += 2;
        e = cudaGetLastError();
        if (e != cudaSuccess) return fail(e, "lm_kpm_moments: double-float conversion");
        const double al = h->t1 * (2.0 / a);
        ma.hop = hopd;
        ma.diag = diagd;
        ma.alpha = make_float2((float)al, (float)(al - (double)(float)al));
        ma.tp = (const float4*)TA;
        ma.out = (float4*)TB;
        e = march(ctx, ma, xr, true);  // T_1 = H~ T_0
        if (e != cudaSuccess) return fail(e, "lm_kpm_moments: recurrence");
        float4* Tn = (float4*)TA;   // T_n
        float4* Tn1 = (float4*)TB;  // T_{n+1}
        for (int64_t n = 0; n < nsteps; ++n) {  // T_{n+2} over T_n, and the dots of T_n and T_{n+1}
            ma.tp = Tn1;
            ma.tpp = Tn;
            ma.out = Tn;
            ma.part = part + (n % kPartPasses) * nblk * 2 * M;
            e = march(ctx, ma, xr);
            if (e != cudaSuccess) return fail(e, "lm_kpm_moments: recurrence");
            std::swap(Tn, Tn1);
            const int64_t np = n % kPartPasses + 1;
            if (np == kPartPasses || n + 1 == nsteps) {
                sum_parts_kernel<<<dim3((unsigned)((2 * M + 127) / 128), (unsigned)np), 128, 0, ctx->stream>>>(
                    part, (int)nblk, M, dots + (size_t)(n + 1 - np) * 2 * (size_t)M);
                ctx->launches++;
            }
        }
        column_dots2_df_kernel<<<dgrid, 256, 0, ctx->stream>>>(Tn, Tn1, N, ld, M, dots + (size_t)nsteps * 2 * (size_t)M);
        ctx->launches++;
        e = cudaGetLastError();
        if (e != cudaSuccess) return fail(e, "lm_kpm_moments: dots");
    } else {
        if (vecs) {
            e = cudaMemcpy2DAsync(TA, sizeof(double2) * (size_t)ld, vecs->d_data, sizeof(double2) * (size_t)vecs->ld,
                                  sizeof(double2) * (size_t)N, (size_t)M, cudaMemcpyDeviceToDevice, ctx->stream);
        } else {
            const dim3 grid((unsigned)((N + 255) / 256), (unsigned)(N < 65535 ? N : 65535));
            set_identity_kernel<<<grid, 256, 0, ctx->stream>>>(TA, N, ld);
            ctx->launches++;
            e = cudaGetLastError();
        }
        if (e != cudaSuccess) return fail(e, "lm_kpm_moments: starting block");
        // T_1 = H~ T_0
        e = launch_stencil_recur(ctx, g, LM_C64, hop2, diag2, TA, nullptr, nullptr, TB, ld, M, 0.5, 0.0, 0.0, nullptr,
                                 0.0, xr);
        if (e != cudaSuccess) return fail(e, "lm_kpm_moments: recurrence");
        double2* Tn = TA;   // T_n
        double2* Tn1 = TB;  // T_{n+1}
        for (int64_t n = 0; n <= nsteps; ++n) {
            double* d = dots + (size_t)n * 2 * (size_t)M;
            column_dots_kernel<<<dgrid, 256, 0, ctx->stream>>>(Tn, Tn, N, ld, M, d);
            column_dots_kernel<<<dgrid, 256, 0, ctx->stream>>>(Tn1, Tn, N, ld, M, d + M);
            ctx->launches += 2;
            e = cudaGetLastError();
            if (e != cudaSuccess) return fail(e, "lm_kpm_moments: dots");
            if (n == nsteps) break;
            // T_{n+2} = 2 H~ T_{n+1} - T_n, written over T_n
            e = launch_stencil_recur(ctx, g, LM_C64, hop2, diag2, Tn1, Tn, nullptr, Tn, ld, M, 1.0, 0.0, 0.0, nullptr,
                                     0.0, xr);
            if (e != cudaSuccess) return fail(e, "lm_kpm_moments: recurrence");
            std::swap(Tn, Tn1);
        }
    }
    std::vector<double> hd(ndots);
    e = cudaMemcpyAsync(hd.data(), dots, sizeof(double) * ndots, cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) return fail(e, "lm_kpm_moments: download");
    release();
    const int waited = vecs ? wait_status(ctx) : LM_OK;
    if (waited != LM_OK) return waited;
    // assemble the moments column by column (sums over columns in column order)
    const double* d0 = hd.data();
    for (int64_t col = 0; col < (per_column ? M : 1); ++col) {
        for (int k = 0; k < nmom; ++k) {
            const int64_t n = k / 2;
            double v = 0.0;
            for (int64_t c = per_column ? col : 0; c < (per_column ? col + 1 : M); ++c) {
                const double mu0 = d0[c], mu1 = d0[M + c];
                const double nn = d0[(size_t)n * 2 * M + c], n1n = d0[(size_t)n * 2 * M + M + c];
                v += (k == 0) ? mu0 : (k == 1) ? mu1 : (k % 2 == 0 ? 2.0 * nn - mu0 : 2.0 * n1n - mu1);
            }
            out[(size_t)col * (size_t)nmom + (size_t)k] = v;
        }
    }
    // |T_n(x)| <= 1 on [-1, 1]: larger moments mean that [emin, emax] misses part of the spectrum
    for (int64_t col = 0; col < (per_column ? M : 1); ++col) {
        const double* mu = out + (size_t)col * (size_t)nmom;
        for (int k = 1; k < nmom; ++k)
            if (!(fabs(mu[k]) <= fabs(mu[0]) * (1.0 + 1e-6) + 1e-12))
                return set_err(ctx, LM_ERR_NONFINITE,
                               "lm_kpm_moments: moments grow: [emin, emax] does not enclose the spectrum");
    }
    return LM_OK;
}

int lm_cheb_apply(lm_ham* h, double emin, double emax, const double* coef, int ncoef, const lm_state* in,
                  lm_state* out) {
    if (!h) return LM_ERR_ARG;
    lm_ctx* ctx = h->ctx;
    CHECK_ARG(ctx, coef != nullptr && ncoef >= 1, "lm_cheb_apply: need at least one coefficient");
    CHECK_ARG(ctx, out != nullptr && out->ctx == ctx, "lm_cheb_apply: bad output state");
    CHECK_ARG(ctx, isfinite(emin) && isfinite(emax) && emax > emin, "lm_cheb_apply: need emin < emax");
    for (int k = 0; k < ncoef; ++k) CHECK_ARG(ctx, isfinite(coef[k]), "lm_cheb_apply: non-finite coefficient");
    if (!h->assembled) return set_err(ctx, LM_ERR_STATE, "lm_cheb_apply: Hamiltonian not assembled");
    const Geom& g = h->lat->g;
    const int64_t N = g.N;
    if (in) CHECK_ARG(ctx, in->ctx == ctx && in->n == N, "lm_cheb_apply: input does not match the lattice");
    const int64_t M = in ? in->m : N;
    CHECK_ARG(ctx, out->n == N && out->m == M, "lm_cheb_apply: output shape differs from the input");
    const double a = 0.5 * (emax - emin), b = 0.5 * (emax + emin);
    cudaSetDevice(ctx->device);
    double2* hop2 = nullptr;
    double* diag2 = nullptr;
    float2* hop2f = nullptr;
    float* diag2f = nullptr;
    double2* TA = nullptr;
    double2* TB = nullptr;
    double2* Y = nullptr;
    float4* hopd = nullptr;  // double-float tables (LM_OPT_KPM, default on)
    float2* diagd = nullptr;
    const bool use_df = ctx->kpm_df != 0 && ncoef > 2;
    const int64_t ld = N;
    if (use_df && (!in || in->precision == LM_C64)) {
        const SeriesPlan plan = series_plan(ctx, g, ham_x_real(h), M, true);
        if (plan.kt)
            return cheb_apply_resident(h, plan, a, b, coef, ncoef, in ? (const double2*)in->d_data : nullptr,
                                       in ? in->ld : 0, out);
    }
    const size_t blk = sizeof(double2) * (size_t)ld * (size_t)M;
    auto release = [&]() {
        cudaStreamSynchronize(ctx->stream);
        for (void* p : {(void*)hop2, (void*)diag2, (void*)hop2f, (void*)diag2f, (void*)TA, (void*)TB, (void*)Y, (void*)hopd,
                        (void*)diagd})
            dev_free(ctx, p);
    };
    cudaError_t e = dev_alloc(ctx, (void**)&hop2, sizeof(double2) * 2 * (size_t)N);
    if (e == cudaSuccess) e = dev_alloc(ctx, (void**)&diag2, sizeof(double) * (size_t)N);
    if (e == cudaSuccess) e = dev_alloc(ctx, (void**)&hop2f, sizeof(float2) * 2 * (size_t)N);
    if (e == cudaSuccess) e = dev_alloc(ctx, (void**)&diag2f, sizeof(float) * (size_t)N);
    if (e == cudaSuccess) e = dev_alloc(ctx, (void**)&TA, blk);
    if (e == cudaSuccess && ncoef > 1) e = dev_alloc(ctx, (void**)&TB, blk);
    if (e == cudaSuccess) e = dev_alloc(ctx, (void**)&Y, blk);
    if (e == cudaSuccess && use_df) e = dev_alloc(ctx, (void**)&hopd, sizeof(float4) * 2 * (size_t)N);
    if (e == cudaSuccess && use_df) e = dev_alloc(ctx, (void**)&diagd, sizeof(float2) * (size_t)N);
    if (e != cudaSuccess) {
        cudaGetLastError();
        release();
        return check_cuda(ctx, e, "lm_cheb_apply: allocation");
    }
    auto fail = [&](cudaError_t err, const char* what) {
        const int rc = check_cuda(ctx, err, what);
        release();
        return rc;
    };
    e = launch_normalise(ctx, g, h->d_hop, h->d_onsite, a, b, hop2, diag2, hop2f, diag2f);
    if (e != cudaSuccess) return fail(e, "lm_cheb_apply: tables");
    const bool xr = ham_x_real(h);
    // T_0
    const dim3 cgrid((unsigned)std::min<int64_t>((N + 255) / 256, 65535), (unsigned)std::min<int64_t>(M, 65535));
    if (in && in->precision != LM_C64) {
        e = launch_convert(ctx, LM_C64, in->d_data, TA, N, M, in->ld, ld);
        if (e != cudaSuccess) return fail(e, "lm_cheb_apply: input block");
    }
    if (use_df) {
        const bool conv = in && in->precision != LM_C64;
        df_tables_kernel<<<(unsigned)std::min<int64_t>((2 * N + 255) / 256, 65535), 256, 0, ctx->stream>>>(
            hop2, diag2, N, hopd, diagd);
        to_df_kernel<<<cgrid, 256, 0, ctx->stream>>>(conv ? TA : in ? (const double2*)in->d_data : nullptr,
                                                     conv || !in ? ld : in->ld, N, M, (float4*)TA, ld);
        ctx->launches += 2;
        e = cudaGetLastError();
        if (e != cudaSuccess) return fail(e, "lm_cheb_apply: double-float conversion");
        auto split = [](double v) { return make_float2((float)v, (float)(v - (double)(float)v)); };
        MarchArgs ma{};
        ma.g = g;
        ma.ld = ld;
        ma.M = M;
        march_plan(ctx, g, M, false, ma);
        ma.hop = hopd;
        ma.diag = diagd;
        ma.alpha = split(h->t1 * (2.0 / a));
        ma.y = (float4*)Y;
        ma.c0 = split(coef[0]);
        ma.c = split(coef[1]);
        ma.tp = (const float4*)TA;
        ma.out = (float4*)TB;
        e = march(ctx, ma, xr, true);  // T_1 = H~ T_0, Y = c_0 T_0 + c_1 T_1
        float4* Tprev = (float4*)TA;
        float4* Tn = (float4*)TB;
        for (int k = 2; k < ncoef && e == cudaSuccess; ++k) {  // T_{n+1} over T_{n-1}, Y += c_{n+1} T_{n+1}
            ma.tp = Tn;
            ma.tpp = Tprev;
            ma.out = Tprev;
            ma.c = split(coef[k]);
            e = march(ctx, ma, xr);
            std::swap(Tprev, Tn);
        }
        if (e != cudaSuccess) return fail(e, "lm_cheb_apply: recurrence");
        from_df_kernel<<<cgrid, 256, 0, ctx->stream>>>((const float4*)Y, ld, N, M,
                                                       out->precision == LM_C64 ? (double2*)out->d_data : nullptr,
                                                       (float2*)out->d_data, out->ld);
        ctx->launches++;
        e = cudaGetLastError();
        if (e != cudaSuccess) return fail(e, "lm_cheb_apply: output");
        release();
        return LM_OK;
    }
    if (!in) {
        const dim3 grid((unsigned)((N + 255) / 256), (unsigned)(N < 65535 ? N : 65535));
        set_identity_kernel<<<grid, 256, 0, ctx->stream>>>(TA, N, ld);
        ctx->launches++;
        e = cudaGetLastError();
    } else if (in->precision == LM_C64) {
        e = cudaMemcpy2DAsync(TA, sizeof(double2) * (size_t)ld, in->d_data, sizeof(double2) * (size_t)in->ld,
                              sizeof(double2) * (size_t)N, (size_t)M, cudaMemcpyDeviceToDevice, ctx->stream);
    }
    if (e != cudaSuccess) return fail(e, "lm_cheb_apply: input block");
    // Y = c_0 T_0
    e = cudaMemcpyAsync(Y, TA, blk, cudaMemcpyDeviceToDevice, ctx->stream);
    if (e == cudaSuccess) e = launch_scale(ctx, LM_C64, Y, N, M, ld, coef[0], 0.0);
    if (e != cudaSuccess) return fail(e, "lm_cheb_apply: first term");
    if (ncoef > 1) {
        // T_1 = H~ T_0, Y += c_1 T_1; then T_{n+1} = 2 H~ T_n - T_{n-1} over T_{n-1}, Y += c_{n+1} T_{n+1}
        e = launch_stencil_recur(ctx, g, LM_C64, hop2, diag2, TA, nullptr, nullptr, TB, ld, M, 0.5, 0.0, 0.0, Y,
                                 coef[1], xr);
        double2* Tprev = TA;
        double2* Tn = TB;
        for (int k = 2; k < ncoef && e == cudaSuccess; ++k) {
            e = launch_stencil_recur(ctx, g, LM_C64, hop2, diag2, Tn, Tprev, nullptr, Tprev, ld, M, 1.0, 0.0, 0.0, Y,
                                     coef[k], xr);
            std::swap(Tprev, Tn);
        }
        if (e != cudaSuccess) return fail(e, "lm_cheb_apply: recurrence");
    }
    if (out->precision == LM_C64)
        e = cudaMemcpy2DAsync(out->d_data, sizeof(double2) * (size_t)out->ld, Y, sizeof(double2) * (size_t)ld,
                              sizeof(double2) * (size_t)N, (size_t)M, cudaMemcpyDeviceToDevice, ctx->stream);
    else
        e = launch_convert(ctx, LM_C32, Y, out->d_data, N, M, ld, out->ld);
    if (e != cudaSuccess) return fail(e, "lm_cheb_apply: output");
    release();
    return LM_OK;
}

int lm_ham_lanczos_bounds(lm_ham* h, int iters, unsigned long long seed, double* emin, double* emax) {
    if (!h) return LM_ERR_ARG;
    lm_ctx* ctx = h->ctx;
    CHECK_ARG(ctx, emin && emax, "lm_ham_lanczos_bounds: null output");
    CHECK_ARG(ctx, iters >= 2 && iters <= 10000, "lm_ham_lanczos_bounds: iters must be in 2..10000");
    if (!h->assembled) return set_err(ctx, LM_ERR_STATE, "lm_ham_lanczos_bounds: Hamiltonian not assembled");
    const Geom& g = h->lat->g;
    const int64_t N = g.N;
    double glo = 0.0, ghi = 0.0;
    lm_ham_bounds(h, &glo, &ghi);
    const int m = (int)std::min<int64_t>(iters, N);
    cudaSetDevice(ctx->device);
    double2* hop2 = nullptr;
    double* diag2 = nullptr;
    float2* hop2f = nullptr;
    float* diag2f = nullptr;
    double2* buf = nullptr;  // three vectors
    double* dot = nullptr;
    auto release = [&]() {
        cudaStreamSynchronize(ctx->stream);
        for (void* p : {(void*)hop2, (void*)diag2, (void*)hop2f, (void*)diag2f, (void*)buf, (void*)dot}) dev_free(ctx, p);
    };
    cudaError_t e = dev_alloc(ctx, (void**)&hop2, sizeof(double2) * 2 * (size_t)N);
    if (e == cudaSuccess) e = dev_alloc(ctx, (void**)&diag2, sizeof(double) * (size_t)N);
    if (e == cudaSuccess) e = dev_alloc(ctx, (void**)&hop2f, sizeof(float2) * 2 * (size_t)N);
    if (e == cudaSuccess) e = dev_alloc(ctx, (void**)&diag2f, sizeof(float) * (size_t)N);
    if (e == cudaSuccess) e = dev_alloc(ctx, (void**)&buf, sizeof(double2) * 3 * (size_t)N);
    if (e == cudaSuccess) e = dev_alloc(ctx, (void**)&dot, sizeof(double));
    if (e != cudaSuccess) {
        cudaGetLastError();
        release();
        return check_cuda(ctx, e, "lm_ham_lanczos_bounds: allocation");
    }
    auto fail = [&](cudaError_t err, const char* what) {
        const int rc = check_cuda(ctx, err, what);
        release();
        return rc;
    };
    // tables for a = 2, b = 0 hold H itself: the recurrence kernel then computes H v - u
    e = launch_normalise(ctx, g, h->d_hop, h->d_onsite, 2.0, 0.0, hop2, diag2, hop2f, diag2f);
    if (e != cudaSuccess) return fail(e, "lm_ham_lanczos_bounds: tables");
    double2* A = buf;          // v_j
    double2* B = buf + N;      // beta_{j-1} v_{j-1}
    double2* Cw = buf + 2 * N; // w
    const unsigned grid = (unsigned)std::min<int64_t>((N + 255) / 256, 4096);
    start_vector_kernel<<<grid, 256, 0, ctx->stream>>>(A, N, seed);
    e = cudaMemsetAsync(B, 0, sizeof(double2) * (size_t)N, ctx->stream);
    if (e != cudaSuccess) return fail(e, "lm_ham_lanczos_bounds: start");
    std::vector<double> al, be;
    auto read_dot = [&](const double2* x, const double2* y, double* v) -> cudaError_t {
        column_dots_kernel<<<1, 256, 0, ctx->stream>>>(x, y, N, N, 1, dot);
        cudaError_t err = cudaGetLastError();
        if (err == cudaSuccess) err = cudaMemcpyAsync(v, dot, sizeof(double), cudaMemcpyDeviceToHost, ctx->stream);
        if (err == cudaSuccess) err = cudaStreamSynchronize(ctx->stream);
        return err;
    };
    for (int j = 0; j < m; ++j) {
        // w = H v_j - beta_{j-1} v_{j-1}
        e = launch_stencil_recur(ctx, g, LM_C64, hop2, diag2, A, B, nullptr, Cw, N, 1, 1.0, 0.0, 0.0, nullptr, 0.0,
                                 ham_x_real(h));
        double alpha = 0.0, bsq = 0.0;
        if (e == cudaSuccess) e = read_dot(A, Cw, &alpha);
        if (e == cudaSuccess) {
            axpy_kernel<<<grid, 256, 0, ctx->stream>>>(Cw, A, -alpha, N);
            e = cudaGetLastError();
        }
        if (e == cudaSuccess) e = read_dot(Cw, Cw, &bsq);
        if (e != cudaSuccess) return fail(e, "lm_ham_lanczos_bounds: iteration");
        al.push_back(alpha);
        const double beta = sqrt(std::max(bsq, 0.0));
        if (j == m - 1 || beta <= 1e-12 * (fabs(ghi) + fabs(glo))) {
            be.push_back(beta);
            break;  // invariant subspace (or the last step): the tridiagonal is complete
        }
        be.push_back(beta);
        // B = beta v_j, v_{j+1} = w / beta, rotate the buffers
        scaled_copy_kernel<<<grid, 256, 0, ctx->stream>>>(B, A, beta, N);
        scaled_copy_kernel<<<grid, 256, 0, ctx->stream>>>(Cw, Cw, 1.0 / beta, N);
        e = cudaGetLastError();
        if (e != cudaSuccess) return fail(e, "lm_ham_lanczos_bounds: iteration");
        std::swap(A, Cw);
    }
    release();
    const int k = (int)al.size();
    std::vector<double> offd(be.begin(), be.begin() + (k - 1));
    const double lo = tridiag_eig(al, offd, 0, glo - 1.0, ghi + 1.0);
    const double hi = tridiag_eig(al, offd, k - 1, glo - 1.0, ghi + 1.0);
    // Ritz values lie inside the spectrum; pad each extreme by its residual beta_m |s_m| (an
    // eigenvalue lies within it) plus 1 % of the width, and never leave the Gershgorin interval
    const double rlo = be.back() * fabs(tridiag_last_component(al, offd, lo));
    const double rhi = be.back() * fabs(tridiag_last_component(al, offd, hi));
    const double w = 0.01 * (hi - lo);
    *emin = std::max(glo, lo - rlo - w);
    *emax = std::min(ghi, hi + rhi + w);
    return LM_OK;
}

}  // extern "C"
