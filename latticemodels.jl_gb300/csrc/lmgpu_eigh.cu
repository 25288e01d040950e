// Hermitian eigensystem on the device (FP64): the eigensolver behind diagonalize and
// densitymatrix (src/spectrum.jl:48-55, :226-257, :317-333), with no vendor library.
//
//   1. The assembled H is written as a dense N x N matrix (column-major).
//   2. Householder reduction to a real symmetric tridiagonal T = Q^H H Q: one cooperative launch
//      with the matrix in shared memory where it fits (2b), else on the lower triangle: per column one reflector (house_kernel), the symmetric product p = A v over
//      64 x 64 tiles with fixed-order partial sums (hemv_tiles_kernel, hemv_reduce_kernel),
//      and the rank-2 update A -= v w^H + w v^H of the lower tiles (her2_tiles_kernel).  The
//      reflectors stay in the strictly lower part of the matrix, as LAPACK's zhetrd keeps them
//      (Q = H_0 H_1 ... H_{n-2}, H_j = I - tau_j v_j v_j^H, v_j[0] = 1 at row j + 1).
//   3. T splits where an off-diagonal is below 2^-50 |T|; every eigenvalue of every block
//      comes from Sturm-count bisection to machine precision (1 to 32 lanes per eigenvalue).
//   4. Eigenvectors of T by inverse iteration with a pivoted tridiagonal LU, three solves from
//      a pseudo-random start; eigenvalues of a block closer than 1e-5 |T| form a cluster that
//      one thread computes in order, orthogonalising each iterate against the cluster's earlier
//      vectors (exactly degenerate levels of H sit in different blocks).
//   5. Back-transformation X = Q Z, columns in shared memory through all reflectors (one reflector
//      per launch where a column does not fit), and the weighted projector P = sum_k w_k x_k x_k^H
//      over lower tiles, accumulated over vector chunks.
//
// GB300 runs FP64 at two FMAs per clock per SM (1.84 reached), so every stage is bound by its FP64
// FMAs: the kernels spend none on anything else (complex products are four DFMAs).
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <numeric>
#include <vector>

#include "lmgpu_internal.cuh"
#include "lmgpu_order.cuh"

namespace {

using namespace lmgpu;

constexpr int kTile = 64;             // tile side of the tridiagonalisation and projector kernels
constexpr int kChunk = 1024;          // eigenvectors per back-transformation chunk
constexpr double kSplitRel = 8.881784197001252e-16;  // 2^-50: off-diagonals below kSplitRel |T| split T
constexpr double kClusterRel = 1e-5;  // eigenvalues closer than kClusterRel |T| form a cluster

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
    return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ double2 cfma(double2 a, double2 b, double2 c) {  // a*b + c
    return make_double2(fma(a.x, b.x, fma(-a.y, b.y, c.x)), fma(a.x, b.y, fma(a.y, b.x, c.y)));
}
__device__ __forceinline__ double2 cfma_conj(double2 a, double2 b, double2 c) {  // conj(a)*b + c
    return make_double2(fma(a.x, b.x, fma(a.y, b.y, c.x)), fma(a.x, b.y, fma(-a.y, b.x, c.y)));
}
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 conjd(double2 a) { return make_double2(a.x, -a.y); }

// ------------------------------------------------------------------------------------------
// 1. Dense assembly.  Square lattice: thread per column c accumulates every entry of column c
// in a fixed order (on-site, then the four bonds), so parallel bonds of a 2-site ring add up
// as the reference's builder adds them (src/operators/builder.jl:296-309).
// ------------------------------------------------------------------------------------------
__global__ void dense_square_kernel(Geom g, const double2* __restrict__ hop, const double* __restrict__ onsite,
                                    double2* __restrict__ A, int64_t lda) {
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= g.N) return;
    double2* col = A + c * lda;
    const Nbr nb = neighbours(g, c);
    col[c] = cadd(col[c], make_double2(onsite ? onsite[c] : 0.0, 0.0));
    if (nb.hxp) col[nb.xp] = cadd(col[nb.xp], conjd(hop[c]));            // H[xp, c] = conj(H[c, xp])
    if (nb.hxm) col[nb.xm] = cadd(col[nb.xm], hop[nb.xm]);               // H[xm, c] (the +x bond of xm)
    if (nb.hyp) col[nb.yp] = cadd(col[nb.yp], conjd(hop[g.N + c]));
    if (nb.hym) col[nb.ym] = cadd(col[nb.ym], hop[g.N + nb.ym]);
}

// General sparse H in ELL form: thread per row i adds its stored entries in slot order.
__global__ void dense_ell_kernel(int64_t n, int w, const int* __restrict__ cols, const double2* __restrict__ vals,
                                 const double* __restrict__ diag, double2* __restrict__ A, int64_t lda) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    A[i + i * lda] = cadd(A[i + i * lda], make_double2(diag[i], 0.0));
    for (int k = 0; k < w; ++k) {
        const int64_t c = cols[(int64_t)k * n + i];
        A[i + c * lda] = cadd(A[i + c * lda], vals[(int64_t)k * n + i]);
    }
}

// ------------------------------------------------------------------------------------------
// 2. Householder tridiagonalisation.
// ------------------------------------------------------------------------------------------
// Block-wide sum in a fixed order (deterministic): every thread passes its partial.
template <int NT>
__device__ __forceinline__ double block_sum(double v, double* sh) {
    const int t = threadIdx.x;
    sh[t] = v;
    __syncthreads();
#pragma unroll
    for (int s = NT / 2; s > 0; s >>= 1) {
        if (t < s) sh[t] += sh[t + s];
        __syncthreads();
    }
    const double r = sh[0];
    __syncthreads();
    return r;
}

// Reflector of column j: x = A[j+1:n, j], alpha = x[0].  H = I - tau v v^H with v = (1,
// x[1:]/(alpha - beta)) maps x to (beta, 0, ...), beta real (the zlarfg convention).  Writes
// d[j], e[j], tau[j], the scaled x back into A and v into vbuf; tau = 0 when x is already
// (real, 0, ...).
__global__ void __launch_bounds__(1024) house_kernel(double2* __restrict__ A, int64_t lda, int64_t n, int64_t j,
                                                     double* __restrict__ d, double* __restrict__ e,
                                                     double2* __restrict__ tau, double2* __restrict__ vbuf) {
    __shared__ double sh[1024];
    const int64_t m = n - 1 - j;  // length of x
    double2* x = A + (j + 1) + j * lda;
    // alpha is read before the reduction's barriers: thread 0 overwrites x[0] at the end
    const double2 alpha = x[0];
    double part = 0.0;
    for (int64_t i = 1 + threadIdx.x; i < m; i += blockDim.x) part = fma(x[i].x, x[i].x, fma(x[i].y, x[i].y, part));
    const double xn2 = block_sum<1024>(part, sh);
    // one thread forms the scalars: in every warp they would take 32 times the FP64 pipe
    __shared__ double2 sc_tau, sc_scal;
    __shared__ double sc_beta;
    if (threadIdx.x == 0) {
        double beta = alpha.x;
        double2 tv = make_double2(0.0, 0.0), scal = make_double2(1.0, 0.0);
        if (xn2 != 0.0 || alpha.y != 0.0) {
            const double nrm = sqrt(alpha.x * alpha.x + alpha.y * alpha.y + xn2);
            beta = alpha.x >= 0.0 ? -nrm : nrm;
            tv = make_double2((beta - alpha.x) / beta, -alpha.y / beta);
            const double2 den = make_double2(alpha.x - beta, alpha.y);  // 1 / (alpha - beta)
            const double dd = den.x * den.x + den.y * den.y;
            scal = make_double2(den.x / dd, -den.y / dd);
        }
        sc_beta = beta;
        sc_tau = tv;
        sc_scal = scal;
    }
    __syncthreads();
    const double beta = sc_beta;
    const double2 tv = sc_tau, scal = sc_scal;
    for (int64_t i = 1 + threadIdx.x; i < m; i += blockDim.x) {
        const double2 v = (tv.x != 0.0 || tv.y != 0.0) ? cmul(x[i], scal) : x[i];
        x[i] = v;
        vbuf[i] = v;
    }
    if (threadIdx.x == 0) {
        vbuf[0] = make_double2(1.0, 0.0);
        x[0] = make_double2(beta, 0.0);
        d[j] = A[j + j * lda].x;
        e[j] = beta;
        tau[j] = tv;
    }
}

// p = A22 v over the lower tiles of the trailing matrix A22 = A[o:n, o:n] (o = j + 1).  Tile
// (I, J), I >= J: part1[J][r] = sum over tile columns of A[r, c] v[c] for r in tile I, and for
// I > J part2[I][c] = sum over tile rows of conj(A[r, c]) v[r] for c in tile J.  The diagonal
// tile takes its upper half from the conjugate of the lower half.
__global__ void __launch_bounds__(256) hemv_tiles_kernel(const double2* __restrict__ A, int64_t lda, int64_t o,
                                                         int64_t m, int nt, const double2* __restrict__ v,
                                                         const double2* __restrict__ tau_j,
                                                         double2* __restrict__ part1, double2* __restrict__ part2) {
    if (tau_j->x == 0.0 && tau_j->y == 0.0) return;
    extern __shared__ double2 S[];  // kTile x (kTile + 1)
    __shared__ double2 red[4][kTile];
    // tile (I, J) from the linear lower-triangle index
    const int64_t q = blockIdx.x;
    int I = (int)((sqrt(8.0 * (double)q + 1.0) - 1.0) * 0.5);
    while ((int64_t)(I + 1) * (I + 2) / 2 <= q) ++I;
    while ((int64_t)I * (I + 1) / 2 > q) --I;
    const int J = (int)(q - (int64_t)I * (I + 1) / 2);
    const int64_t r0 = (int64_t)I * kTile, c0 = (int64_t)J * kTile;
    const int t = threadIdx.x;
    const int ld = kTile + 1;
    for (int k = t; k < kTile * kTile; k += 256) {
        const int rr = k % kTile, cc = k / kTile;
        const int64_t r = r0 + rr, c = c0 + cc;
        double2 a = make_double2(0.0, 0.0);
        if (r < m && c < m) {
            if (I != J || rr >= cc) a = A[(o + r) + (o + c) * lda];
            else a = conjd(A[(o + c) + (o + r) * lda]);
        }
        S[rr + cc * ld] = a;
    }
    __syncthreads();
    // row sums: thread (rr, group of 16 columns)
    {
        const int rr = t % kTile, g = t / kTile;
        double2 acc = make_double2(0.0, 0.0);
#pragma unroll 4
        for (int cc = g * 16; cc < g * 16 + 16; ++cc) {
            const int64_t c = c0 + cc;
            if (c < m) acc = cfma(S[rr + cc * ld], v[c], acc);
        }
        red[g][rr] = acc;
    }
    __syncthreads();
    if (t < kTile) {
        const int64_t r = r0 + t;
        if (r < m) part1[(int64_t)J * m + r] = cadd(cadd(red[0][t], red[1][t]), cadd(red[2][t], red[3][t]));
    }
    if (I == J) return;
    __syncthreads();
    // column sums: thread (cc, group of 16 rows)
    {
        const int cc = t % kTile, g = t / kTile;
        double2 acc = make_double2(0.0, 0.0);
#pragma unroll 4
        for (int rr = g * 16; rr < g * 16 + 16; ++rr) {
            const int64_t r = r0 + rr;
            if (r < m) acc = cfma_conj(S[rr + cc * ld], v[r], acc);
        }
        red[g][cc] = acc;
    }
    __syncthreads();
    if (t < kTile) {
        const int64_t c = c0 + t;
        if (c < m) part2[(int64_t)I * m + c] = cadd(cadd(red[0][t], red[1][t]), cadd(red[2][t], red[3][t]));
    }
}

// p[r] = tau (sum_{J <= I} part1[J][r] + sum_{I' > I} part2[I'][r]), I = r / kTile, in a fixed
// order; pdot[block] = sum over the block's rows of conj(p[r]) v[r].
__global__ void __launch_bounds__(256) hemv_reduce_kernel(int64_t m, int nt, const double2* __restrict__ part1,
                                                          const double2* __restrict__ part2,
                                                          const double2* __restrict__ v, const double2* __restrict__ tau_j,
                                                          double2* __restrict__ p, double2* __restrict__ pdot) {
    __shared__ double sh[256];
    const double2 tv = *tau_j;
    const int64_t r = (int64_t)blockIdx.x * 256 + threadIdx.x;
    double2 dp = make_double2(0.0, 0.0);
    if (r < m && (tv.x != 0.0 || tv.y != 0.0)) {
        const int I = (int)(r / kTile);
        double2 acc = make_double2(0.0, 0.0);
        for (int J = 0; J <= I; ++J) acc = cadd(acc, part1[(int64_t)J * m + r]);
        for (int I2 = I + 1; I2 < nt; ++I2) acc = cadd(acc, part2[(int64_t)I2 * m + r]);
        const double2 pr = cmul(tv, acc);
        p[r] = pr;
        dp = cfma_conj(pr, v[r], dp);
    }
    const double sx = block_sum<256>(dp.x, sh);
    const double sy = block_sum<256>(dp.y, sh);
    if (threadIdx.x == 0) pdot[blockIdx.x] = make_double2(sx, sy);
}

// A22 -= v w^H + w v^H on the lower tiles, w = p - (tau / 2) (p^H v) v; the diagonal stays
// real.  Every block sums the nb partial dots itself (fixed order).
__global__ void __launch_bounds__(256) her2_tiles_kernel(double2* __restrict__ A, int64_t lda, int64_t o, int64_t m,
                                                         const double2* __restrict__ v, const double2* __restrict__ p,
                                                         const double2* __restrict__ pdot, int nb,
                                                         const double2* __restrict__ tau_j) {
    const double2 tv = *tau_j;
    if (tv.x == 0.0 && tv.y == 0.0) return;
    __shared__ double2 wsh[2][kTile];
    __shared__ double2 vsh[2][kTile];
    const int64_t q = blockIdx.x;
    int I = (int)((sqrt(8.0 * (double)q + 1.0) - 1.0) * 0.5);
    while ((int64_t)(I + 1) * (I + 2) / 2 <= q) ++I;
    while ((int64_t)I * (I + 1) / 2 > q) --I;
    const int J = (int)(q - (int64_t)I * (I + 1) / 2);
    const int64_t r0 = (int64_t)I * kTile, c0 = (int64_t)J * kTile;
    double2 dot = make_double2(0.0, 0.0);
    for (int b = 0; b < nb; ++b) dot = cadd(dot, pdot[b]);
    const double2 al = cmul(make_double2(-0.5 * tv.x, -0.5 * tv.y), dot);  // -(tau/2) p^H v
    const int t = threadIdx.x;
    if (t < 2 * kTile) {
        const int side = t / kTile, k = t % kTile;
        const int64_t idx = (side == 0 ? r0 : c0) + k;
        double2 vv = make_double2(0.0, 0.0), ww = make_double2(0.0, 0.0);
        if (idx < m) {
            vv = v[idx];
            ww = cfma(al, vv, p[idx]);
        }
        vsh[side][k] = vv;
        wsh[side][k] = ww;
    }
    __syncthreads();
    for (int k = t; k < kTile * kTile; k += 256) {
        const int rr = k % kTile, cc = k / kTile;
        const int64_t r = r0 + rr, c = c0 + cc;
        if (r >= m || c >= m || (I == J && rr < cc)) continue;
        double2* a = A + (o + r) + (o + c) * lda;
        double2 x = *a;
        // x -= v_r conj(w_c) + w_r conj(v_c)
        const double2 vr = vsh[0][rr], wr = wsh[0][rr], vc = vsh[1][cc], wc = wsh[1][cc];
        x.x -= fma(vr.x, wc.x, fma(vr.y, wc.y, fma(wr.x, vc.x, wr.y * vc.y)));
        x.y -= fma(vr.y, wc.x, fma(-vr.x, wc.y, fma(wr.y, vc.x, -wr.x * vc.y)));
        if (r == c) x.y = 0.0;
        *a = x;
    }
}

// ------------------------------------------------------------------------------------------
// 2b. The same reduction in one cooperative launch, for matrices whose columns fit in the shared
// memory of all SMs together (n <= 8 SMs).  CTA b keeps the columns b, b + G, ... (at most 8, full
// columns, both triangles), so a product p_c = sum_r conj(A[r, c]) v_r needs no sum over CTAs and
// the row x_c = conj(A[j, c]) of the next reflector is spread over all of them.  Per column j:
//   warp 4 updates row j of the own columns (the next x) and posts x and a partial norm; the pass
//   warps apply the pending rank-2 update to rows r > j meanwhile (8 DFMAs per element);
//   exchange 1; the pass warps multiply the columns by x (4 DFMAs), warp 4 forms the reflector's
//   scalars; warp 4 posts p and a partial dot p^H v; exchange 2.
// v is never formed: v = scal xt with xt = x, xt[0] = alpha - beta, so scal folds into the
// per-column factors.  The update uses w = p + al v, v w^H + w v^H = v (p + 2 Re(al) v)^H + p v^H.
// An exchange: every value has a word of its own per column, set to a sentinel before the launch; a CTA
// posts its values, adds 1 to a counter without a fence, waits for the counter and loads what it
// needs, looking again at a word that still holds the sentinel.  A barrier with a fence took 5100
// clocks with the loads after it, this 3700; polling the words without the counter 12600 (each of the
// 152 stores into a line that all SMs poll costs a round trip between the dies).
// What bounds it: GB300's FP64 rate of 2 DFMAs per clock and SM in the early columns (storing
// both triangles costs 12 instead of 8 DFMAs per element, but no sum over CTAs), the exchanges and warp 4's
// chain in the late ones.  A warp-wide FP64 instruction holds a partition's pipe for 64 clocks even
// for one lane, so warp 4 has a lane per component of a complex scalar, and takes its root and
// reciprocals by Newton's iteration.  N = 864: 11.4 ms (5 ms of DFMAs); 13.5 ms with two fenced
// barriers and the update and product in one pass after the first, 49.8 ms with launches per column.
// ------------------------------------------------------------------------------------------
constexpr int kTriThreads = 160;      // 4 warps on the pass, 1 on the scalars
constexpr int kTriMaxCols = 8;        // columns per CTA
// Shared-memory limits of the resident kernels.  They are also the kernels' attribute, which is the device's,
// not a context's: a value that followed the matrix could be lowered by another thread before the launch.
constexpr int kTriMaxSmem = 224 * 1024;
constexpr int kBackMaxSmem = 220 * 1024;

// Sum of NV doubles per lane over the warp; lane k (k < NV, a power of two <= 32) returns the
// total of value k.  Halving the values with every exchange takes NV + log2(32 / NV) adds per warp.
template <int NV>
__device__ __forceinline__ double warp_fold(double (&v)[NV]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int w = NV / 2; w >= 1; w /= 2) {
        const bool up = (lane & w) != 0;
#pragma unroll
        for (int i = 0; i < w; ++i) {
            const double keep = up ? v[i + w] : v[i];
            const double send = up ? v[i] : v[i + w];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, w);
        }
    }
    double r = v[0];
#pragma unroll
    for (int w = NV; w < 32; w *= 2) r += __shfl_xor_sync(0xffffffffu, r, w);
    return r;  // lane l holds value l & (NV - 1)
}

struct TriArgs {
    double2* A;            // n x n column-major; column j receives the reflector v_j
    int64_t n;
    double* d;
    double* e;
    double2* tau;
    // Exchanged values, each written once per launch over the sentinel (all bits set):
    double2* xg;           // n x n: x of column j at j n
    double2* pg;           // n x n: p
    double* ng;            // G x n: partial norms
    double* dg;            // G x n: partial dots
    unsigned* ctr;         // columns' exchanges done, by all CTAs (zeroed)
    int* err;
};

// A value of the exchange is there when its bits are no longer the sentinel's; a NaN is stored as the
// plain quiet NaN.  Values are single 8-byte words, so no barrier or fence orders them.
__device__ __forceinline__ void post_word(double* p, double v) {
    long long u = __double_as_longlong(v);
    if (u == -1ll) u = 0x7ff8000000000000ll;
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(u) : "memory");
}
__device__ __forceinline__ long long peek_word(const double* p) {
    long long u;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(u) : "l"(p) : "memory");
    return u;
}
__device__ __forceinline__ void peek_pair(const double2* p, long long& x, long long& y) {
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(x), "=l"(y) : "l"(p) : "memory");
}

constexpr int kTriPolls = 1 << 20;  // bound of a wait for posted values (about half a second)

// One thread: adds this CTA to the exchange's counter and waits until all have come.  Most values are
// there then; no fence orders them, so each is still checked.
__device__ __forceinline__ bool meet(unsigned* ctr, unsigned target) {
    asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(ctr) : "memory");
    unsigned seen;
    int it = 0;
    do {
        asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(ctr) : "memory");
        if (++it > kTriPolls) return false;
    } while ((int)(seen - target) < 0);
    return true;
}
// The pass warps wait here until warp 4 has seen an exchange complete: polling the values themselves meanwhile
// slows their arrival, and polling a word of shared memory takes issue slots from warp 4 (11.4, 13.3 and
// 13.8 ms for N = 864).
__device__ __forceinline__ void gate_arrive(int id) {
    __syncwarp();
    asm volatile("barrier.arrive %0, %1;" ::"r"(id), "n"(kTriThreads) : "memory");
}
__device__ __forceinline__ void gate_wait(int id) {
    __syncwarp();
    asm volatile("barrier.sync %0, %1;" ::"r"(id), "n"(kTriThreads) : "memory");
}

// Waits for the pairs q[row[i]] with row[i] < n.  False when the wait gave up.
template <int U>
__device__ __forceinline__ bool wait_pairs(const double2* q, const int (&row)[U], int n, double2 (&v)[U]) {
    long long x[U], y[U];
#pragma unroll
    for (int i = 0; i < U; ++i) {
        x[i] = y[i] = 0;
        if (row[i] < n) peek_pair(q + row[i], x[i], y[i]);
    }
    bool ok = true;
#pragma unroll
    for (int i = 0; i < U; ++i) {
        int it = 0;
        while (x[i] == -1ll || y[i] == -1ll) {
            if (++it > kTriPolls) {
                ok = false;
                break;
            }
            peek_pair(q + row[i], x[i], y[i]);
        }
        v[i] = make_double2(__longlong_as_double(x[i]), __longlong_as_double(y[i]));
    }
    return ok;
}

// Sum over the warp of the words q[0 .. G), G <= 256, in a fixed order.
__device__ __forceinline__ bool wait_sum(const double* q, int G, int lane, double& sum) {
    constexpr int U = 8;
    long long x[U];
#pragma unroll
    for (int i = 0; i < U; ++i) {
        x[i] = 0;
        if (lane + 32 * i < G) x[i] = peek_word(q + lane + 32 * i);
    }
    bool ok = true;
    double s = 0.0;
#pragma unroll
    for (int i = 0; i < U; ++i) {
        int it = 0;
        while (x[i] == -1ll) {
            if (++it > kTriPolls) {
                ok = false;
                break;
            }
            x[i] = peek_word(q + lane + 32 * i);
        }
        if (32 * i < G) s = i == 0 ? __longlong_as_double(x[i]) : s + __longlong_as_double(x[i]);
    }
#pragma unroll
    for (int w = 16; w >= 1; w /= 2) s += __shfl_xor_sync(0xffffffffu, s, w);
    sum = s;
    return ok;
}

// 1 / sqrt(t) and 1 / d by Newton's iteration from the FP32 approximations, on arguments scaled into
// [1, 4) and [1, 2): two steps take their 22 bits beyond FP64's 53.  A quarter of the FP64 instructions of
// sqrt and a division.  Zero, subnormal and extreme arguments go the plain way.  Within 1.5 and 1 units in the
// last place of the exact values by the last step's roundings; 1.28 and 0.50 are the largest found.
__device__ __forceinline__ double newton_rsqrt(double t) {
    const int hi = __double2hiint(t), lo = __double2loint(t);
    const int ex = (hi >> 20) - 1023;
    if (ex < -900 || ex > 900) return 1.0 / sqrt(t);
    const int sc = ex & ~1, mh = hi - (sc << 20);
    const unsigned y = __float_as_uint(rsqrtf(__uint_as_float(((unsigned)(mh - (896 << 20)) << 3) | ((unsigned)lo >> 29))));
    const double m = __hiloint2double(mh, lo);
    double r = __hiloint2double((int)((y >> 3) + (896u << 20)), (int)(y << 29));
#pragma unroll
    for (int i = 0; i < 2; ++i) r = fma(0.5 * r, fma(-(m * r), r, 1.0), r);
    return __hiloint2double(__double2hiint(r) - ((sc / 2) << 20), __double2loint(r));
}
__device__ __forceinline__ double newton_recip(double d) {  // d > 0
    const int hi = __double2hiint(d), lo = __double2loint(d);
    const int ex = (hi >> 20) - 1023;
    if (ex < -900 || ex > 900) return 1.0 / d;
    const int mh = hi - (ex << 20);
    const unsigned y = __float_as_uint(__frcp_rn(__uint_as_float(((unsigned)(mh - (896 << 20)) << 3) | ((unsigned)lo >> 29))));
    const double m = __hiloint2double(mh, lo);
    double r = __hiloint2double((int)((y >> 3) + (896u << 20)), (int)(y << 29));
#pragma unroll
    for (int i = 0; i < 2; ++i) r = fma(r, fma(-m, r, 1.0), r);
    return __hiloint2double(__double2hiint(r) - (ex << 20), __double2loint(r));
}

__global__ void newton_kernel(const double* __restrict__ x, int64_t n, double* __restrict__ rs, double* __restrict__ rd) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    rs[i] = newton_rsqrt(x[i]);
    rd[i] = newton_recip(x[i]);
}

template <int NC>
__global__ void __launch_bounds__(kTriThreads, 1) tridiag_resident_kernel(TriArgs a) {
    extern __shared__ double2 sm[];
    const int n = (int)a.n, G = (int)gridDim.x, b = (int)blockIdx.x, t = threadIdx.x;
    const int warp = t >> 5, lane = t & 31;
    double2* S = sm;                  // column k at S + k n
    double2* ps = sm + (size_t)(NC + 2) * n;
    __shared__ double2 Gk[NC], Fk[NC], acc_sh[4][NC];
    for (int k = 0; k < NC; ++k) {
        const int c = b + k * G;
        if (c < n)
            for (int r = t; r < n; r += kTriThreads) S[(size_t)k * n + r] = a.A[r + (int64_t)c * a.n];
    }
    if (t < NC) Gk[t] = Fk[t] = make_double2(0.0, 0.0);
    for (int r = t; r < n; r += kTriThreads) ps[r] = sm[(size_t)NC * n + r] = sm[(size_t)(NC + 1) * n + r] = make_double2(0.0, 0.0);
    __syncthreads();
    constexpr int U = NC + 2;  // rows of a pass thread (n <= 152 NC takes one batch)
    constexpr int kFold = NC > 4 ? 8 : NC > 2 ? 4 : 2;  // a power of two >= NC (2 to 8)
    // warp 4: lane 2 k + i holds component i of column k's complex scalars (a warp-wide FP64 instruction
    // costs the same for one lane as for 32)
    const int kk = (lane >> 1) & (kFold - 1), im = lane & 1;
    const int kc = kk < NC ? kk : 0;
    const int c = b + kk * G;
    const bool own = warp == 4 && lane < 2 * NC && c < n;
    auto mul_part = [&](double2 u, double w0, double w1) {  // component im of u w: w0 this lane's part, w1 the other
        return fma(u.x, w0, im ? u.y * w1 : -u.y * w1);
    };
    auto other = [](double v) { return __shfl_xor_sync(0xffffffffu, v, 1); };
    unsigned met = 0;
    for (int j = 0; j + 1 < n; ++j) {
        double2* xp = sm + (size_t)(NC + ((j & 1) ^ 1)) * n;  // xt of the previous column
        double2* xn = sm + (size_t)(NC + (j & 1)) * n;        // x, then xt, of this one
        const double2* xj = a.xg + (int64_t)j * n;
        const double2* pj = a.pg + (int64_t)j * n;
        bool ok = true;
        double2 tv = make_double2(0.0, 0.0), scal = tv, den = tv, ts = tv;
        double vc = 0.0, tvc = 0.0;  // component im of v_c and of tau v_c
        auto row = [&](int q) { return j + 1 + 32 * (((warp + 3) & 3) + 4 * q) + lane; };  // of a pass thread
        if (warp == 4) {
            // row j of the own columns, updated: x_c = conj(A[j, c])
            double x = 0.0;
            if (own && c >= j) {
                const double2 v = S[(size_t)kc * n + j], xo = xp[j], po = ps[j], g = Gk[kc], f = Fk[kc];
                x = im ? v.y : v.x;
                x = fma(-xo.x, im ? g.y : g.x, x);
                x = fma(im ? -xo.y : xo.y, im ? g.x : g.y, x);
                x = fma(-po.x, im ? f.y : f.x, x);
                x = fma(im ? -po.y : po.y, im ? f.x : f.y, x);
                if (im) x = -x;
                if (c > j) post_word((double*)(xj + c) + im, x);
                else if (!im) a.d[j] = x;
            }
            double nn = own && c > j + 1 ? x * x : 0.0;
#pragma unroll
            for (int w = kFold; w >= 1; w /= 2) nn += __shfl_xor_sync(0xffffffffu, nn, w);
            met += G;
            __syncwarp();
            if (lane == 0) {
                post_word(a.ng + (int64_t)j * G + b, nn);
                ok = meet(a.ctr, met);
            }
            gate_arrive(1);
            // the reflector's scalars (the zlarfg convention, as house_kernel), by every lane
            double s;
            long long ax, ay;
            peek_pair(xj + j + 1, ax, ay);
            ok = wait_sum(a.ng + (int64_t)j * G, G, lane, s) && ok;
            for (int it = 0; ax == -1ll || ay == -1ll;) {
                if (++it > kTriPolls) {
                    ok = false;
                    break;
                }
                peek_pair(xj + j + 1, ax, ay);
            }
            const double2 alpha = make_double2(__shfl_sync(0xffffffffu, __longlong_as_double(ax), 0),
                                               __shfl_sync(0xffffffffu, __longlong_as_double(ay), 0));
            double beta = alpha.x;
            if (s != 0.0 || alpha.y != 0.0) {
                const double nn2 = fma(alpha.x, alpha.x, fma(alpha.y, alpha.y, s));
                const double rs = newton_rsqrt(nn2);
                double nrm = nn2 * rs;
                nrm = fma(fma(-nrm, nrm, nn2), 0.5 * rs, nrm);
                beta = alpha.x >= 0.0 ? -nrm : nrm;
                const double rb = alpha.x >= 0.0 ? -rs : rs;  // 1 / beta
                den = make_double2(alpha.x - beta, alpha.y);
                const double dd = fma(den.x, den.x, den.y * den.y);
                tv = make_double2(-den.x * rb, -alpha.y * rb);
                if (dd < 0x1p-1000) {  // 1 / dd may overflow where den / dd does not
                    scal = make_double2(den.x / dd, -den.y / dd);
                } else {
                    const double rd = newton_recip(dd);
                    scal = make_double2(den.x * rd, -den.y * rd);
                }
                const double tp = mul_part(tv, im ? scal.y : scal.x, im ? scal.x : scal.y), tq = other(tp);
                ts = make_double2(im ? tq : tp, im ? tp : tq);
            }
            if (b == 0 && lane == 0) {
                a.e[j] = beta;
                a.tau[j] = tv;
            }
            // v_c = scal xt_c and tau v_c
            const double xc = c == j + 1 ? (im ? den.y : den.x) : x;
            const double xo = other(xc);
            vc = mul_part(scal, xc, xo);
            const double vo = other(vc);
            tvc = mul_part(tv, vc, vo);
            if (!own || c <= j) vc = tvc = 0.0;
        } else {
            // the pending update of the own columns, rows r > j, while x travels
            for (int q = 0, r; (r = row(q)) < n; ++q) {
                const double2 xo = make_double2(-xp[r].x, -xp[r].y), po = make_double2(-ps[r].x, -ps[r].y);
#pragma unroll
                for (int k = 0; k < NC; ++k) {
                    if (b + k * G <= j || b + k * G >= n) continue;
                    double2 v = S[(size_t)k * n + r];
                    v = cfma(xo, Gk[k], v);
                    v = cfma(po, Fk[k], v);
                    S[(size_t)k * n + r] = v;
                }
            }
            // products with the new x (row j + 1 enters with xt = den once the scalars are known)
            double2 acc[NC];
#pragma unroll
            for (int k = 0; k < NC; ++k) acc[k] = make_double2(0.0, 0.0);
            gate_wait(1);
            for (int q = 0; row(q) < n; q += U) {
                double2 x[U];
                int rows[U];
#pragma unroll
                for (int i = 0; i < U; ++i) rows[i] = row(q + i);
                ok = wait_pairs(xj, rows, n, x) && ok;
#pragma unroll
                for (int i = 0; i < U; ++i) {
                    const int r = rows[i];
                    if (r >= n) break;
                    xn[r] = x[i];
                    if (r == j + 1) x[i] = make_double2(0.0, 0.0);
#pragma unroll
                    for (int k = 0; k < NC; ++k) {
                        if (b + k * G <= j || b + k * G >= n) continue;
                        acc[k] = cfma_conj(S[(size_t)k * n + r], x[i], acc[k]);
                    }
                }
            }
            constexpr int NV = 2 * kFold;
            double v[NV];
#pragma unroll
            for (int i = 0; i < NV; ++i) v[i] = i / 2 < NC ? ((i & 1) ? acc[i / 2 < NC ? i / 2 : 0].y : acc[i / 2 < NC ? i / 2 : 0].x) : 0.0;
            const double tot = warp_fold<NV>(v);
            if (lane < 2 * NC) {
                double* dst = (double*)&acc_sh[warp][lane >> 1];
                dst[lane & 1] = tot;
            }
        }
        if (__syncthreads_or(!ok)) {
            if (t == 0) *(volatile int*)a.err = 1;
            return;
        }
        if (warp == 4) {
            double pc = 0.0;
            if (own && c > j) {
                const double2 s1 = S[(size_t)kc * n + j + 1];
                const double* q0 = (const double*)&acc_sh[0][kc] + im;
                double q = (q0[0] + q0[2 * NC]) + (q0[4 * NC] + q0[6 * NC]);
                q = fma(s1.x, im ? den.y : den.x, q);
                pc = fma(im ? -s1.y : s1.y, im ? den.x : den.y, q);
            }
            const double qo = other(pc);
            pc = mul_part(ts, pc, qo);
            if (own && c > j) {
                post_word((double*)(pj + c) + im, pc);
                ((double*)(a.A + c + (int64_t)j * n))[im] = vc;
            }
            double dp = own && c > j ? pc * tvc : 0.0;  // Re(tau conj(p) v), summed over both components
#pragma unroll
            for (int w = kFold; w >= 1; w /= 2) dp += __shfl_xor_sync(0xffffffffu, dp, w);
            met += G;
            __syncwarp();
            if (lane == 0) {
                post_word(a.dg + (int64_t)j * G + b, dp);
                ok = meet(a.ctr, met);
            }
            gate_arrive(2);
            double s;
            ok = wait_sum(a.dg + (int64_t)j * G, G, lane, s) && ok;  // -2 Re(al), al = -(tau / 2) p^H v
            // F = conj(v), G = scal (conj(p) + 2 Re(al) conj(v))
            const double f = im ? -vc : vc;
            const double g = fma(-s, f, im ? -pc : pc);
            const double go = other(g);
            const double gs = mul_part(scal, g, go);
            if (lane < 2 * NC) {
                const bool on = own && c > j;
                ((double*)&Fk[kc])[im] = on ? f : 0.0;
                ((double*)&Gk[kc])[im] = on ? gs : 0.0;
            }
            if (lane == 0) xn[j + 1] = den;
        } else {
            gate_wait(2);
            for (int q = 0; row(q) < n; q += U) {
                double2 p[U];
                int rows[U];
#pragma unroll
                for (int i = 0; i < U; ++i) rows[i] = row(q + i);
                ok = wait_pairs(pj, rows, n, p) && ok;
#pragma unroll
                for (int i = 0; i < U; ++i)
                    if (rows[i] < n) ps[rows[i]] = p[i];
            }
        }
        if (__syncthreads_or(!ok)) {
            if (t == 0) *(volatile int*)a.err = 1;
            return;
        }
    }
    // the last diagonal entry: column n - 1, row n - 1, with the last update
    if (t < NC && b + t * G == n - 1) {
        double2 v = S[(size_t)t * n + n - 1];
        if (n > 1) {
            const double2* xp = sm + (size_t)(NC + ((n - 2) & 1)) * n;
            v = cfma(make_double2(-xp[n - 1].x, -xp[n - 1].y), Gk[t], v);
            v = cfma(make_double2(-ps[n - 1].x, -ps[n - 1].y), Fk[t], v);
        }
        a.A[(n - 1) + (int64_t)(n - 1) * a.n] = v;
    }
}

// ------------------------------------------------------------------------------------------
// 3. Bisection: `split` lanes per (block, local index k) look for the k-th smallest eigenvalue of
// the block T[s:s+len, s:s+len]; every pass cuts the interval into split + 1 parts by Sturm counts
// at the lanes' points.  The count is the number of sign changes of the leading principal minors
// p_{i+1} = (d_i - x) p_i - e_{i-1}^2 p_{i-1} (Wilkinson's form; each step is the exact one of a
// diagonal entry and a squared off-diagonal within a few ulp), rescaled by a power of two every
// four steps; a zero minor takes the sign opposite to the one before.  T comes scaled to norm 1.
// What bounds it: the FP64 pipe's latency and rate.  The pivot form q = d - x - e^2 / q holds one
// division (a dozen dependent DFMAs) per row, the minors two multiplications and an addition:
// N = 864 takes 1.8 ms (28 ms with one lane per eigenvalue and the pivot form).
// ------------------------------------------------------------------------------------------
struct BisectJob {
    int s, len, k, pad;
    double lo, hi;
};

__device__ __forceinline__ int sturm_count(const double2* __restrict__ de, int len, double x) {
    // de[i] = (d_i, e_{i-1}^2), de[0].y unused
    double p0 = 1.0, p1 = de[0].x - x;
    int neg = (p1 <= 0.0);  // sign of the current minor; p_0 > 0
    int cnt = neg;
    int i = 1;
    auto step = [&](double2 q) {
        const double p2 = fma(q.x - x, p1, -(q.y * p0));
        const int hi = __double2hiint(p2);
        const bool zero = ((hi << 1) | __double2loint(p2)) == 0;
        const int ng = zero ? neg ^ 1 : (int)((unsigned)hi >> 31);
        cnt += ng ^ neg;
        neg = ng;
        p0 = p1;
        p1 = p2;
    };
    for (; i + 4 <= len; i += 4) {
        double2 q[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) q[u] = de[i + u];
#pragma unroll
        for (int u = 0; u < 4; ++u) step(q[u]);
        const int ex = max(__double2hiint(p0) & 0x7ff00000, __double2hiint(p1) & 0x7ff00000);
        const double sc = __hiloint2double(0x7fe00000 - max(ex, 0x00100000), 0);  // the larger one to [1, 2)
        p0 *= sc;
        p1 *= sc;
    }
    for (; i < len; ++i) step(de[i]);
    return cnt;
}

// tiny: absolute width at which the search stops (far below the rounding of T itself)
__global__ void __launch_bounds__(32) bisect_kernel(const double2* __restrict__ de, const BisectJob* __restrict__ jobs,
                                                    int64_t njobs, int split, double tiny, double* __restrict__ out) {
    const int64_t q = ((int64_t)blockIdx.x * 32 + threadIdx.x) / split;
    const int lane = threadIdx.x, i = lane % split, base = lane - i;
    BisectJob job{0, 1, 0, 0, 0.0, 0.0};
    if (q < njobs) job = jobs[q];
    double lo = job.lo, hi = job.hi;
    const double frac = (double)(i + 1) / (double)(split + 1);
    const unsigned group = split == 32 ? 0xffffffffu : ((1u << split) - 1u) << base;
    for (int it = 0; it < 200; ++it) {
        const bool done = !(hi - lo > 2.0 * DBL_EPSILON * fmax(fabs(lo), fabs(hi)) + tiny);
        if (__all_sync(0xffffffffu, done)) break;
        const double x = fma(hi - lo, frac, lo);
        const bool above = done || sturm_count(de + job.s, job.len, x) > job.k;
        __syncwarp();
        const unsigned m = (__ballot_sync(0xffffffffu, above) & group) >> base;
        const int first = m ? __ffs(m) - 1 : split;  // the first point with more than k eigenvalues below
        const double xl = __shfl_sync(0xffffffffu, x, base + max(first - 1, 0));
        const double xh = __shfl_sync(0xffffffffu, x, base + min(first, split - 1));
        if (!done) {
            const double l0 = lo, h0 = hi;
            if (first > 0) lo = fmax(lo, xl);
            if (first < split) hi = fmin(hi, xh);
            if (lo == l0 && hi == h0) lo = hi = 0.5 * (lo + hi);  // the interval holds no more doubles
        }
    }
    if (i == 0 && q < njobs) out[q] = 0.5 * (lo + hi);
}

// ------------------------------------------------------------------------------------------
// 4. Inverse iteration, thread per cluster.  Members of cluster q are mem[q0 .. q0+cnt) with
// eigenvalue lam[], block (s, len) and a vector in vec (len used rows).  Scratch per cluster: the
// multipliers, reciprocal pivots, two superdiagonals (len each) and the pivot flags.
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ double hash_unit(uint64_t a, uint64_t b) {  // deterministic value in [-1, 1)
    uint64_t x = a * 0x9E3779B97F4A7C15ull ^ (b + 0x632BE59BD9B4E019ull);
    x ^= x >> 31; x *= 0xBF58476D1CE4E5B9ull; x ^= x >> 29; x *= 0x94D049BB133111EBull; x ^= x >> 32;
    return (double)(x >> 11) * (2.0 / 9007199254740992.0) - 1.0;
}

// Thread-per-cluster arrays are interleaved (row i of cluster q at [i ncl + q], of member mi at
// [i nmem + mi]), so a warp's accesses are consecutive, and every sweep loads kSteinRows rows
// before it uses them.  The pivots are kept as reciprocals: one division per row in the
// factorisation and none in the three solves.  432 vectors of N = 864 take 1.9 ms (5.6 ms with a
// division per row and solve and a vector per thread in memory order).
constexpr int kSteinRows = 8;

__global__ void __launch_bounds__(32) stein_kernel(const double* __restrict__ d, const double* __restrict__ e,
                                                   int64_t ncl, int64_t nmem, const int64_t* __restrict__ cl_first,
                                                   const int64_t* __restrict__ cl_count,
                                                   const int64_t* __restrict__ mem_s,
                                                   const int64_t* __restrict__ mem_len,
                                                   const double* __restrict__ mem_lam,
                                                   const int64_t* __restrict__ mem_seed, double* __restrict__ vec,
                                                   double* __restrict__ scratch, int64_t lmax, double pert) {
    const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= ncl) return;
    const int64_t f = cl_first[q], cnt = cl_count[q];
    const int64_t s = mem_s[f], len = mem_len[f];
    double* __restrict__ dl = scratch + q;               // multipliers
    double* __restrict__ rd = dl + ncl * lmax;           // reciprocal pivots
    double* __restrict__ du = rd + ncl * lmax;           // first superdiagonal
    double* __restrict__ du2 = du + ncl * lmax;          // second; NaN-free, 0 where no interchange
    unsigned char* __restrict__ piv = (unsigned char*)(scratch + 4 * ncl * lmax) + q;  // rows i, i + 1 interchanged
    for (int64_t u = 0; u < cnt; ++u) {
        const int64_t mi = f + u;
        const double lam = mem_lam[mi];
        double* __restrict__ x = vec + mi;
        if (len == 1) {
            x[0] = 1.0;
            continue;
        }
        auto recip = [&](double p) { return 1.0 / (fabs(p) < pert ? (p < 0.0 ? -pert : pert) : p); };
        // LU of T_b - lam I with partial pivoting
        double dc = d[s] - lam, uc = e[s];
        for (int64_t i0 = 0; i0 + 1 < len; i0 += kSteinRows) {
            double ev[kSteinRows + 1], dv[kSteinRows];
#pragma unroll
            for (int k = 0; k <= kSteinRows; ++k) ev[k] = i0 + k + 1 < len ? e[s + i0 + k] : 0.0;
#pragma unroll
            for (int k = 0; k < kSteinRows; ++k) dv[k] = i0 + k + 1 < len ? d[s + i0 + k + 1] : 0.0;
#pragma unroll
            for (int k = 0; k < kSteinRows; ++k) {
                const int64_t i = i0 + k;
                if (i + 1 < len) {
                    const double l = ev[k], dn = dv[k] - lam, un = ev[k + 1];
                    const bool swap = fabs(dc) < fabs(l);
                    const double p = swap ? l : dc;
                    const double r = recip(p);
                    const double fct = (swap ? dc : l) * r;
                    rd[i * ncl] = r;
                    dl[i * ncl] = fct;
                    du[i * ncl] = swap ? dn : uc;
                    du2[i * ncl] = swap ? un : 0.0;
                    piv[i * ncl] = swap;
                    dc = swap ? fma(-fct, dn, uc) : fma(-fct, uc, dn);
                    uc = swap ? -fct * un : un;
                }
            }
        }
        rd[(len - 1) * ncl] = recip(dc);
        double fac = 1.0;
        for (int it = 0; it < 4; ++it) {
            // orthogonalise against the cluster's earlier vectors
            if (mi > f && it == 0)
                for (int64_t i = 0; i < len; ++i) x[i * nmem] = hash_unit((uint64_t)mem_seed[mi], (uint64_t)i);
            for (int64_t p = f; p < mi; ++p) {
                const double* z = vec + p;
                double dot = 0.0;
#pragma unroll 8
                for (int64_t i = 0; i < len; ++i) dot = fma(z[i * nmem], x[i * nmem], dot);
                for (int64_t i0 = 0; i0 < len; i0 += kSteinRows) {
                    double zv[kSteinRows], xv[kSteinRows];
#pragma unroll
                    for (int k = 0; k < kSteinRows; ++k) {
                        const int64_t i = min(i0 + k, len - 1);
                        zv[k] = z[i * nmem];
                        xv[k] = x[i * nmem];
                    }
#pragma unroll
                    for (int k = 0; k < kSteinRows; ++k)
                        if (i0 + k < len) x[(i0 + k) * nmem] = fma(-dot, zv[k], xv[k]);
                }
            }
            if (it == 3) break;
            // solve L U y = fac x in place: forwards
            const bool fresh = it == 0 && mi == f;  // the start vector is formed on the way
            double xc = fac * (fresh ? hash_unit((uint64_t)mem_seed[mi], 0) : x[0]);
            for (int64_t i0 = 0; i0 + 1 < len; i0 += kSteinRows) {
                double lv[kSteinRows], xv[kSteinRows];
                unsigned char pv[kSteinRows];
#pragma unroll
                for (int k = 0; k < kSteinRows; ++k) {
                    const int64_t i = min(i0 + k, len - 2);
                    lv[k] = dl[i * ncl];
                    pv[k] = piv[i * ncl];
                    xv[k] = fac * (fresh ? hash_unit((uint64_t)mem_seed[mi], (uint64_t)(i + 1)) : x[(i + 1) * nmem]);
                }
#pragma unroll
                for (int k = 0; k < kSteinRows; ++k)
                    if (i0 + k + 1 < len) {
                        const double top = pv[k] ? xv[k] : xc, low = pv[k] ? xc : xv[k];
                        x[(i0 + k) * nmem] = top;
                        xc = fma(-lv[k], top, low);
                    }
            }
            // backwards, with the largest entry on the way
            double x1 = xc * rd[(len - 1) * ncl], x2 = 0.0, mx = fabs(x1);
            x[(len - 1) * nmem] = x1;
            for (int64_t i0 = len - 2; i0 >= 0; i0 -= kSteinRows) {
                double rv[kSteinRows], uv[kSteinRows], wv[kSteinRows], xv[kSteinRows];
#pragma unroll
                for (int k = 0; k < kSteinRows; ++k) {
                    const int64_t i = max(i0 - k, (int64_t)0);
                    rv[k] = rd[i * ncl];
                    uv[k] = du[i * ncl];
                    wv[k] = du2[i * ncl];
                    xv[k] = x[i * nmem];
                }
#pragma unroll
                for (int k = 0; k < kSteinRows; ++k)
                    if (i0 - k >= 0) {
                        const double v = fma(-uv[k], x1, fma(-wv[k], x2, xv[k])) * rv[k];
                        x[(i0 - k) * nmem] = v;
                        x2 = x1;
                        x1 = v;
                        mx = fmax(mx, fabs(v));
                    }
            }
            // normalise (largest entry first, then the 2-norm); the factor is applied by the next use
            const double sm = mx > 0.0 ? 1.0 / mx : 1.0;
            double nrm = 0.0;
#pragma unroll 8
            for (int64_t i = 0; i < len; ++i) {
                const double v = x[i * nmem] * sm;
                nrm = fma(v, v, nrm);
            }
            fac = sm / sqrt(nrm);
            if (cnt > 1 || it == 2) {
                for (int64_t i0 = 0; i0 < len; i0 += kSteinRows) {
                    double xv[kSteinRows];
#pragma unroll
                    for (int k = 0; k < kSteinRows; ++k) xv[k] = x[min(i0 + k, len - 1) * nmem];
#pragma unroll
                    for (int k = 0; k < kSteinRows; ++k)
                        if (i0 + k < len) x[(i0 + k) * nmem] = xv[k] * fac;
                }
                fac = 1.0;
            }
        }
        // final normalisation and sign: the entry of largest magnitude is positive
        double nrm = 0.0, mx = 0.0, xm = 1.0;
#pragma unroll 8
        for (int64_t i = 0; i < len; ++i) {
            const double v = x[i * nmem];
            nrm = fma(v, v, nrm);
            if (fabs(v) > mx) { mx = fabs(v); xm = v; }
        }
        const double inv = (xm < 0.0 ? -1.0 : 1.0) / sqrt(nrm);
        for (int64_t i0 = 0; i0 < len; i0 += kSteinRows) {
            double xv[kSteinRows];
#pragma unroll
            for (int k = 0; k < kSteinRows; ++k) xv[k] = x[min(i0 + k, len - 1) * nmem];
#pragma unroll
            for (int k = 0; k < kSteinRows; ++k)
                if (i0 + k < len) x[(i0 + k) * nmem] = xv[k] * inv;
        }
    }
}

// X[:, k] = Z[:, k] as complex (column k's block rows from the member vector, zero elsewhere)
__global__ void scatter_vectors_kernel(int64_t n, int64_t nv, const int64_t* __restrict__ col_mem,
                                       const int64_t* __restrict__ mem_s, const int64_t* __restrict__ mem_len,
                                       const double* __restrict__ vec, int64_t nmem, double2* __restrict__ X,
                                       int64_t ldx) {
    const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t k = blockIdx.y;
    if (r >= n || k >= nv) return;
    const int64_t mi = col_mem[k];
    const int64_t s = mem_s[mi], len = mem_len[mi];
    X[r + k * ldx] = make_double2((r >= s && r < s + len) ? vec[(r - s) * nmem + mi] : 0.0, 0.0);
}

// ------------------------------------------------------------------------------------------
// 5. Back-transformation: X <- H_j X = X - tau_j v_j (v_j^H X) on rows j+1.., one block per
// column (the dot, then the update; the second read of the column comes from L2).
// ------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) apply_reflector_kernel(const double2* __restrict__ A, int64_t lda, int64_t n,
                                                              int64_t j, const double2* __restrict__ tau,
                                                              double2* __restrict__ X, int64_t ldx, int64_t nv) {
    __shared__ double sh[256];
    const double2 tv = tau[j];
    if (tv.x == 0.0 && tv.y == 0.0) return;
    const int64_t k = blockIdx.x;
    if (k >= nv) return;
    const int64_t o = j + 1, m = n - o;
    const double2* v = A + o + j * lda;  // v[0] = 1 (stored as beta), v[i] = A[o+i, j]
    double2* x = X + o + k * ldx;
    double2 dp = make_double2(0.0, 0.0);
    for (int64_t i = threadIdx.x; i < m; i += 256) {
        const double2 vi = i == 0 ? make_double2(1.0, 0.0) : v[i];
        dp = cfma_conj(vi, x[i], dp);
    }
    const double sx = block_sum<256>(dp.x, sh);
    const double sy = block_sum<256>(dp.y, sh);
    const double2 g = cmul(tv, make_double2(-sx, -sy));  // -tau (v^H x)
    for (int64_t i = threadIdx.x; i < m; i += 256) {
        const double2 vi = i == 0 ? make_double2(1.0, 0.0) : v[i];
        x[i] = cfma(vi, g, x[i]);
    }
}

// The same for C columns per CTA kept in shared memory through every reflector: a column never
// depends on another, so the whole back-transformation is one launch without a grid-wide step.
// Reflector j - 1 is on its way (cp.async) while j is applied; a thread reads only the rows it
// copied, so the two block barriers per reflector are those of the dot.  Bound by the FP64 rate
// (8 DFMAs per row, column and reflector): 432 columns of N = 864 in 4.2 ms (2.1 ms of DFMAs),
// against 8.3 ms with one launch per reflector (9.6 us each, mostly its tree sum over 256 threads).
constexpr int kBackThreads = 128;
constexpr int kBackMaxCols = 8;

template <int C>
__global__ void __launch_bounds__(kBackThreads) back_resident_kernel(const double2* __restrict__ A, int64_t lda, int n,
                                                                     const double2* __restrict__ tau,
                                                                     double2* __restrict__ X, int64_t ldx, int64_t nv) {
    extern __shared__ double2 sm[];
    __shared__ double2 part[kBackThreads / 32][C];
    __shared__ double2 gsh[C];
    double2* xs = sm;                                   // column k at xs + k n
    auto vb = [&](int j) { return sm + (size_t)(C + (j & 1)) * n; };  // reflector j
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const int64_t k0 = (int64_t)blockIdx.x * C;
    auto first_row = [&](int o) { return t + (o > t ? (o - t + kBackThreads - 1) / kBackThreads * kBackThreads : 0); };
    auto fetch = [&](int j) {
        if (j >= 0)
            for (int r = first_row(j + 1); r < n; r += kBackThreads) {
                const unsigned dst = (unsigned)__cvta_generic_to_shared(vb(j) + r);
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(A + r + (int64_t)j * lda));
            }
        asm volatile("cp.async.commit_group;");
    };
    fetch(n - 2);
#pragma unroll
    for (int k = 0; k < C; ++k)
        for (int r = t; r < n; r += kBackThreads)
            xs[(size_t)k * n + r] = k0 + k < nv ? X[r + (k0 + k) * ldx] : make_double2(0.0, 0.0);
    for (int j = n - 2; j >= 0; --j) {
        fetch(j - 1);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        const double2 tv = tau[j];
        if (tv.x == 0.0 && tv.y == 0.0) continue;
        const double2* v = vb(j);
        double2 acc[C];
#pragma unroll
        for (int k = 0; k < C; ++k) acc[k] = make_double2(0.0, 0.0);
        const int rb = first_row(j + 1);
        for (int r = rb; r < n; r += kBackThreads) {
            const double2 vi = r == j + 1 ? make_double2(1.0, 0.0) : v[r];
#pragma unroll
            for (int k = 0; k < C; ++k) acc[k] = cfma_conj(vi, xs[(size_t)k * n + r], acc[k]);
        }
        constexpr int NV = C <= 1 ? 2 : C <= 2 ? 4 : C <= 4 ? 8 : 16;
        double f[NV];
#pragma unroll
        for (int i = 0; i < NV; ++i) f[i] = i / 2 < C ? ((i & 1) ? acc[i / 2 < C ? i / 2 : 0].y : acc[i / 2 < C ? i / 2 : 0].x) : 0.0;
        const double tot = warp_fold<NV>(f);
        if (lane < 2 * C) ((double*)&part[warp][lane >> 1])[lane & 1] = tot;
        __syncthreads();
        if (t < C) {
            const double2 d = cadd(cadd(part[0][t], part[1][t]), cadd(part[2][t], part[3][t]));
            gsh[t] = cmul(tv, make_double2(-d.x, -d.y));  // -tau (v^H x)
        }
        __syncthreads();
        for (int r = rb; r < n; r += kBackThreads) {
            const double2 vi = r == j + 1 ? make_double2(1.0, 0.0) : v[r];
#pragma unroll
            for (int k = 0; k < C; ++k) xs[(size_t)k * n + r] = cfma(vi, gsh[k], xs[(size_t)k * n + r]);
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
    for (int k = 0; k < C; ++k)
        if (k0 + k < nv)
            for (int r = t; r < n; r += kBackThreads) X[r + (k0 + k) * ldx] = xs[(size_t)k * n + r];
}

// P[r, c] += sum_k w_k X[r, k] conj(X[c, k]) on the lower TS x TS tiles of P (I >= J); the
// weights are staged per chunk of 16 vectors.  Bound by the FP64 rate, so the tile side is the
// one that fills the SMs: 64 where there are several tiles per SM, 32 below (N = 864: 105 tiles of
// 64 leave 47 SMs idle, 1.83 ms; 378 of 32 take 1.4 ms).
template <int TS>
__global__ void __launch_bounds__(256) projector_tiles_kernel(const double2* __restrict__ X, int64_t ldx, int64_t n,
                                                              int64_t nv, const double* __restrict__ w,
                                                              double2* __restrict__ P, int64_t ldp) {
    constexpr int Q = TS / 16;
    __shared__ double2 xr[16][TS];
    __shared__ double2 xc[16][TS];
    const int64_t q = blockIdx.x;
    int I = (int)((sqrt(8.0 * (double)q + 1.0) - 1.0) * 0.5);
    while ((int64_t)(I + 1) * (I + 2) / 2 <= q) ++I;
    while ((int64_t)I * (I + 1) / 2 > q) --I;
    const int J = (int)(q - (int64_t)I * (I + 1) / 2);
    const int64_t r0 = (int64_t)I * TS, c0 = (int64_t)J * TS;
    const int t = threadIdx.x;
    const int tr = t % 16, tc = t / 16;  // thread owns rows tr + 16 a, columns tc + 16 b (a, b < Q)
    double2 acc[Q][Q];
#pragma unroll
    for (int a = 0; a < Q; ++a)
#pragma unroll
        for (int b = 0; b < Q; ++b) acc[a][b] = make_double2(0.0, 0.0);
    for (int64_t k0 = 0; k0 < nv; k0 += 16) {
        for (int u = t; u < 16 * TS; u += 256) {
            const int kk = u / TS, rr = u % TS;
            const int64_t k = k0 + kk;
            double2 a = make_double2(0.0, 0.0), b = make_double2(0.0, 0.0);
            if (k < nv) {
                const double wk = w[k];
                if (r0 + rr < n) {
                    a = X[(r0 + rr) + k * ldx];
                    a = make_double2(a.x * wk, a.y * wk);
                }
                if (c0 + rr < n) b = X[(c0 + rr) + k * ldx];
            }
            xr[kk][rr] = a;
            xc[kk][rr] = b;
        }
        __syncthreads();
#pragma unroll 4
        for (int kk = 0; kk < 16; ++kk) {
            double2 ra[Q], cb[Q];
#pragma unroll
            for (int a = 0; a < Q; ++a) ra[a] = xr[kk][tr + 16 * a];
#pragma unroll
            for (int b = 0; b < Q; ++b) cb[b] = xc[kk][tc + 16 * b];
#pragma unroll
            for (int a = 0; a < Q; ++a)
#pragma unroll
                for (int b = 0; b < Q; ++b) acc[a][b] = cfma_conj(cb[b], ra[a], acc[a][b]);  // ra conj(cb)
        }
        __syncthreads();
    }
#pragma unroll
    for (int a = 0; a < Q; ++a)
#pragma unroll
        for (int b = 0; b < Q; ++b) {
            const int64_t r = r0 + tr + 16 * a, c = c0 + tc + 16 * b;
            if (r < n && c < n && r >= c) {
                double2* pp = P + r + c * ldp;
                *pp = cadd(*pp, acc[a][b]);
            }
        }
}

// upper triangle of P from its lower triangle; the diagonal made real
__global__ void hermitian_fill_kernel(double2* __restrict__ P, int64_t ldp, int64_t n) {
    const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    for (int64_t c = blockIdx.y; c < n; c += gridDim.y) {
        if (r < c) P[r + c * ldp] = conjd(P[c + r * ldp]);
        else if (r == c) P[r + c * ldp].y = 0.0;
    }
}

// convert a c64 block into c32 (column-major, leading dimensions given)
__global__ void to_c32_kernel(const double2* __restrict__ src, int64_t lds, float2* __restrict__ dst, int64_t ldd,
                              int64_t n, int64_t ncols) {
    const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    for (int64_t c = blockIdx.y; c < ncols; c += gridDim.y) {
        const double2 v = src[r + c * lds];
        dst[r + c * ldd] = make_float2((float)v.x, (float)v.y);
    }
}

inline unsigned grid_y(int64_t ncols) { return (unsigned)std::min<int64_t>(std::max<int64_t>(ncols, 1), 65535); }

}  // namespace

// ------------------------------------------------------------------------------------------
// Host side.
// ------------------------------------------------------------------------------------------
struct lm_eigsys {
    lm_ctx* ctx = nullptr;
    int64_t n = 0;
    double2* d_A = nullptr;     // n x n; Householder vectors below the subdiagonal after the reduction
    double2* d_tau = nullptr;   // n - 1 reflector scalars
    double* d_d = nullptr;      // tridiagonal (device copies after splitting)
    double* d_e = nullptr;
    std::vector<double> d, e;   // host copies; e zero where T splits
    double tnorm = 0.0;
    std::vector<int64_t> blk_s, blk_len;  // blocks of T
    // eigenvalues ascending, with their block and index within the block
    std::vector<double> w;
    std::vector<int64_t> w_blk, w_k;
};

namespace {

template <typename T>
int dalloc_t(lm_ctx* ctx, T** p, size_t count, const char* what) {
    cudaError_t e = dev_alloc(ctx, (void**)p, sizeof(T) * std::max<size_t>(count, 1));
    if (e != cudaSuccess) {
        *p = nullptr;
        cudaGetLastError();
        return set_err(ctx, e == cudaErrorMemoryAllocation ? LM_ERR_OOM : LM_ERR_CUDA,
                       std::string("eigensolver: cannot allocate ") + what);
    }
    return LM_OK;
}

template <typename T>
int upload_vec(lm_ctx* ctx, T** dptr, const std::vector<T>& h, const char* what) {
    int rc = dalloc_t(ctx, dptr, h.size(), what);
    if (rc != LM_OK) return rc;
    if (!h.empty())
        CUDA_TRY(ctx, cudaMemcpyAsync(*dptr, h.data(), sizeof(T) * h.size(), cudaMemcpyHostToDevice, ctx->stream),
                 "eigensolver: upload");
    return LM_OK;
}

struct DevFree {
    explicit DevFree(lm_ctx* c) : ctx(c) {}
    lm_ctx* ctx;
    std::vector<void*> ptrs;
    ~DevFree() {
        for (void* p : ptrs) dev_free(ctx, p);
    }
    template <typename T>
    T* keep(T* p) {
        ptrs.push_back((void*)p);
        return p;
    }
};

void free_eigsys(lm_eigsys* e) {
    dev_free(e->ctx, e->d_A);
    dev_free(e->ctx, e->d_tau);
    dev_free(e->ctx, e->d_d);
    dev_free(e->ctx, e->d_e);
    e->d_A = nullptr;
    e->d_tau = nullptr;
    e->d_d = nullptr;
    e->d_e = nullptr;
}

// Columns per CTA of the resident tridiagonalisation, 0 where it does not apply: every column and
// three more vectors of n complex numbers have to fit in an SM's shared memory.
int tri_resident_cols(const lm_ctx* ctx, int64_t n) {
    const int64_t c = (n + ctx->sm_count - 1) / ctx->sm_count;
    return n >= 2 && c <= kTriMaxCols && (c + 3) * n * (int64_t)sizeof(double2) <= kTriMaxSmem ? (int)c : 0;
}

template <int NC>
cudaError_t launch_tri(lm_ctx* ctx, TriArgs a, int grid) {
    const size_t smem = sizeof(double2) * (size_t)(NC + 3) * (size_t)a.n;
    cudaError_t e = cudaFuncSetAttribute(tridiag_resident_kernel<NC>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTriMaxSmem);
    if (e != cudaSuccess) return e;
    void* args[] = {&a};
    return cudaLaunchCooperativeKernel((const void*)tridiag_resident_kernel<NC>, dim3(grid), dim3(kTriThreads), args, smem,
                                       ctx->stream);
}

// One launch sequence per column on the lower tiles: matrices beyond the resident form.
int reduce_tiles(lm_eigsys* es, DevFree& tmp) {
    lm_ctx* ctx = es->ctx;
    const int64_t n = es->n;
    int rc = LM_OK;
    const int64_t m0 = std::max<int64_t>(n - 1, 1);
    const int nt0 = (int)((m0 + kTile - 1) / kTile);
    double2 *d_v = nullptr, *d_p = nullptr, *d_part1 = nullptr, *d_part2 = nullptr, *d_pdot = nullptr;
    rc = dalloc_t(ctx, &d_v, (size_t)m0, "reflector");
    if (rc == LM_OK) rc = dalloc_t(ctx, &d_p, (size_t)m0, "product");
    if (rc == LM_OK) rc = dalloc_t(ctx, &d_part1, (size_t)nt0 * (size_t)m0, "partial sums");
    if (rc == LM_OK) rc = dalloc_t(ctx, &d_part2, (size_t)nt0 * (size_t)m0, "partial sums");
    if (rc == LM_OK) rc = dalloc_t(ctx, &d_pdot, (size_t)(m0 + 255) / 256, "partial dots");
    tmp.keep(d_v); tmp.keep(d_p); tmp.keep(d_part1); tmp.keep(d_part2); tmp.keep(d_pdot);
    if (rc != LM_OK) return rc;
    constexpr int kSmem = (int)sizeof(double2) * kTile * (kTile + 1);
    CUDA_TRY(ctx, cudaFuncSetAttribute(hemv_tiles_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem),
             "eigensolver: shared memory attribute");
    for (int64_t j = 0; j + 1 < n; ++j) {
        const int64_t m = n - 1 - j, o = j + 1;
        const int nt = (int)((m + kTile - 1) / kTile);
        const int64_t ntiles = (int64_t)nt * (nt + 1) / 2;
        const int nb = (int)((m + 255) / 256);
        house_kernel<<<1, 1024, 0, ctx->stream>>>(es->d_A, n, n, j, es->d_d, es->d_e, es->d_tau, d_v);
        hemv_tiles_kernel<<<(unsigned)ntiles, 256, kSmem, ctx->stream>>>(es->d_A, n, o, m, nt, d_v, es->d_tau + j,
                                                                       d_part1, d_part2);
        hemv_reduce_kernel<<<nb, 256, 0, ctx->stream>>>(m, nt, d_part1, d_part2, d_v, es->d_tau + j, d_p, d_pdot);
        her2_tiles_kernel<<<(unsigned)ntiles, 256, 0, ctx->stream>>>(es->d_A, n, o, m, d_v, d_p, d_pdot, nb,
                                                                     es->d_tau + j);
        ctx->launches += 4;
        if ((j & 255) == 0) CUDA_TRY(ctx, cudaGetLastError(), "eigensolver: tridiagonalisation");
    }
    CUDA_TRY(ctx, cudaGetLastError(), "eigensolver: tridiagonalisation");
    return LM_OK;
}

int reduce_resident(lm_eigsys* es, DevFree& tmp) {
    lm_ctx* ctx = es->ctx;
    const int64_t n = es->n;
    // two or more columns per CTA: fewer CTAs make the barriers cheaper, and below 300 rows the
    // pass over a column is shorter than a barrier
    const int nc = std::max(tri_resident_cols(ctx, n), (int)std::min<int64_t>(n, 2));
    const int grid = (int)((n + nc - 1) / nc);
    // x, p, partial norms and dots of every column, over the sentinel; and the error word
    const size_t words = 4 * (size_t)n * (size_t)n + 2 * (size_t)grid * (size_t)n;
    double* buf = nullptr;
    int rc = dalloc_t(ctx, &buf, words + 2, "tridiagonalisation exchange");
    tmp.keep(buf);
    if (rc != LM_OK) return reduce_tiles(es, tmp);  // its buffers are smaller
    TriArgs a;
    a.A = es->d_A;
    a.n = n;
    a.d = es->d_d;
    a.e = es->d_e;
    a.tau = es->d_tau;
    a.err = (int*)buf;
    a.ctr = (unsigned*)(buf + 1);
    a.xg = (double2*)(buf + 2);
    a.pg = a.xg + n * n;
    a.ng = (double*)(a.pg + n * n);
    a.dg = a.ng + (size_t)grid * n;
    CUDA_TRY(ctx, cudaMemsetAsync(buf, 0, 16, ctx->stream), "eigensolver: clear status");
    CUDA_TRY(ctx, cudaMemsetAsync(buf + 2, 0xff, sizeof(double) * words, ctx->stream), "eigensolver: clear exchange");
    cudaError_t e;
    switch (nc) {
        case 2: e = launch_tri<2>(ctx, a, grid); break;
        case 3: e = launch_tri<3>(ctx, a, grid); break;
        case 4: e = launch_tri<4>(ctx, a, grid); break;
        case 5: e = launch_tri<5>(ctx, a, grid); break;
        case 6: e = launch_tri<6>(ctx, a, grid); break;
        case 7: e = launch_tri<7>(ctx, a, grid); break;
        default: e = launch_tri<8>(ctx, a, grid); break;
    }
    CUDA_TRY(ctx, e, "eigensolver: tridiagonalisation");
    ctx->launches++;
    int err = 0;
    CUDA_TRY(ctx, cudaMemcpyAsync(&err, a.err, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream), "eigensolver: status");
    CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream), "eigensolver: synchronize");
    if (err) return set_err(ctx, LM_ERR_TIMEOUT, "eigensolver: a wait of the tridiagonalisation gave up");
    return LM_OK;
}

// Householder reduction of es->d_A (filled with the dense H), then splitting and bisection.
int reduce_and_solve(lm_eigsys* es) {
    lm_ctx* ctx = es->ctx;
    const int64_t n = es->n;
    int rc = dalloc_t(ctx, &es->d_tau, (size_t)std::max<int64_t>(n - 1, 1), "reflector scalars");
    if (rc == LM_OK) rc = dalloc_t(ctx, &es->d_d, (size_t)n, "tridiagonal");
    if (rc == LM_OK) rc = dalloc_t(ctx, &es->d_e, (size_t)std::max<int64_t>(n - 1, 1), "tridiagonal");
    if (rc != LM_OK) return rc;
    DevFree tmp(ctx);
    rc = tri_resident_cols(ctx, n) ? reduce_resident(es, tmp) : reduce_tiles(es, tmp);
    if (rc != LM_OK) return rc;
    es->d.assign((size_t)n, 0.0);
    es->e.assign((size_t)std::max<int64_t>(n - 1, 0), 0.0);
    // d[n-1] is the last diagonal entry of the reduced matrix
    CUDA_TRY(ctx, cudaMemcpyAsync(es->d_d + (n - 1), es->d_A + (n - 1) + (n - 1) * n, sizeof(double),
                                  cudaMemcpyDeviceToDevice, ctx->stream),
             "eigensolver: last diagonal");
    CUDA_TRY(ctx, cudaMemcpyAsync(es->d.data(), es->d_d, sizeof(double) * n, cudaMemcpyDeviceToHost, ctx->stream),
             "eigensolver: download");
    if (n > 1)
        CUDA_TRY(ctx, cudaMemcpyAsync(es->e.data(), es->d_e, sizeof(double) * (n - 1), cudaMemcpyDeviceToHost,
                                      ctx->stream),
                 "eigensolver: download");
    CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream), "eigensolver: synchronize");
    for (double v : es->d)
        if (!std::isfinite(v)) return set_err(ctx, LM_ERR_NONFINITE, "eigensolver: non-finite tridiagonal");
    for (double v : es->e)
        if (!std::isfinite(v)) return set_err(ctx, LM_ERR_NONFINITE, "eigensolver: non-finite tridiagonal");
    // norm, splitting
    double tn = 0.0;
    for (int64_t i = 0; i < n; ++i) {
        double r = fabs(es->d[(size_t)i]);
        if (i > 0) r += fabs(es->e[(size_t)i - 1]);
        if (i + 1 < n) r += fabs(es->e[(size_t)i]);
        tn = std::max(tn, r);
    }
    es->tnorm = tn;
    es->blk_s.clear();
    es->blk_len.clear();
    int64_t s0 = 0;
    for (int64_t i = 0; i + 1 < n; ++i) {
        if (fabs(es->e[(size_t)i]) <= kSplitRel * tn) {
            es->e[(size_t)i] = 0.0;
            es->blk_s.push_back(s0);
            es->blk_len.push_back(i + 1 - s0);
            s0 = i + 1;
        }
    }
    es->blk_s.push_back(s0);
    es->blk_len.push_back(n - s0);
    if (n > 1)
        CUDA_TRY(ctx, cudaMemcpyAsync(es->d_e, es->e.data(), sizeof(double) * (n - 1), cudaMemcpyHostToDevice,
                                      ctx->stream),
                 "eigensolver: upload");
    // bisection jobs on T scaled by a power of two to norm about 1
    const int ex = tn > 0.0 ? std::ilogb(tn) : 0;
    std::vector<double2> de((size_t)n);
    for (int64_t i = 0; i < n; ++i) {
        const double ei = i > 0 ? std::scalbn(es->e[(size_t)i - 1], -ex) : 0.0;
        de[(size_t)i] = make_double2(std::scalbn(es->d[(size_t)i], -ex), ei * ei);
    }
    std::vector<BisectJob> jobs;
    jobs.reserve((size_t)n);
    for (size_t b = 0; b < es->blk_s.size(); ++b) {
        const int64_t s = es->blk_s[b], len = es->blk_len[b];
        double lo = 1e300, hi = -1e300;
        for (int64_t i = s; i < s + len; ++i) {
            double r = 0.0;
            if (i > s) r += fabs(es->e[(size_t)i - 1]);
            if (i + 1 < s + len) r += fabs(es->e[(size_t)i]);
            lo = std::min(lo, std::scalbn(es->d[(size_t)i] - r, -ex));
            hi = std::max(hi, std::scalbn(es->d[(size_t)i] + r, -ex));
        }
        const double pad = 2.0 * DBL_EPSILON * std::max(fabs(lo), fabs(hi)) * (double)len + 2.0 * DBL_MIN;
        for (int64_t k = 0; k < len; ++k)
            jobs.push_back(BisectJob{(int)s, (int)len, (int)k, 0, lo - pad, hi + pad});
    }
    double2* d_de = nullptr;
    double* d_out = nullptr;
    BisectJob* d_jobs = nullptr;
    rc = upload_vec(ctx, &d_de, de, "bisection");
    if (rc == LM_OK) rc = upload_vec(ctx, &d_jobs, jobs, "bisection");
    if (rc == LM_OK) rc = dalloc_t(ctx, &d_out, (size_t)n, "bisection");
    tmp.keep(d_de); tmp.keep(d_jobs); tmp.keep(d_out);
    if (rc != LM_OK) return rc;
    // lanes per eigenvalue: as many as keep about one warp per SM partition (a warp instruction holds
    // a partition's FP64 pipe for 64 clocks, so a second warp costs more than its extra cuts save:
    // N = 864 with 4 / 16 lanes takes 3.1 / 1.8 ms)
    int split = 32;
    while (split > 1 && n * split > 128ll * ctx->sm_count) split >>= 1;
    bisect_kernel<<<(unsigned)((n * split + 31) / 32), 32, 0, ctx->stream>>>(d_de, d_jobs, n, split, 0x1p-80, d_out);
    ctx->launches++;
    CUDA_TRY(ctx, cudaGetLastError(), "eigensolver: bisection");
    std::vector<double> vals((size_t)n);
    CUDA_TRY(ctx, cudaMemcpyAsync(vals.data(), d_out, sizeof(double) * n, cudaMemcpyDeviceToHost, ctx->stream),
             "eigensolver: download");
    CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream), "eigensolver: synchronize");
    for (double& v : vals) v = std::scalbn(v, ex);
    // eigenvalues ascending; ties keep the block order
    std::vector<int64_t> ord((size_t)n);
    std::iota(ord.begin(), ord.end(), 0);
    std::stable_sort(ord.begin(), ord.end(), [&](int64_t a, int64_t b) { return vals[(size_t)a] < vals[(size_t)b]; });
    es->w.resize((size_t)n);
    es->w_blk.resize((size_t)n);
    es->w_k.resize((size_t)n);
    std::vector<int64_t> blk_of_start;
    for (int64_t i = 0; i < n; ++i) {
        const int64_t t = ord[(size_t)i];
        es->w[(size_t)i] = vals[(size_t)t];
        es->w_k[(size_t)i] = jobs[(size_t)t].k;
        // block index from the job's start row
        const int64_t s = jobs[(size_t)t].s;
        es->w_blk[(size_t)i] = std::lower_bound(es->blk_s.begin(), es->blk_s.end(), s) - es->blk_s.begin();
    }
    return LM_OK;
}

int check_lm_state_dense(lm_ctx* ctx, const lm_state* st, int64_t n, int kind, const char* who) {
    if (!st) return set_err(ctx, LM_ERR_ARG, std::string(who) + ": null state");
    if (st->ctx != ctx) return set_err(ctx, LM_ERR_ARG, std::string(who) + ": state belongs to another context");
    if (st->n != n || st->kind != kind)
        return set_err(ctx, LM_ERR_ARG, std::string(who) + ": state shape does not match the eigensystem");
    return LM_OK;
}

// Columns per CTA of the resident back-transformation: one wave over the SMs where shared memory
// allows it (C columns and two reflectors of n complex numbers); 0 where not one column fits.
int back_resident_cols(const lm_ctx* ctx, int64_t n, int64_t nv) {
    const int64_t fit = kBackMaxSmem / (n * (int64_t)sizeof(double2)) - 2;
    const int64_t want = (nv + ctx->sm_count - 1) / ctx->sm_count;
    return n >= 2 && fit >= 1 ? (int)std::min<int64_t>({want, fit, (int64_t)kBackMaxCols}) : 0;
}

template <int C>
cudaError_t launch_back_t(lm_eigsys* es, double2* X, int64_t ldx, int64_t nv) {
    const size_t smem = sizeof(double2) * (size_t)(C + 2) * (size_t)es->n;
    cudaError_t e = cudaFuncSetAttribute(back_resident_kernel<C>, cudaFuncAttributeMaxDynamicSharedMemorySize, kBackMaxSmem);
    if (e != cudaSuccess) return e;
    back_resident_kernel<C><<<(unsigned)((nv + C - 1) / C), kBackThreads, smem, es->ctx->stream>>>(
        es->d_A, es->n, (int)es->n, es->d_tau, X, ldx, nv);
    es->ctx->launches++;
    return cudaGetLastError();
}

cudaError_t launch_back(lm_eigsys* es, double2* X, int64_t ldx, int64_t nv, int cols) {
    switch (cols) {
        case 1: return launch_back_t<1>(es, X, ldx, nv);
        case 2: return launch_back_t<2>(es, X, ldx, nv);
        case 3: return launch_back_t<3>(es, X, ldx, nv);
        case 4: return launch_back_t<4>(es, X, ldx, nv);
        case 5: return launch_back_t<5>(es, X, ldx, nv);
        case 6: return launch_back_t<6>(es, X, ldx, nv);
        case 7: return launch_back_t<7>(es, X, ldx, nv);
        default: return launch_back_t<8>(es, X, ldx, nv);
    }
}

// Eigenvectors of global indices idx[0..nv) (ascending eigenvalue order) into the complex n x nv
// block X (ldx): inverse iteration on T, then X = Q Z.
int eigvectors(lm_eigsys* es, const std::vector<int64_t>& idx, double2* X, int64_t ldx) {
    lm_ctx* ctx = es->ctx;
    const int64_t n = es->n, nv = (int64_t)idx.size();
    if (nv == 0) return LM_OK;
    // clusters: every requested eigenvalue with its cluster-mates (same block, consecutive
    // within the block, gaps below kClusterRel |T|), each cluster once
    const double ctol = kClusterRel * es->tnorm;
    // per block: global indices in block order
    std::vector<std::vector<int64_t>> in_blk(es->blk_s.size());
    for (int64_t i = 0; i < n; ++i) in_blk[(size_t)es->w_blk[(size_t)i]].push_back(i);
    for (auto& v : in_blk)
        std::sort(v.begin(), v.end(), [&](int64_t a, int64_t b) { return es->w_k[(size_t)a] < es->w_k[(size_t)b]; });
    std::vector<int64_t> pos_in_blk((size_t)n);
    for (auto& v : in_blk)
        for (size_t u = 0; u < v.size(); ++u) pos_in_blk[(size_t)v[u]] = (int64_t)u;
    std::vector<int64_t> cl_first, cl_count, mem_s, mem_len, mem_seed, col_mem((size_t)nv, -1);
    std::vector<double> mem_lam;
    std::vector<char> seen((size_t)n, 0);
    std::vector<int64_t> mem_of((size_t)n, -1);
    for (int64_t c = 0; c < nv; ++c) {
        const int64_t g = idx[(size_t)c];
        if (!seen[(size_t)g]) {
            const auto& bl = in_blk[(size_t)es->w_blk[(size_t)g]];
            int64_t lo = pos_in_blk[(size_t)g], hi = lo;
            while (lo > 0 && es->w[(size_t)bl[(size_t)lo]] - es->w[(size_t)bl[(size_t)lo - 1]] < ctol) --lo;
            while (hi + 1 < (int64_t)bl.size() && es->w[(size_t)bl[(size_t)hi + 1]] - es->w[(size_t)bl[(size_t)hi]] < ctol) ++hi;
            cl_first.push_back((int64_t)mem_lam.size());
            cl_count.push_back(hi - lo + 1);
            const int64_t b = es->w_blk[(size_t)g];
            for (int64_t u = lo; u <= hi; ++u) {
                const int64_t gg = bl[(size_t)u];
                seen[(size_t)gg] = 1;
                mem_of[(size_t)gg] = (int64_t)mem_lam.size();
                mem_lam.push_back(es->w[(size_t)gg]);
                mem_s.push_back(es->blk_s[(size_t)b]);
                mem_len.push_back(es->blk_len[(size_t)b]);
                mem_seed.push_back(gg);
            }
        }
        col_mem[(size_t)c] = mem_of[(size_t)g];
    }
    const int64_t nmem = (int64_t)mem_lam.size(), ncl = (int64_t)cl_first.size();
    int64_t lmax = 1;
    for (int64_t l : mem_len) lmax = std::max(lmax, l);
    DevFree tmp(ctx);
    int64_t *d_clf = nullptr, *d_clc = nullptr, *d_ms = nullptr, *d_ml = nullptr, *d_seed = nullptr, *d_col = nullptr;
    double *d_lam = nullptr, *d_vec = nullptr, *d_scr = nullptr;
    int rc = upload_vec(ctx, &d_clf, cl_first, "inverse iteration");
    if (rc == LM_OK) rc = upload_vec(ctx, &d_clc, cl_count, "inverse iteration");
    if (rc == LM_OK) rc = upload_vec(ctx, &d_ms, mem_s, "inverse iteration");
    if (rc == LM_OK) rc = upload_vec(ctx, &d_ml, mem_len, "inverse iteration");
    if (rc == LM_OK) rc = upload_vec(ctx, &d_seed, mem_seed, "inverse iteration");
    if (rc == LM_OK) rc = upload_vec(ctx, &d_col, col_mem, "inverse iteration");
    if (rc == LM_OK) rc = upload_vec(ctx, &d_lam, mem_lam, "inverse iteration");
    if (rc == LM_OK) rc = dalloc_t(ctx, &d_vec, (size_t)nmem * (size_t)lmax, "tridiagonal eigenvectors");
    if (rc == LM_OK) rc = dalloc_t(ctx, &d_scr, (size_t)ncl * (size_t)lmax * 4 + ((size_t)ncl * (size_t)lmax + 7) / 8,
                                   "inverse iteration scratch");
    tmp.keep(d_clf); tmp.keep(d_clc); tmp.keep(d_ms); tmp.keep(d_ml); tmp.keep(d_seed); tmp.keep(d_col);
    tmp.keep(d_lam); tmp.keep(d_vec); tmp.keep(d_scr);
    if (rc != LM_OK) return rc;
    const double pert = DBL_EPSILON * std::max(es->tnorm, DBL_MIN);
    stein_kernel<<<(unsigned)((ncl + 31) / 32), 32, 0, ctx->stream>>>(es->d_d, es->d_e, ncl, nmem, d_clf, d_clc, d_ms,
                                                                     d_ml, d_lam, d_seed, d_vec, d_scr, lmax, pert);
    scatter_vectors_kernel<<<dim3((unsigned)((n + 255) / 256), (unsigned)nv), 256, 0, ctx->stream>>>(
        n, nv, d_col, d_ms, d_ml, d_vec, nmem, X, ldx);
    ctx->launches += 2;
    CUDA_TRY(ctx, cudaGetLastError(), "eigensolver: inverse iteration");
    const int bc = back_resident_cols(ctx, n, nv);
    if (bc) CUDA_TRY(ctx, launch_back(es, X, ldx, nv, bc), "eigensolver: back-transformation");
    for (int64_t j = bc ? -1 : n - 2; j >= 0; --j) {
        apply_reflector_kernel<<<(unsigned)nv, 256, 0, ctx->stream>>>(es->d_A, n, n, j, es->d_tau, X, ldx, nv);
        ctx->launches++;
        if ((j & 255) == 0) CUDA_TRY(ctx, cudaGetLastError(), "eigensolver: back-transformation");
    }
    CUDA_TRY(ctx, cudaGetLastError(), "eigensolver: back-transformation");
    // the temporaries are freed on return: wait for the kernels that read them
    CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream), "eigensolver: synchronize");
    return LM_OK;
}

int eigsys_from_dense(lm_ctx* ctx, int64_t n, lm_eigsys** out) {
    lm_eigsys* es = *out;
    int rc = reduce_and_solve(es);
    if (rc != LM_OK) {
        free_eigsys(es);
        delete es;
        *out = nullptr;
    }
    (void)ctx;
    (void)n;
    return rc;
}

}  // namespace

extern "C" {

int lm_newton_reciprocals(lm_ctx* ctx, int64_t n, const double* x, double* rsqrt, double* recip) {
    if (!ctx) return LM_ERR_ARG;
    CHECK_ARG(ctx, n >= 1 && x && rsqrt && recip, "lm_newton_reciprocals: bad argument");
    cudaSetDevice(ctx->device);
    DevFree tmp(ctx);
    double* d = nullptr;
    const int rc = dalloc_t(ctx, &d, 3 * (size_t)n, "arguments");
    tmp.keep(d);
    if (rc != LM_OK) return rc;
    const size_t bytes = sizeof(double) * (size_t)n;
    CUDA_TRY(ctx, cudaMemcpyAsync(d, x, bytes, cudaMemcpyHostToDevice, ctx->stream), "upload");
    newton_kernel<<<(unsigned)((n + 255) / 256), 256, 0, ctx->stream>>>(d, n, d + n, d + 2 * n);
    CUDA_TRY(ctx, cudaGetLastError(), "lm_newton_reciprocals");
    CUDA_TRY(ctx, cudaMemcpyAsync(rsqrt, d + n, bytes, cudaMemcpyDeviceToHost, ctx->stream), "download");
    CUDA_TRY(ctx, cudaMemcpyAsync(recip, d + 2 * n, bytes, cudaMemcpyDeviceToHost, ctx->stream), "download");
    CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream), "sync");
    return LM_OK;
}

int lm_eigsys_create(lm_ham* h, lm_eigsys** out) {
    if (!h || !out) return LM_ERR_ARG;
    lm_ctx* ctx = h->ctx;
    *out = nullptr;
    if (!h->assembled) return set_err(ctx, LM_ERR_STATE, "lm_eigsys_create: Hamiltonian not assembled");
    cudaSetDevice(ctx->device);
    const Geom& g = h->lat->g;
    lm_eigsys* es = new lm_eigsys();
    es->ctx = ctx;
    es->n = g.N;
    int rc = dalloc_t(ctx, &es->d_A, (size_t)g.N * (size_t)g.N, "dense Hamiltonian");
    if (rc != LM_OK) {
        delete es;
        return rc;
    }
    rc = check_cuda(ctx, cudaMemsetAsync(es->d_A, 0, sizeof(double2) * (size_t)g.N * (size_t)g.N, ctx->stream),
                    "lm_eigsys_create: clear");
    if (rc == LM_OK) {
        dense_square_kernel<<<(unsigned)((g.N + 255) / 256), 256, 0, ctx->stream>>>(g, h->d_hop, h->d_onsite, es->d_A,
                                                                                   g.N);
        ctx->launches++;
        rc = check_cuda(ctx, cudaGetLastError(), "lm_eigsys_create: dense assembly");
    }
    if (rc != LM_OK) {
        free_eigsys(es);
        delete es;
        return rc;
    }
    *out = es;
    return eigsys_from_dense(ctx, g.N, out);
}

int lm_eigsys_create_ell(lm_ell* h, lm_eigsys** out) {
    if (!h || !out) return LM_ERR_ARG;
    lm_ctx* ctx = h->ctx;
    *out = nullptr;
    cudaSetDevice(ctx->device);
    lm_eigsys* es = new lm_eigsys();
    es->ctx = ctx;
    es->n = h->n;
    int rc = dalloc_t(ctx, &es->d_A, (size_t)h->n * (size_t)h->n, "dense Hamiltonian");
    if (rc != LM_OK) {
        delete es;
        return rc;
    }
    rc = check_cuda(ctx, cudaMemsetAsync(es->d_A, 0, sizeof(double2) * (size_t)h->n * (size_t)h->n, ctx->stream),
                    "lm_eigsys_create_ell: clear");
    if (rc == LM_OK) {
        dense_ell_kernel<<<(unsigned)((h->n + 255) / 256), 256, 0, ctx->stream>>>(h->n, h->w, h->d_cols, h->d_vals,
                                                                                 h->d_diag, es->d_A, h->n);
        ctx->launches++;
        rc = check_cuda(ctx, cudaGetLastError(), "lm_eigsys_create_ell: dense assembly");
    }
    if (rc != LM_OK) {
        free_eigsys(es);
        delete es;
        return rc;
    }
    *out = es;
    return eigsys_from_dense(ctx, h->n, out);
}

int lm_eigsys_destroy(lm_eigsys* e) {
    if (!e) return LM_OK;
    cudaSetDevice(e->ctx->device);
    cudaStreamSynchronize(e->ctx->stream);
    free_eigsys(e);
    delete e;
    return LM_OK;
}

int lm_eigsys_size(const lm_eigsys* e, int64_t* n) {
    if (!e || !n) return LM_ERR_ARG;
    *n = e->n;
    return LM_OK;
}

int lm_eigsys_values(const lm_eigsys* e, double* out) {
    if (!e || !out) return LM_ERR_ARG;
    std::copy(e->w.begin(), e->w.end(), out);
    return LM_OK;
}

int lm_eigsys_vectors(lm_eigsys* e, int64_t first, lm_state* out) {
    if (!e) return LM_ERR_ARG;
    lm_ctx* ctx = e->ctx;
    int rc = check_lm_state_dense(ctx, out, e->n, LM_KETS, "lm_eigsys_vectors");
    if (rc != LM_OK) return rc;
    CHECK_ARG(ctx, first >= 0 && first + out->m <= e->n, "lm_eigsys_vectors: index range outside the spectrum");
    cudaSetDevice(ctx->device);
    DevFree tmp(ctx);
    double2* X = nullptr;
    const bool direct = out->precision == LM_C64;
    for (int64_t c0 = 0; c0 < out->m; c0 += kChunk) {
        const int64_t nv = std::min<int64_t>(kChunk, out->m - c0);
        std::vector<int64_t> idx((size_t)nv);
        for (int64_t k = 0; k < nv; ++k) idx[(size_t)k] = first + c0 + k;
        if (direct) {
            rc = eigvectors(e, idx, (double2*)out->d_data + c0 * out->ld, out->ld);
        } else {
            if (!X) {
                rc = dalloc_t(ctx, &X, (size_t)e->n * (size_t)kChunk, "eigenvector chunk");
                if (rc != LM_OK) return rc;
                tmp.keep(X);
            }
            rc = eigvectors(e, idx, X, e->n);
            if (rc == LM_OK) {
                to_c32_kernel<<<dim3((unsigned)((e->n + 255) / 256), grid_y(nv)), 256, 0, ctx->stream>>>(
                    X, e->n, (float2*)out->d_data + c0 * out->ld, out->ld, e->n, nv);
                ctx->launches++;
                rc = check_cuda(ctx, cudaGetLastError(), "lm_eigsys_vectors: conversion");
            }
        }
        if (rc != LM_OK) return rc;
    }
    if (X) CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream), "lm_eigsys_vectors: synchronize");
    return LM_OK;
}

int lm_eigsys_projector(lm_eigsys* e, const double* weights, lm_state* out) {
    if (!e) return LM_ERR_ARG;
    lm_ctx* ctx = e->ctx;
    int rc = check_lm_state_dense(ctx, out, e->n, LM_DENSITY, "lm_eigsys_projector");
    if (rc != LM_OK) return rc;
    CHECK_ARG(ctx, weights != nullptr, "lm_eigsys_projector: null weights");
    for (int64_t k = 0; k < e->n; ++k)
        CHECK_ARG(ctx, std::isfinite(weights[k]), "lm_eigsys_projector: non-finite weight");
    cudaSetDevice(ctx->device);
    const int64_t n = e->n;
    DevFree tmp(ctx);
    double2* P = nullptr;
    int64_t ldp = out->ld;
    if (out->precision == LM_C64) {
        P = (double2*)out->d_data;
    } else {
        rc = dalloc_t(ctx, &P, (size_t)n * (size_t)n, "projector");
        if (rc != LM_OK) return rc;
        tmp.keep(P);
        ldp = n;
    }
    CUDA_TRY(ctx, cudaMemset2DAsync(P, sizeof(double2) * ldp, 0, sizeof(double2) * n, n, ctx->stream),
             "lm_eigsys_projector: clear");
    std::vector<int64_t> nz;
    for (int64_t k = 0; k < n; ++k)
        if (weights[k] != 0.0) nz.push_back(k);
    double2* X = nullptr;
    double* d_w = nullptr;
    if (!nz.empty()) {
        const int64_t cw = std::min<int64_t>(kChunk, (int64_t)nz.size());
        rc = dalloc_t(ctx, &X, (size_t)n * (size_t)cw, "eigenvector chunk");
        if (rc == LM_OK) rc = dalloc_t(ctx, &d_w, (size_t)cw, "weights");
        if (rc != LM_OK) {
            dev_free(ctx, X);
            dev_free(ctx, d_w);
            return rc;
        }
        tmp.keep(X);
        tmp.keep(d_w);
    }
    const int nt64 = (int)((n + 63) / 64);
    const int ts = (int64_t)nt64 * (nt64 + 1) / 2 >= 4 * ctx->sm_count ? 64 : 32;
    const int nt = (int)((n + ts - 1) / ts);
    const int64_t ntiles = (int64_t)nt * (nt + 1) / 2;
    std::vector<double> wc;
    for (size_t c0 = 0; c0 < nz.size(); c0 += kChunk) {
        const size_t nv = std::min<size_t>(kChunk, nz.size() - c0);
        std::vector<int64_t> idx(nz.begin() + c0, nz.begin() + c0 + nv);
        wc.assign(nv, 0.0);
        for (size_t k = 0; k < nv; ++k) wc[k] = weights[idx[k]];
        rc = eigvectors(e, idx, X, n);
        if (rc != LM_OK) return rc;
        CUDA_TRY(ctx, cudaMemcpyAsync(d_w, wc.data(), sizeof(double) * nv, cudaMemcpyHostToDevice, ctx->stream),
                 "lm_eigsys_projector: weights");
        if (ts == 64)
            projector_tiles_kernel<64><<<(unsigned)ntiles, 256, 0, ctx->stream>>>(X, n, n, (int64_t)nv, d_w, P, ldp);
        else
            projector_tiles_kernel<32><<<(unsigned)ntiles, 256, 0, ctx->stream>>>(X, n, n, (int64_t)nv, d_w, P, ldp);
        ctx->launches++;
        CUDA_TRY(ctx, cudaGetLastError(), "lm_eigsys_projector: accumulation");
        CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream), "lm_eigsys_projector: synchronize");  // wc reuse
    }
    hermitian_fill_kernel<<<dim3((unsigned)((n + 255) / 256), grid_y(n)), 256, 0, ctx->stream>>>(P, ldp, n);
    ctx->launches++;
    CUDA_TRY(ctx, cudaGetLastError(), "lm_eigsys_projector: fill");
    if (out->precision != LM_C64) {
        to_c32_kernel<<<dim3((unsigned)((n + 255) / 256), grid_y(n)), 256, 0, ctx->stream>>>(P, n, (float2*)out->d_data,
                                                                                             out->ld, n, n);
        ctx->launches++;
        CUDA_TRY(ctx, cudaGetLastError(), "lm_eigsys_projector: conversion");
    }
    CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream), "lm_eigsys_projector: synchronize");
    return LM_OK;
}

}  // extern "C"
