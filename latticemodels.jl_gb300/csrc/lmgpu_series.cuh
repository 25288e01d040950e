// Chebyshev series of a square-lattice Hamiltonian with every ket on chip (lmgpu_series.cu).
#pragma once
#include "lmgpu_internal.cuh"

namespace lmgpu {

constexpr int kSeriesMaxK = 63;  // orders of a propagator (cf[] below); a real series has no limit

// One launch: out = sum_k c_k T_k(H~) in over the columns of a block.
struct SeriesArgs {
    int Lx = 0, Ly = 0, per_x = 0, per_y = 0;
    int nseg = 0, cols = 0;            // thread layout (series_plan)
    int K = 0;                         // highest order
    int64_t M = 0, ld_in = 0, ld_out = 0;
    const double2* in = nullptr;       // null: the identity
    double2* out = nullptr;            // ComplexF64 output, or
    float2* out32 = nullptr;           // ComplexF32 output
    int transpose = 0;                 // store the conjugate transpose
    const double2* gauge = nullptr;    // g of every site: H = G H' G^dagger, x-hops of H' real; null: g = 1
    const void* hy = nullptr;          // 2 H'[s, s + y] / a
    const void* diag = nullptr;        // 2 (V - b) / a
    double alpha = 0.0;                // 2 H'[s, s + x] / a
    double2 phase = {1.0, 0.0};        // factor of the input (propagator)
    const float2* cd = nullptr;        // K + 1 double-float coefficients (real series)
    double cf[kSeriesMaxK + 1] = {};   // c_k = cf[k], or -i cf[k] for odd k (propagator)
};

// Whether the form takes this lattice, and which: kets per CTA (0: not), thread layout and shared
// memory.  x_real: every x-hop is t1 already; otherwise the gauge needs an open x axis.
struct SeriesPlan {
    int kt = 0, nseg = 0, cols = 0;
    size_t smem = 0;
};
SeriesPlan series_plan(lm_ctx* ctx, const Geom& g, bool x_real, int64_t M, bool df);

// Gauge and stencil tables of H (hops of modulus t1 and on-site term; 2/a scales them): gauge may be null when x_real.  Double
// tables (hy, diag) or double-float ones (hyd, diagd); null pointers are skipped.
cudaError_t launch_gauge_tables(lm_ctx* ctx, const Geom& g, const double2* hop, const double* onsite, double t1, double a,
                                double b, bool x_real, double2* gauge, double2* hy, double* diag, float4* hyd,
                                float2* diagd);
// FP64 propagator (cf) / double-float real series (cd).
cudaError_t launch_series_f64(lm_ctx* ctx, const SeriesPlan& p, SeriesArgs a);
cudaError_t launch_series_df(lm_ctx* ctx, const SeriesPlan& p, SeriesArgs a);

}  // namespace lmgpu
