// The tangent of one static step (luna-cpp's step_tangent, src/hydro/finite_volume.hpp:2023-2062): dQ^n+1 = J dQ^n at
// fixed dt, for the FP64 policy, order 1, the per-face loop; the step itself runs after it with the production kernels,
// so Q^n+1 is step()'s. The linearisation point is the adjoint's (k_sweep_fit: its gradients and clip pattern), so the
// tangent and the adjoint are transposes of one map (the dot test). Passes, over the step's own rows as the adjoint's:
//   k_tangent_prims   dW = J dU of primitive() per cell (primitive_tangent, euler.hpp:131-142);
//   k_tangent_sweep   dg per cell: dg0 = sum_k c_k (dW_k - dW_i) over the tile's staged dW, then the limited gradient's
//                     tangent at its clip pattern (limited_gradient_tangent, finite_volume.hpp:811-833: a clipped
//                     variable is g0 (bound - W_i) / (g0 . o_last)); merged rows dW, dg;
//   k_tangent_fluxes  per face: both face states' tangents (side_tangent: the half step and g . r, a fallen-back side
//                     carries dW) and the Riemann solve's, by forward-mode dual numbers through the same HLLC/HLL code
//                     as the step (each branch the forward took), times |A| (TangentFluxes, :1971-2004);
//   k_tangent_update  dQ_i -= dt sum_k sign_k dF_k in list order (TangentUpdate, :2006-2022).
#pragma once

#include "adjoint.cuh"

namespace luna {
namespace fwd {

// A forward-mode dual number: a value and its derivative along one direction. The free functions below are found by
// argument-dependent lookup from the templated device physics (T = Dual), so the tangent differentiates the very
// expressions the step evaluates; comparisons look at values only (the forward's branch).
struct Dual {
    double v, d;
    __device__ __forceinline__ Dual() : v(0), d(0) {}
    __device__ __forceinline__ Dual(double x) : v(x), d(0) {}  // NOLINT: constants enter the physics as T(c)
    __device__ __forceinline__ Dual(double x, double dx) : v(x), d(dx) {}
    __device__ __forceinline__ Dual& operator+=(const Dual& o) {
        v += o.v;
        d += o.d;
        return *this;
    }
    __device__ __forceinline__ Dual& operator-=(const Dual& o) {
        v -= o.v;
        d -= o.d;
        return *this;
    }
    __device__ __forceinline__ Dual& operator*=(const Dual& o) {
        d = d * o.v + v * o.d;
        v *= o.v;
        return *this;
    }
};
__device__ __forceinline__ Dual operator+(const Dual& a, const Dual& b) { return {a.v + b.v, a.d + b.d}; }
__device__ __forceinline__ Dual operator-(const Dual& a, const Dual& b) { return {a.v - b.v, a.d - b.d}; }
__device__ __forceinline__ Dual operator-(const Dual& a) { return {-a.v, -a.d}; }
__device__ __forceinline__ Dual operator*(const Dual& a, const Dual& b) { return {a.v * b.v, a.d * b.v + a.v * b.d}; }
__device__ __forceinline__ Dual operator/(const Dual& a, const Dual& b) {
    const double q = a.v / b.v;
    return {q, (a.d - q * b.d) / b.v};
}
__device__ __forceinline__ bool operator<(const Dual& a, const Dual& b) { return a.v < b.v; }
__device__ __forceinline__ bool operator>(const Dual& a, const Dual& b) { return a.v > b.v; }
__device__ __forceinline__ bool operator<=(const Dual& a, const Dual& b) { return a.v <= b.v; }
__device__ __forceinline__ bool operator>=(const Dual& a, const Dual& b) { return a.v >= b.v; }
__device__ __forceinline__ Dual sqrt(const Dual& a) {
    const double r = ::sqrt(a.v);
    return {r, r > 0 ? a.d / (2 * r) : 0.0};
}
__device__ __forceinline__ Dual fabs(const Dual& a) { return a.v < 0 ? -a : a; }
__device__ __forceinline__ Dual fmin(const Dual& a, const Dual& b) { return b.v < a.v ? b : a; }
__device__ __forceinline__ Dual fmax(const Dual& a, const Dual& b) { return b.v > a.v ? b : a; }

// HLL (euler.hpp:444-461) for any arithmetic type T (the step's hll_flux is double only).
template <int D, class T>
__device__ __forceinline__ void hll_flux_t(const T* L, const T* R, const T* n, const T* w, T gamma, T inverse_gm1, T* F,
                                           bool moving_frame = false) {
    constexpr int P = D + 1;
    Side<D, T> l, r;
    T rel[D];
#pragma unroll
    for (int k = 0; k < D; ++k) rel[k] = L[1 + k] - w[k];
    side_with<D, T>(L, n, w, inverse_gm1, dot<D>(rel, n), l);
    {
        const T c2 = gamma * L[P] / L[0];
        l.c = c2 > T(0) ? sqrt(c2) : T(0);
    }
#pragma unroll
    for (int k = 0; k < D; ++k) rel[k] = R[1 + k] - w[k];
    side_with<D, T>(R, n, w, inverse_gm1, dot<D>(rel, n), r);
    {
        const T c2 = gamma * R[P] / R[0];
        r.c = c2 > T(0) ? sqrt(c2) : T(0);
    }
    const T SL = fmin(l.vn - l.c, r.vn - r.c);
    const T SR = fmax(l.vn + l.c, r.vn + r.c);
    if (SL >= T(0)) {
#pragma unroll
        for (int v = 0; v < D + 2; ++v) F[v] = l.F[v];
    } else if (SR <= T(0)) {
#pragma unroll
        for (int v = 0; v < D + 2; ++v) F[v] = r.F[v];
    } else {
        const T inv_dS = T(1) / (SR - SL);
#pragma unroll
        for (int v = 0; v < D + 2; ++v) F[v] = (SR * l.F[v] - SL * r.F[v] + SL * SR * (r.U[v] - l.U[v])) * inv_dS;
    }
    if (moving_frame) to_lab<D, T>(F, w);
}

}  // namespace fwd

// primitive_tangent (euler.hpp:131-142): dW = J dU; a floored density or energy has derivative 0 in what it replaced.
template <int D>
__device__ __forceinline__ void primitive_tangent(const double* U, const double* dU, const GasDev& gas, double* dW) {
    constexpr int P = D + 1;
    const double rho = fmax(U[0], gas.smallr), inv_rho = 1.0 / rho;
    double v[D];
#pragma unroll
    for (int k = 0; k < D; ++k) v[k] = U[1 + k] * inv_rho;
    const double smalle = gas.smallc * gas.smallc / gas.gamma / (gas.gamma - 1.0);
    const int floors = (U[0] >= gas.smallr ? 0 : 1) | (U[P] - 0.5 * rho * dot<D>(v, v) >= smalle * rho ? 0 : 2);
    const double drho = floors & 1 ? 0.0 : dU[0];
    double dv[D];
#pragma unroll
    for (int k = 0; k < D; ++k) dv[k] = (dU[1 + k] - v[k] * drho) * inv_rho;
    const double dkinetic = 0.5 * drho * dot<D>(v, v) + rho * dot<D>(v, dv);
    const double de = floors & 2 ? smalle * drho : dU[P] - dkinetic;
    dW[0] = drho;
#pragma unroll
    for (int k = 0; k < D; ++k) dW[1 + k] = dv[k];
    dW[P] = (gas.gamma - 1.0) * de;
}

// dW rows of bar_stride doubles (what the tiles stage).
template <int D>
__global__ void __launch_bounds__(256) k_tangent_prims(int n, const double* __restrict__ q, const double* __restrict__ dq,
                                                       const double* __restrict__ vol, GasDev gas, double* __restrict__ dprims) {
    constexpr int V = D + 2, B = bar_stride<D>();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double inv = 1.0 / vol[i];
    double U[V], dU[V], dW[B];
#pragma unroll
    for (int v = 0; v < V; ++v) {
        U[v] = q[V * static_cast<int64_t>(i) + v] * inv;
        dU[v] = dq[V * static_cast<int64_t>(i) + v] * inv;
    }
    primitive_tangent<D>(U, dU, gas, dW);
#pragma unroll
    for (int v = V; v < B; ++v) dW[v] = 0;
    store_bar<B>(dprims + B * static_cast<int64_t>(i), dW);
}

// The limited gradient's tangent per cell at the stored fit and clip pattern (k_sweep_fit's rows and clip words), one
// block a tile.
template <int D>
__global__ void __launch_bounds__(kTileCells, adj_min_blocks<D>()) k_tangent_sweep(MeshDev<D> m, GeometryDev<D, double> geo, int tile0,
                                                                                 const double* __restrict__ dprims, const double* __restrict__ wg,
                                                                                 const double* __restrict__ fit, const int32_t* __restrict__ clip,
                                                                                 double* __restrict__ dwg) {
    constexpr int V = D + 2;
    using FL = FitLayout<D>;
    extern __shared__ double2 staged_rows[];
    double* rows = reinterpret_cast<double*>(staged_rows);
    const int tile = tile0 + static_cast<int>(blockIdx.x);
    stage_rows<D>(geo, tile, dprims, bar_stride<D>(), rows);
    const int64_t t = static_cast<int64_t>(tile) * kTileCells + threadIdx.x;
    const int i = geo.order[t];
    if (i < 0) return;
    const int count = m.start[i + 1] - m.start[i];
    const int64_t slot0 = static_cast<int64_t>(geo.slice_base[t >> 5]) * 32 + (t & 31);
    double dWi[V], dg[V * D];
#pragma unroll
    for (int v = 0; v < V; ++v) dWi[v] = rows[kFitStaged * threadIdx.x + v];
#pragma unroll
    for (int c = 0; c < V * D; ++c) dg[c] = 0;
    for (int k = 0; k < count; ++k) {
        const int64_t slot = slot0 + 32 * static_cast<int64_t>(k);
        const double2 c01 = geo.c01[slot];
        double c[D], dWj[kFitStaged];
        c[0] = c01.x;
        c[1] = c01.y;
        if constexpr (D == 3) c[2] = geo.c2[slot];
        load_bar<V>(rows + kFitStaged * static_cast<int>(geo.nbr[slot] & kIndexMask), dWj);
#pragma unroll
        for (int v = 0; v < V; ++v) {
            const double ddW = dWj[v] - dWi[v];
#pragma unroll
            for (int a = 0; a < D; ++a) dg[D * v + a] += c[a] * ddW;
        }
    }
    const double* fr = fit + static_cast<int64_t>(FL::width) * i;
#pragma unroll
    for (int v = 0; v < V; ++v) {
        const int word = clip[V * static_cast<int64_t>(i) + v];
        if (!(word & 1)) continue;
        if (word & 4) {
#pragma unroll
            for (int a = 0; a < D; ++a) dg[D * v + a] = 0.0;
            continue;
        }
        const int64_t slot = slot0 + 32 * static_cast<int64_t>(clip_entry(word));
        double o[D], g0[D];
        const double2 o01 = geo.off01[slot];
        o[0] = o01.x;
        o[1] = o01.y;
        if constexpr (D == 3) o[2] = geo.off2[slot];
#pragma unroll
        for (int a = 0; a < D; ++a) g0[a] = fr[FL::g0 + D * v + a];
        const unsigned int holder = geo.nbr[slot0 + 32 * static_cast<int64_t>(bound_entry(word))] & kIndexMask;
        const double dbound = rows[kFitStaged * static_cast<int>(holder) + v];
        const double den = dot<D>(g0, o);
        const double s = (fr[FL::bound + v] - wg[static_cast<int64_t>(wg_stride<D>()) * i + v]) / den;
        const double ds = (dbound - dWi[v] - s * dot<D>(dg + D * v, o)) / den;
#pragma unroll
        for (int a = 0; a < D; ++a) dg[D * v + a] = dg[D * v + a] * s + g0[a] * ds;
    }
    store_wg<D>(dwg, i, dWi, dg);
}

#ifndef LUNA_TANGENT_MIN_BLOCKS
#define LUNA_TANGENT_MIN_BLOCKS 3
#endif
// side_tangent (finite_volume.hpp:1346-1366): the face state's tangent, by duals through the half step; a side that
// fell back (rho or P of the face state not positive) carries dW.
template <int D>
__device__ __forceinline__ void side_tangent(const double* W, const double* dW, const double* g, const double* dg, const double* r, double dt,
                                             double gamma, bool fallback, double* dWf) {
    constexpr int V = D + 2;
    if (fallback) {
#pragma unroll
        for (int v = 0; v < V; ++v) dWf[v] = dW[v];
        return;
    }
    fwd::Dual Wd[V], gd[V * D], A[V];
#pragma unroll
    for (int v = 0; v < V; ++v) Wd[v] = fwd::Dual(W[v], dW[v]);
#pragma unroll
    for (int c = 0; c < V * D; ++c) gd[c] = fwd::Dual(g[c], dg[c]);
    half_step_rate<D, fwd::Dual>(Wd, gd, fwd::Dual(gamma), A);
#pragma unroll
    for (int v = 0; v < V; ++v) {
        fwd::Dual f = Wd[v] - fwd::Dual(0.5 * dt) * A[v];
#pragma unroll
        for (int a = 0; a < D; ++a) f += gd[D * v + a] * fwd::Dual(r[a]);
        dWf[v] = f.d;
    }
}

template <int D, int Riemann>
__global__ void __launch_bounds__(128, LUNA_TANGENT_MIN_BLOCKS) k_tangent_fluxes(int faces, const FaceRow<double>* __restrict__ face_rows,
                                                                               const double* __restrict__ wg, const double* __restrict__ dwg,
                                                                               double dt, GasDev gas, double* __restrict__ dflux) {
    constexpr int V = D + 2;
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= faces) return;
    FaceRow<double> r;
    load_face_row<double>(face_rows + f, r);
    double dF[V];
#pragma unroll
    for (int v = 0; v < V; ++v) dF[v] = 0;
    if (r.mag != 0) {
        fwd::Dual Ld[V], Rd[V], n[D], w[D], F[V];
        const auto side = [&](int i, const double* off, fwd::Dual* out) {
            double W[V], g[V * D], dW[V], dg[V * D], Wf[V], dWf[V];
            load_wg<D>(wg, i, W, g);
            load_wg<D>(dwg, i, dW, dg);
            const bool fallback = side_value<D>(W, g, off, dt, gas.gamma, Wf);
            side_tangent<D>(W, dW, g, dg, off, dt, gas.gamma, fallback, dWf);
#pragma unroll
            for (int v = 0; v < V; ++v) out[v] = fwd::Dual(Wf[v], dWf[v]);
        };
        side(r.o, r.offo, Ld);
        side(r.j, r.offj, Rd);
#pragma unroll
        for (int a = 0; a < D; ++a) {
            n[a] = fwd::Dual(r.n[a]);
            w[a] = fwd::Dual(0.0);
        }
        if constexpr (Riemann == 1)
            fwd::hll_flux_t<D, fwd::Dual>(Ld, Rd, n, w, fwd::Dual(gas.gamma), fwd::Dual(gas.inverse_gm1), F);
        else
            hllc_flux<D, fwd::Dual>(Ld, Rd, n, w, fwd::Dual(gas.gamma), fwd::Dual(gas.inverse_gm1), F, false);
#pragma unroll
        for (int v = 0; v < V; ++v) dF[v] = F[v].d * r.mag;
    }
#pragma unroll
    for (int v = 0; v < V; ++v) dflux[V * static_cast<int64_t>(f) + v] = dF[v];
}

// Flux rows as k_update reads them (load_row_windowed: the buffer extends 24 B past its last row).
template <int D>
__global__ void __launch_bounds__(256) k_tangent_update(MeshDev<D> m, double* __restrict__ dq, const double* __restrict__ dflux, double dt) {
    constexpr int V = D + 2;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m.n) return;
    double dsum[V];
#pragma unroll
    for (int v = 0; v < V; ++v) dsum[v] = 0;
    const int first = m.start[i], end = m.start[i + 1];
    constexpr int kBatch = 2;
    for (int k0 = first; k0 < end; k0 += kBatch) {
        int32_t e[kBatch];
        double row[kBatch][V];
#pragma unroll
        for (int b = 0; b < kBatch; ++b) e[b] = k0 + b < end ? m.list[k0 + b] : 0;
#pragma unroll
        for (int b = 0; b < kBatch; ++b)
            if (k0 + b < end) load_row_windowed<V>(dflux + V * static_cast<int64_t>(list_face(e[b])), row[b]);
#pragma unroll
        for (int b = 0; b < kBatch; ++b) {
            if (k0 + b >= end) break;
            const double sign = e[b] >= 0 ? 1.0 : -1.0;
#pragma unroll
            for (int v = 0; v < V; ++v) dsum[v] += sign * row[b][v];
        }
    }
#pragma unroll
    for (int v = 0; v < V; ++v) dq[V * static_cast<int64_t>(i) + v] = dq[V * static_cast<int64_t>(i) + v] - dt * dsum[v];
}

}  // namespace luna
