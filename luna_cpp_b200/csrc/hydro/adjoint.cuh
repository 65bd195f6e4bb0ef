// The adjoint of one static step (luna-cpp's step_adjoint, src/hydro/finite_volume.hpp:2201-2231): Qbar^n = J^T Qbar^n+1
// at fixed dt, for the FP64 policy, order 1, the per-face loop. Four passes, no atomics (the same bits every run), over
// the rows that the step itself streams (geometry.cuh: the gradient operator's c_k and the face offsets by tile, the face
// rows, the merged W/g rows):
//   k_sweep_fit      the forward sweep again, keeping what the gradient's adjoint needs (SweepFitHook<false>,
//                    finite_volume.hpp:1763-1926): the unlimited gradient g0 and, per variable, the last clip (its entry
//                    and flags), the bound and the entry that the bound came through;
//   k_faces_adjoint  once per face: the Riemann adjoint -> the bars of both face states (AdjointFaces, :2078-2102);
//   k_cell_adjoint   per cell: face-state adjoints -> W and g bars, the limited gradient's adjoint (AdjointCell,
//                    :2107-2169) -> g0's bar; g0 = sum_k c_k (W_k - W_i) then gives each neighbour c_k . g0bar and the
//                    cell minus their sum: each neighbour's share (with the bound's bar at its entry) takes the place of
//                    the cell's face-state bar in the face's row, which no other cell reads;
//   k_gather_adjoint per cell: its neighbours' shares from its faces' rows, then the primitive adjoint into Qbar
//                    (:2171-2195).
// What the passes spend is gather instructions (an L1 line a lane and load), so every row is read in its widest loads and
// none is read twice. Measured against the passes over the mesh arrays, which solved every fit by Cholesky and gathered
// 20 bars and the geometry for each neighbour: at 72 x 64 x 60 cells one step_adjoint and one step_tangent 2.98 -> 1.96 ms
// (k_sweep_fit 406 -> 195 us, k_gather_adjoint 261 -> 76, k_tangent_fluxes 467 -> 200, k_tangent_sweep 135 -> 84); 8 steps
// of the 512^2 rollout with its backward 5.4 -> 4.2 ms.
#pragma once

#include "geometry.cuh"
#include "kernels.cuh"

namespace luna {

// A cell's fit row: the unlimited gradient (V D doubles), then each variable's bound (V).
template <int D>
struct FitLayout {
    static constexpr int V = D + 2;
    static constexpr int g0 = 0, bound = V * D, width = bound + V;
};
// A variable's clip word: bit 0 clipped, 1 at the upper bound, 2 to zero; the last clip's entry; the entry of the bound
// (a list has at most kBigTileRows entries).
constexpr int kClipEntryBits = 14, kClipEntryMask = (1 << kClipEntryBits) - 1;
static_assert(kBigTileRows <= kClipEntryMask, "a list entry fits its field of the clip word");
__host__ __device__ constexpr int clip_word(int flags, int entry, int bound) { return flags | entry << 3 | bound << (3 + kClipEntryBits); }
__host__ __device__ constexpr int clip_entry(int word) { return (word >> 3) & kClipEntryMask; }
__host__ __device__ constexpr int bound_entry(int word) { return (word >> (3 + kClipEntryBits)) & kClipEntryMask; }
// Doubles of one side of a face's bar row, and of a tangent's dW row: whole 16-B units.
template <int D>
constexpr int bar_stride() {
    return D == 3 ? 6 : 4;
}
// Doubles a staged row of the derivative sweeps takes: V, padded to an odd number of 16-B units (see kStagedDoubles).
constexpr int kFitStaged = 6;

// V doubles of a row of bar_stride at p (16-B aligned) in 16-B loads and stores.
template <int V>
__device__ __forceinline__ void load_bar(const double* p, double* out) {
#pragma unroll
    for (int v = 0; v + 1 < V; v += 2) {
        const double2 w = *reinterpret_cast<const double2*>(p + v);
        out[v] = w.x;
        out[v + 1] = w.y;
    }
    if constexpr (V % 2) out[V - 1] = p[V - 1];
}
template <int V>
__device__ __forceinline__ void store_bar(double* p, const double* in) {
#pragma unroll
    for (int v = 0; v + 1 < V; v += 2) *reinterpret_cast<double2*>(p + v) = make_double2(in[v], in[v + 1]);
    if constexpr (V % 2) p[V - 1] = in[V - 1];
}
// A merged row (W then g, wg_stride doubles, 32-B aligned) and its store.
template <int D>
__device__ __forceinline__ void load_wg(const double* rows, int i, double* W, double* g) {
    constexpr int V = D + 2, S = wg_stride<D>();
    double row[S];
    const double* p = rows + static_cast<int64_t>(S) * i;
#pragma unroll
    for (int c = 0; c < S; c += 4) ldg256(p + c, row + c);
#pragma unroll
    for (int v = 0; v < V; ++v) W[v] = row[v];
#pragma unroll
    for (int c = 0; c < V * D; ++c) g[c] = row[V + c];
}
template <int D>
__device__ __forceinline__ void store_wg(double* rows, int i, const double* W, const double* g) {
    constexpr int V = D + 2, S = wg_stride<D>();
    double2* p = reinterpret_cast<double2*>(rows + static_cast<int64_t>(S) * i);
    const auto at = [&](int c) { return c < V ? W[c] : c < V + V * D ? g[c - V] : 0.0; };
#pragma unroll
    for (int c = 0; c < S; c += 2) p[c / 2] = make_double2(at(c), at(c + 1));
}
// The block's tile staged: kFitStaged doubles of each staged cell from its row of `stride` doubles (16-B aligned).
template <int D>
__device__ __forceinline__ void stage_rows(const GeometryDev<D, double>& geo, int tile, const double* __restrict__ from, int stride, double* rows) {
    const int s0 = geo.stage_start[tile], staged = geo.stage_start[tile + 1] - s0;
    for (int r = threadIdx.x; r < staged; r += kTileCells) {
        const double* src = from + static_cast<int64_t>(stride) * geo.stage_cells[s0 + r];
#pragma unroll
        for (int q = 0; q < (D == 3 ? 6 : 4); q += 2) cp_async16(rows + kFitStaged * r + q, src + q);
    }
    cp_async_wait_all();
    __syncthreads();
}

// primitive_adjoint (euler.hpp:143-162).
template <int D>
__device__ __forceinline__ void primitive_adjoint(const double* U, const double* Wbar, const GasDev& gas, double* Ubar) {
    constexpr int P = D + 1;
    const double rho = fmax(U[0], gas.smallr), inv_rho = 1.0 / rho;
    double v[D], vb[D];
#pragma unroll
    for (int k = 0; k < D; ++k) {
        v[k] = U[1 + k] * inv_rho;
        vb[k] = U[1 + k] * (1.0 / rho);
    }
    const double smalle = gas.smallc * gas.smallc / gas.gamma / (gas.gamma - 1.0);
    const int floors = (U[0] >= gas.smallr ? 0 : 1) | (U[P] - 0.5 * rho * dot<D>(vb, vb) >= smalle * rho ? 0 : 2);
    const double ebar = (gas.gamma - 1.0) * Wbar[P];
    double rhobar = Wbar[0], energybar = 0;
    double vbar[D];
#pragma unroll
    for (int k = 0; k < D; ++k) vbar[k] = Wbar[1 + k];
    if (floors & 2) {
        rhobar += smalle * ebar;
    } else {
        energybar = ebar;
        rhobar -= 0.5 * dot<D>(v, v) * ebar;
        const double s = rho * ebar;
#pragma unroll
        for (int k = 0; k < D; ++k) vbar[k] = vbar[k] - v[k] * s;
    }
    rhobar -= dot<D>(v, vbar) * inv_rho;
    Ubar[0] = floors & 1 ? 0.0 : rhobar;
#pragma unroll
    for (int k = 0; k < D; ++k) Ubar[1 + k] = vbar[k] * inv_rho;
    Ubar[P] = energybar;
}

// half_step_adjoint (euler.hpp:241-272): adds J^T halfbar to Wbar and gbar.
template <int D>
__device__ __forceinline__ void half_step_adjoint(const double* W, const double* g, double dt, double gamma, const double* halfbar, double* Wbar,
                                                  double* gbar) {
    constexpr int P = D + 1;
    const double rho = W[0], inv_rho = 1.0 / W[0], rho_c2 = gamma * W[P];
    double Abar[D + 2];
#pragma unroll
    for (int v = 0; v < D + 2; ++v) {
        Wbar[v] += halfbar[v];
        Abar[v] = -0.5 * dt * halfbar[v];
    }
    double inv_rhobar = 0, rho_c2bar = 0;
#pragma unroll
    for (int d = 0; d < D; ++d) {
        const double vn = W[1 + d];
        Wbar[1 + d] += Abar[0] * g[0 * D + d];
        gbar[0 * D + d] += Abar[0] * vn;
        Wbar[0] += Abar[0] * g[(1 + d) * D + d];
        gbar[(1 + d) * D + d] += Abar[0] * rho;
#pragma unroll
        for (int k = 0; k < D; ++k) {
            Wbar[1 + d] += Abar[1 + k] * g[(1 + k) * D + d];
            gbar[(1 + k) * D + d] += Abar[1 + k] * vn;
            if (k == d) {
                inv_rhobar += Abar[1 + k] * g[P * D + d];
                gbar[P * D + d] += Abar[1 + k] * inv_rho;
            }
        }
        rho_c2bar += Abar[P] * g[(1 + d) * D + d];
        gbar[(1 + d) * D + d] += Abar[P] * rho_c2;
        Wbar[1 + d] += Abar[P] * g[P * D + d];
        gbar[P * D + d] += Abar[P] * vn;
    }
    Wbar[0] -= inv_rho * inv_rho * inv_rhobar;
    Wbar[P] += gamma * rho_c2bar;
}

// detail::side_with_adjoint (euler.hpp:375-398); vbar_in may be null (zero). Returns vn's bar.
template <int D>
__device__ __forceinline__ double side_with_adjoint(const double* W, const double* n, double inverse_gm1, const Side<D, double>& s,
                                                    const double* Fbar, const double* Ubar, double Ebar, const double* vbar_in, double* Wbar) {
    constexpr int P = D + 1;
    const double m = W[0] * s.vn;
    double vbar[D];
#pragma unroll
    for (int k = 0; k < D; ++k) vbar[k] = vbar_in ? vbar_in[k] : 0.0;
    Ebar += Fbar[P] * s.vn + Ubar[P];
    double Pbar = Fbar[P] * s.vn, vnbar = Fbar[P] * (s.E + W[P]), mbar = Fbar[0], rhobar = Ubar[0];
#pragma unroll
    for (int k = 0; k < D; ++k) {
        Pbar += Fbar[1 + k] * n[k];
        mbar += Fbar[1 + k] * s.v[k];
        vbar[k] += Fbar[1 + k] * m + Ubar[1 + k] * W[0];
        rhobar += Ubar[1 + k] * s.v[k];
    }
    rhobar += mbar * s.vn;
    vnbar += mbar * W[0];
    Pbar += Ebar * inverse_gm1;
    rhobar += Ebar * (0.5 * dot<D>(s.v, s.v));
    const double e = Ebar * W[0];
#pragma unroll
    for (int k = 0; k < D; ++k) vbar[k] = vbar[k] + s.v[k] * e;
    Wbar[0] += rhobar;
#pragma unroll
    for (int k = 0; k < D; ++k) Wbar[1 + k] += vbar[k];
    Wbar[P] += Pbar;
    return vnbar;
}

// HLLC::flux_adjoint (euler.hpp:738-832) for a static face (w = 0): only the case the forward took is differentiated; a
// guarded divisor has derivative 0.
template <int D>
__device__ void hllc_flux_adjoint(const double* L, const double* R, const double* n, const GasDev& gas, const double* Fbar, double* Lbar,
                                  double* Rbar) {
    constexpr int P = D + 1;
    constexpr double eps = 1e-20;
    const double vnL = dot<D>(L + 1, n), vnR = dot<D>(R + 1, n);
    const double inv_rhoL = 1.0 / L[0], inv_rhoR = 1.0 / R[0];
    const double c2L = gas.gamma * L[P] * inv_rhoL, c2R = gas.gamma * R[P] * inv_rhoR;
    const bool ok = c2L >= 0 && c2R >= 0;
    const double cL = c2L > 0 ? sqrt(c2L) : 0.0, cR = c2R > 0 ? sqrt(c2R) : 0.0;
    const double sl = vnL - cL, sr = vnR - cR, tl = vnL + cL, tr = vnR + cR;
    const double SL = fmin(sl, sr), SR = fmax(tl, tr);
    const double denomL = L[0] * (SL - vnL), denomR = R[0] * (SR - vnR);
    const double den_raw = denomL - denomR;
    const double SM = (R[P] - L[P] + denomL * vnL - denomR * vnR) / nonzero(den_raw);
    const bool left = ok && (SL >= 0 || SM >= 0);
    const bool star = ok && SL < 0 && (SM >= 0 || SR > 0);
    const bool sl_from_left = !(sr < sl), sr_from_left = !(tr > tl);
    double W[D + 2];
#pragma unroll
    for (int v = 0; v < D + 2; ++v) W[v] = left ? L[v] : R[v];
    const double zero[D] = {};
    Side<D, double> s;
    side_with<D, double>(W, n, zero, gas.inverse_gm1, left ? vnL : vnR, s);
    double Wbar[D + 2];
#pragma unroll
    for (int v = 0; v < D + 2; ++v) Wbar[v] = 0;
    double vnLbar = 0, vnRbar = 0;
    if (!star) {
        const double zeroU[D + 2] = {};
        const double r = side_with_adjoint<D>(W, n, gas.inverse_gm1, s, Fbar, zeroU, 0.0, nullptr, Wbar);
        if (left)
            vnLbar += r;
        else
            vnRbar += r;
    } else {
        const double S = left ? SL : SR, denom = left ? denomL : denomR, inv_side = left ? inv_rhoL : inv_rhoR;
        const bool guard_q = fabs(S - SM) < eps, guard_denom = fabs(denom) < eps, guard_den = fabs(den_raw) < eps;
        const double q = nonzero(S - SM), rho_star = denom / q, inv_denom = 1.0 / nonzero(denom);
        const double a2 = SM - s.vn, a3 = SM + W[P] * inv_denom, E_star = s.E * inv_side + a2 * a3;
        double v_star[D];
#pragma unroll
        for (int k = 0; k < D; ++k) v_star[k] = s.v[k] + n[k] * a2;
        double Sbar = 0, rho_starbar = 0, E_starbar = 0;
        double sUbar[D + 2], v_starbar[D];
#pragma unroll
        for (int v = 0; v < D + 2; ++v) {
            const double U_star = v == 0 ? rho_star : v == P ? rho_star * E_star : rho_star * v_star[v - 1];
            Sbar += Fbar[v] * (U_star - s.U[v]);
            sUbar[v] = -S * Fbar[v];
            const double U_starbar = S * Fbar[v];
            if (v == 0) {
                rho_starbar += U_starbar;
            } else if (v == P) {
                rho_starbar += U_starbar * E_star;
                E_starbar = U_starbar * rho_star;
            } else {
                rho_starbar += U_starbar * v_star[v - 1];
                v_starbar[v - 1] = U_starbar * rho_star;
            }
        }
        const double a2bar = dot<D>(v_starbar, n) + E_starbar * a3, a3bar = E_starbar * a2;
        double SMbar = a3bar + a2bar, vnbar = -a2bar;
        const double inv_denombar = a3bar * W[P];
        const double denombar = (guard_denom ? 0.0 : -inv_denom * inv_denom * inv_denombar) + rho_starbar / q;
        const double qbar = guard_q ? 0.0 : -rho_starbar * rho_star / q;
        Sbar += qbar;
        SMbar -= qbar;
        const double sEbar = E_starbar * inv_side, inv_sidebar = E_starbar * s.E;
        vnbar += side_with_adjoint<D>(W, n, gas.inverse_gm1, s, Fbar, sUbar, sEbar, v_starbar, Wbar);
        Wbar[P] += a3bar * inv_denom;
        const double den = nonzero(den_raw), numbar = SMbar / den, denbar = guard_den ? 0.0 : -SMbar * SM / den;
        double denomLbar = denbar + numbar * vnL, denomRbar = -denbar - numbar * vnR;
        if (left)
            denomLbar += denombar;
        else
            denomRbar += denombar;
        vnLbar += numbar * denomL;
        vnRbar -= numbar * denomR;
        Rbar[P] += numbar;
        Lbar[P] -= numbar;
        if (left)
            vnLbar += vnbar;
        else
            vnRbar += vnbar;
        double invLbar = left ? inv_sidebar : 0.0, invRbar = left ? 0.0 : inv_sidebar;
        double SLbar = denomLbar * L[0], SRbar = denomRbar * R[0];
        if (left)
            SLbar += Sbar;
        else
            SRbar += Sbar;
        Lbar[0] += denomLbar * (SL - vnL);
        vnLbar -= denomLbar * L[0];
        Rbar[0] += denomRbar * (SR - vnR);
        vnRbar -= denomRbar * R[0];
        double cLbar = 0, cRbar = 0;
        if (sl_from_left) {
            vnLbar += SLbar;
            cLbar -= SLbar;
        } else {
            vnRbar += SLbar;
            cRbar -= SLbar;
        }
        if (sr_from_left) {
            vnLbar += SRbar;
            cLbar += SRbar;
        } else {
            vnRbar += SRbar;
            cRbar += SRbar;
        }
        if (c2L > 0) {
            const double c2bar = cLbar / (2 * cL);
            Lbar[P] += c2bar * gas.gamma * inv_rhoL;
            invLbar += c2bar * gas.gamma * L[P];
        }
        if (c2R > 0) {
            const double c2bar = cRbar / (2 * cR);
            Rbar[P] += c2bar * gas.gamma * inv_rhoR;
            invRbar += c2bar * gas.gamma * R[P];
        }
        Lbar[0] -= inv_rhoL * inv_rhoL * invLbar;
        Rbar[0] -= inv_rhoR * inv_rhoR * invRbar;
    }
#pragma unroll
    for (int v = 0; v < D + 2; ++v) {
        Lbar[v] += left ? Wbar[v] : 0.0;
        Rbar[v] += left ? 0.0 : Wbar[v];
    }
#pragma unroll
    for (int k = 0; k < D; ++k) {
        Lbar[1 + k] += vnLbar * n[k];
        Rbar[1 + k] += vnRbar * n[k];
    }
}

// HLL::flux_adjoint (euler.hpp:509-540) for a static face, with detail::side_adjoint (:402-413).
template <int D>
__device__ void hll_flux_adjoint(const double* L, const double* R, const double* n, const GasDev& gas, const double* Fbar, double* Lbar,
                                 double* Rbar) {
    constexpr int P = D + 1;
    const double zero[D] = {};
    Side<D, double> l, r;
    side_with<D, double>(L, n, zero, gas.inverse_gm1, dot<D>(L + 1, n), l);
    side_with<D, double>(R, n, zero, gas.inverse_gm1, dot<D>(R + 1, n), r);
    const double c2l = gas.gamma * L[P] / L[0], c2r = gas.gamma * R[P] / R[0];
    l.c = c2l > 0 ? sqrt(c2l) : 0.0;
    r.c = c2r > 0 ? sqrt(c2r) : 0.0;
    const double a = l.vn - l.c, b = r.vn - r.c, A = l.vn + l.c, B = r.vn + r.c;
    const double SLm = fmin(a, b), SRm = fmax(A, B);
    const int wave = SLm >= 0 ? 1 : SRm <= 0 ? 2 : 0;
    const bool sl_from_left = !(b < a), sr_from_left = !(B > A);
    const double SL = sl_from_left ? l.vn - l.c : r.vn - r.c, SR = sr_from_left ? l.vn + l.c : r.vn + r.c;
    double lF[D + 2], rF[D + 2], lU[D + 2], rU[D + 2];
#pragma unroll
    for (int v = 0; v < D + 2; ++v) lF[v] = rF[v] = lU[v] = rU[v] = 0;
    double SLbar = 0, SRbar = 0;
    if (wave == 1) {
#pragma unroll
        for (int v = 0; v < D + 2; ++v) lF[v] = Fbar[v];
    } else if (wave == 2) {
#pragma unroll
        for (int v = 0; v < D + 2; ++v) rF[v] = Fbar[v];
    } else {
        const double inv_dS = 1.0 / (SR - SL);
#pragma unroll
        for (int v = 0; v < D + 2; ++v) {
            const double dU = r.U[v] - l.U[v], F = (SR * l.F[v] - SL * r.F[v] + SL * SR * dU) * inv_dS;
            const double N = Fbar[v] * inv_dS;
            SRbar += -Fbar[v] * F * inv_dS + N * (l.F[v] + SL * dU);
            SLbar += Fbar[v] * F * inv_dS + N * (-r.F[v] + SR * dU);
            lF[v] = SR * N;
            rF[v] = -SL * N;
            rU[v] = SL * SR * N;
            lU[v] = -SL * SR * N;
        }
    }
    double lvn = 0, lc = 0, rvn = 0, rc = 0;
    if (sl_from_left) {
        lvn += SLbar;
        lc -= SLbar;
    } else {
        rvn += SLbar;
        rc -= SLbar;
    }
    if (sr_from_left) {
        lvn += SRbar;
        lc += SRbar;
    } else {
        rvn += SRbar;
        rc += SRbar;
    }
    // detail::side_adjoint for both sides
    lvn += side_with_adjoint<D>(L, n, gas.inverse_gm1, l, lF, lU, 0.0, nullptr, Lbar);
    rvn += side_with_adjoint<D>(R, n, gas.inverse_gm1, r, rF, rU, 0.0, nullptr, Rbar);
#pragma unroll
    for (int k = 0; k < D; ++k) {
        Lbar[1 + k] += lvn * n[k];
        Rbar[1 + k] += rvn * n[k];
    }
    if (c2l > 0) {
        const double c2bar = lc / (2 * l.c);
        Lbar[P] += c2bar * gas.gamma / L[0];
        Lbar[0] -= c2bar * c2l / L[0];
    }
    if (c2r > 0) {
        const double c2bar = rc / (2 * r.c);
        Rbar[P] += c2bar * gas.gamma / R[0];
        Rbar[0] -= c2bar * c2r / R[0];
    }
}

// FaceFlux::side_value (finite_volume.hpp:1342-1347): the double face state and whether it fell back to W.
template <int D>
__device__ __forceinline__ bool side_value(const double* W, const double* g, const double* r, double dt, double gamma, double* Wf) {
    constexpr int V = D + 2;
    double A[V];
    half_step_rate<D, double>(W, g, gamma, A);
#pragma unroll
    for (int v = 0; v < V; ++v) Wf[v] = W[v] - 0.5 * dt * A[v];
#pragma unroll
    for (int v = 0; v < V; ++v) Wf[v] += dot<D>(g + D * v, r);
    const bool fallback = !(Wf[0] > 0 && Wf[D + 1] > 0);
    if (fallback)
#pragma unroll
        for (int v = 0; v < V; ++v) Wf[v] = W[v];
    return fallback;
}

// Resident blocks an SM the adjoint's register-heavy kernels are cut for; with it k_sweep_fit and k_cell_adjoint request
// two entries' rows together. Measured (one entry at a time, 4 blocks in 2D too -> now): Jacobian products at 72 x 64 x 60
// 1.95 -> 1.90 ms, an eight-step rollout of 512^2 and back 4.08 -> 3.87 ms.
#ifndef LUNA_ADJ_MIN_BLOCKS
#define LUNA_ADJ_MIN_BLOCKS 4  // in 3D
#endif
#ifndef LUNA_ADJ_MIN_BLOCKS_2D
#define LUNA_ADJ_MIN_BLOCKS_2D 5
#endif
template <int D>
constexpr int adj_min_blocks() {
    return D == 3 ? LUNA_ADJ_MIN_BLOCKS : LUNA_ADJ_MIN_BLOCKS_2D;
}

// The sweep again with the fit kept (Sweep<false, true, SweepFitHook<false>>), one block a tile as k_sweep_tiles: the
// merged rows W, g (limited in list order: no round-off rule, so that every clip is the reference's), the fit rows
// [N][FitLayout::width] and the clip words [N][V].
template <int D, bool Limit>
__global__ void __launch_bounds__(kTileCells, adj_min_blocks<D>()) k_sweep_fit(MeshDev<D> m, GeometryDev<D, double> geo, int tile0,
                                                                             const double* __restrict__ prims, double* __restrict__ wg,
                                                                             double* __restrict__ fit, int32_t* __restrict__ clip) {
    constexpr int V = D + 2;
    using FL = FitLayout<D>;
    extern __shared__ double2 staged_rows[];
    double* rows = reinterpret_cast<double*>(staged_rows);
    const int tile = tile0 + static_cast<int>(blockIdx.x);
    stage_rows<D>(geo, tile, prims, PS, rows);
    const int64_t t = static_cast<int64_t>(tile) * kTileCells + threadIdx.x;
    const int i = geo.order[t];
    if (i < 0) return;
    const int count = m.start[i + 1] - m.start[i];
    const int64_t slot0 = static_cast<int64_t>(geo.slice_base[t >> 5]) * 32 + (t & 31);
    const unsigned long long once = l2_evict_first();
    double Wi[V], lo[V], hi[V], g[V * D];
    int lo_k[V], hi_k[V];
#pragma unroll
    for (int v = 0; v < V; ++v) {
        Wi[v] = rows[kFitStaged * threadIdx.x + v];
        lo[v] = finite_max<double>();
        hi[v] = -finite_max<double>();
        lo_k[v] = hi_k[v] = 0;
#pragma unroll
        for (int a = 0; a < D; ++a) g[D * v + a] = 0;
    }
    bool any_tiny = false;
    constexpr int kBatch = 2;  // entries whose rows are requested together
    for (int k0 = 0; k0 < count; k0 += kBatch) {
        unsigned int word[kBatch];
        double c[kBatch][D];
#pragma unroll
        for (int b = 0; b < kBatch; ++b) {
            if (k0 + b >= count) continue;
            const int64_t slot = slot0 + 32 * static_cast<int64_t>(k0 + b);
            word[b] = geo.nbr[slot];
            const double2 c01 = geo.c01[slot];
            c[b][0] = c01.x;
            c[b][1] = c01.y;
            if constexpr (D == 3) c[b][2] = geo.c2[slot];
        }
#pragma unroll
        for (int b = 0; b < kBatch; ++b) {
            const int k = k0 + b;
            if (k >= count) continue;
            const double* rj = rows + kFitStaged * static_cast<int>(word[b] & kIndexMask);
            double Wj[kFitStaged];
#pragma unroll
            for (int q = 0; q < (D == 3 ? 6 : 4); q += 2) {
                const double2 w2 = *reinterpret_cast<const double2*>(rj + q);
                Wj[q] = w2.x;
                Wj[q + 1] = w2.y;
            }
            const bool tiny_face = (word[b] & kTinyBit) != 0;
            any_tiny = any_tiny || tiny_face;
#pragma unroll
            for (int v = 0; v < V; ++v) {
                const double dW = Wj[v] - Wi[v];
#pragma unroll
                for (int a = 0; a < D; ++a) g[D * v + a] += c[b][a] * dW;
                if (!tiny_face) {  // neighbour_range (finite_volume.hpp:572-588) leaves the tiny faces out
                    if (Wj[v] < lo[v]) lo[v] = Wj[v], lo_k[v] = k;
                    if (Wj[v] > hi[v]) hi[v] = Wj[v], hi_k[v] = k;
                }
            }
        }
    }
    double* fr = fit + static_cast<int64_t>(FL::width) * i;
    store_bar<V * D>(fr + FL::g0, g);
    int flag[V], clip_k[V];
#pragma unroll
    for (int v = 0; v < V; ++v) flag[v] = clip_k[v] = 0;
    if constexpr (Limit) {
        for (int k = 0; k < count; ++k) {
            const int64_t slot = slot0 + 32 * static_cast<int64_t>(k);
            if (any_tiny && (geo.nbr[slot] & kTinyBit)) continue;
            const double2 o01 = ldg_hint(geo.off01 + slot, once);
            double offset[D];
            offset[0] = o01.x;
            offset[1] = o01.y;
            if constexpr (D == 3) offset[2] = ldg_hint(geo.off2 + slot, once);
#pragma unroll
            for (int v = 0; v < V; ++v) {
                double* gv = g + D * v;
                const double dp = dot<D>(gv, offset);
                if (dp > 0 && Wi[v] + dp > hi[v]) {
                    const double s = hi[v] > Wi[v] ? (hi[v] - Wi[v]) / dp : 0.0;
#pragma unroll
                    for (int a = 0; a < D; ++a) gv[a] = gv[a] * s;
                    flag[v] = hi[v] > Wi[v] ? 3 : 7, clip_k[v] = k;
                } else if (dp < 0 && Wi[v] + dp < lo[v]) {
                    const double s = lo[v] < Wi[v] ? (lo[v] - Wi[v]) / dp : 0.0;
#pragma unroll
                    for (int a = 0; a < D; ++a) gv[a] = gv[a] * s;
                    flag[v] = lo[v] < Wi[v] ? 1 : 5, clip_k[v] = k;
                }
            }
        }
    }
#pragma unroll
    for (int v = 0; v < V; ++v) {
        const bool upper = (flag[v] & 2) != 0;
        fr[FL::bound + v] = upper ? hi[v] : lo[v];
        clip[V * static_cast<int64_t>(i) + v] = clip_word(flag[v], clip_k[v], upper ? hi_k[v] : lo_k[v]);
    }
    store_wg<D>(wg, i, Wi, g);
}

// AdjointFaces (finite_volume.hpp:2078-2102): per face, the bars of its two face states from Qbar's jump across it, into
// the face's row of two sides.
template <int D, int Riemann>
__global__ void __launch_bounds__(128, adj_min_blocks<D>()) k_faces_adjoint(int faces, const FaceRow<double>* __restrict__ face_rows,
                                                                          const double* __restrict__ wg, const double* __restrict__ qbar, double dt,
                                                                          GasDev gas, double* __restrict__ face_bar) {
    constexpr int V = D + 2, B = bar_stride<D>();
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= faces) return;
    FaceRow<double> r;
    load_face_row<double>(face_rows + f, r);
    double Lbar[V], Rbar[V];
#pragma unroll
    for (int v = 0; v < V; ++v) Lbar[v] = Rbar[v] = 0;
    if (r.mag != 0) {
        double L[V], R[V], Fbar[V];
#pragma unroll
        for (int v = 0; v < V; ++v)
            Fbar[v] = r.mag * dt * (qbar[V * static_cast<int64_t>(r.j) + v] - qbar[V * static_cast<int64_t>(r.o) + v]);
        {
            double W[V], g[V * D];
            load_wg<D>(wg, r.o, W, g);
            side_value<D>(W, g, r.offo, dt, gas.gamma, L);
        }
        {
            double W[V], g[V * D];
            load_wg<D>(wg, r.j, W, g);
            side_value<D>(W, g, r.offj, dt, gas.gamma, R);
        }
        if constexpr (Riemann == 1)
            hll_flux_adjoint<D>(L, R, r.n, gas, Fbar, Lbar, Rbar);
        else
            hllc_flux_adjoint<D>(L, R, r.n, gas, Fbar, Lbar, Rbar);
    }
    double* row = face_bar + 2 * B * static_cast<int64_t>(f);
    store_bar<V>(row, Lbar);
    store_bar<V>(row + B, Rbar);
}

// AdjointCell (finite_volume.hpp:2107-2169), one thread a cell in the tiles' order (its entry rows are coalesced). The
// half step's adjoint is linear in its bar, and a cell's sides differ only in r: the bars are summed over the faces first
// and it is applied once.
template <int D>
__global__ void __launch_bounds__(kTileCells, adj_min_blocks<D>()) k_cell_adjoint(MeshDev<D> m, GeometryDev<D, double> geo,
                                                                                const double* __restrict__ wg, double* face_bar,
                                                                                const double* __restrict__ fit, const int32_t* __restrict__ clip,
                                                                                double dt, GasDev gas, double* __restrict__ wbar) {
    constexpr int V = D + 2, P = D + 1, B = bar_stride<D>();
    using FL = FitLayout<D>;
    const int64_t t = static_cast<int64_t>(blockIdx.x) * kTileCells + threadIdx.x;
    const int i = geo.order[t];
    if (i < 0) return;
    const int first = m.start[i], count = m.start[i + 1] - first;
    const int64_t slot0 = static_cast<int64_t>(geo.slice_base[t >> 5]) * 32 + (t & 31);
    double Wi[V], Wi_bar[V], gi_bar[V * D];
    {
        double gi[V * D], half[V], S[V];  // S: the bars of the sides that did not fall back, summed
        load_wg<D>(wg, i, Wi, gi);
        half_step_rate<D, double>(Wi, gi, gas.gamma, half);
#pragma unroll
        for (int v = 0; v < V; ++v) {
            half[v] = Wi[v] - 0.5 * dt * half[v];
            Wi_bar[v] = S[v] = 0;
        }
#pragma unroll
        for (int c = 0; c < V * D; ++c) gi_bar[c] = 0;
        constexpr int kBatch = 2;  // entries whose rows are requested together
        for (int k0 = 0; k0 < count; k0 += kBatch) {
            int32_t e[kBatch];
            double mb[kBatch][V], r[kBatch][D];
#pragma unroll
            for (int b = 0; b < kBatch; ++b) e[b] = k0 + b < count ? m.list[first + k0 + b] : 0;
#pragma unroll
            for (int b = 0; b < kBatch; ++b) {
                if (k0 + b >= count) continue;
                const int64_t slot = slot0 + 32 * static_cast<int64_t>(k0 + b);
                load_bar<V>(face_bar + B * (2 * static_cast<int64_t>(list_face(e[b])) + (e[b] >= 0 ? 0 : 1)), mb[b]);
                const double2 o01 = geo.off01[slot];
                r[b][0] = o01.x;
                r[b][1] = o01.y;
                if constexpr (D == 3) r[b][2] = geo.off2[slot];
            }
#pragma unroll
            for (int b = 0; b < kBatch; ++b) {
                if (k0 + b >= count) continue;
                const bool fallback = !(half[0] + dot<D>(gi, r[b]) > 0 && half[P] + dot<D>(gi + D * P, r[b]) > 0);  // side_value
                if (fallback) {
#pragma unroll
                    for (int v = 0; v < V; ++v) Wi_bar[v] += mb[b][v];
                } else {
#pragma unroll
                    for (int v = 0; v < V; ++v) {
                        S[v] += mb[b][v];
#pragma unroll
                        for (int q = 0; q < D; ++q) gi_bar[D * v + q] += r[b][q] * mb[b][v];
                    }
                }
            }
        }
        half_step_adjoint<D>(Wi, gi, dt, gas.gamma, S, Wi_bar, gi_bar);
    }
    const double* fr = fit + static_cast<int64_t>(FL::width) * i;
    double bound[V];
    int bound_k[V];
#pragma unroll
    for (int v = 0; v < V; ++v) {  // gi_bar becomes g0's bar
        const int word = clip[V * static_cast<int64_t>(i) + v];
        bound[v] = 0;
        bound_k[v] = -1;
        if ((word & 1) && (word & 4)) {
#pragma unroll
            for (int a = 0; a < D; ++a) gi_bar[D * v + a] = 0;
        } else if (word & 1) {
            const int64_t slot = slot0 + 32 * static_cast<int64_t>(clip_entry(word));
            double o[D], g0[D];
            const double2 o01 = geo.off01[slot];
            o[0] = o01.x;
            o[1] = o01.y;
            if constexpr (D == 3) o[2] = geo.off2[slot];
#pragma unroll
            for (int a = 0; a < D; ++a) g0[a] = fr[FL::g0 + D * v + a];
            const double den = dot<D>(g0, o);
            const double s = (fr[FL::bound + v] - Wi[v]) / den, tb = dot<D>(gi_bar + D * v, g0) / den;
#pragma unroll
            for (int a = 0; a < D; ++a) gi_bar[D * v + a] = gi_bar[D * v + a] * s - o[a] * (s * tb);
            bound[v] = tb;
            bound_k[v] = bound_entry(word);
            Wi_bar[v] -= tb;
        }
    }
    for (int k = 0; k < count; ++k) {
        const int64_t slot = slot0 + 32 * static_cast<int64_t>(k);
        const int32_t e = m.list[first + k];
        const double2 c01 = geo.c01[slot];
        double c[D], share[V];
        c[0] = c01.x;
        c[1] = c01.y;
        if constexpr (D == 3) c[2] = geo.c2[slot];
#pragma unroll
        for (int v = 0; v < V; ++v) {
            share[v] = dot<D>(c, gi_bar + D * v);
            Wi_bar[v] -= share[v];
            if (k == bound_k[v]) share[v] += bound[v];
        }
        store_bar<V>(face_bar + B * (2 * static_cast<int64_t>(list_face(e)) + (e >= 0 ? 0 : 1)), share);
    }
#pragma unroll
    for (int v = 0; v < V; ++v) wbar[V * static_cast<int64_t>(i) + v] = Wi_bar[v];
}

// AdjointGather (finite_volume.hpp:2171-2195): Qbar_j += primitive_adjoint(W_j bar) / V_j, W_j's bar its own and its
// neighbours' shares, from the other side of each of its faces' rows.
template <int D>
__global__ void __launch_bounds__(128) k_gather_adjoint(MeshDev<D> m, const double* __restrict__ q, const double* __restrict__ wbar,
                                                        const double* __restrict__ face_bar, GasDev gas, double* __restrict__ qbar) {
    constexpr int V = D + 2, B = bar_stride<D>();
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= m.n) return;
    double W_bar[V];
#pragma unroll
    for (int v = 0; v < V; ++v) W_bar[v] = wbar[V * static_cast<int64_t>(j) + v];
    constexpr int kBatch = 4;  // rows requested together
    const int first = m.start[j], end = m.start[j + 1];
    for (int k0 = first; k0 < end; k0 += kBatch) {
        int32_t e[kBatch];
        double share[kBatch][V];
#pragma unroll
        for (int b = 0; b < kBatch; ++b) e[b] = k0 + b < end ? m.list[k0 + b] : 0;
#pragma unroll
        for (int b = 0; b < kBatch; ++b)
            if (k0 + b < end) load_bar<V>(face_bar + B * (2 * static_cast<int64_t>(list_face(e[b])) + (e[b] >= 0 ? 1 : 0)), share[b]);
#pragma unroll
        for (int b = 0; b < kBatch; ++b)
            if (k0 + b < end)
#pragma unroll
                for (int v = 0; v < V; ++v) W_bar[v] += share[b][v];
    }
    const double inv = 1.0 / m.vol[j];
    double Uj[V], U_bar[V];
#pragma unroll
    for (int v = 0; v < V; ++v) Uj[v] = q[V * static_cast<int64_t>(j) + v] * inv;
    primitive_adjoint<D>(Uj, W_bar, gas, U_bar);
#pragma unroll
    for (int v = 0; v < V; ++v) qbar[V * static_cast<int64_t>(j) + v] += U_bar[v] * inv;
}

}  // namespace luna
