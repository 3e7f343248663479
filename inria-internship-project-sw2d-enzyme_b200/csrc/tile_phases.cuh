// tile_phases.cuh — the edge bodies of a tile held in shared memory, shared by the fused flux kernel
// (sw2d_tile.cu) and the run kernel of small meshes (sw2d_run.cu), and the cp.async helpers both
// stage a tile with.
#pragma once

#include "sw2d_internal.cuh"

namespace sw2d {

// Asynchronous global -> shared copies (cp.async, sm_80+): every copy of a tile is issued before
// the first is waited for, so the loads of a tile are in flight together.
__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cpa16(void* s, const void* g)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(smem_addr(s)), "l"(g) : "memory");
}
__device__ __forceinline__ void cpa8(void* s, const void* g)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(smem_addr(s)), "l"(g) : "memory");
}
__device__ __forceinline__ void cpa4(void* s, const void* g)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(smem_addr(s)), "l"(g) : "memory");
}
__device__ __forceinline__ void cpa_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// One internal edge of a tile: Riemann states from the staged cells, lambda_max, HLLC.  `lam(side, v)`
// takes the CFL contribution of a side's cell, `put(side, slot)` its balance slot when the flux is
// computed; both are called for the sides whose cell belongs to the tile.  The arithmetic is
// edge_internal's (sp_phases.cuh).  Returns the status bits; lm and f are kept for recording.
struct TileEdge {
    int a, b;                // local L and R
    double2 n, cf;           // normal, {coefL, coefR}
    double len, phig;
    double2 ga, gb;          // slopes of L and R
    double2 da, db;          // midpoint - centroid of L and R
};

template <int kScheme, bool kBlending, int kModel, class D, class Lam, class Put>
__device__ __forceinline__ unsigned tile_edge(const DevMesh& m, const TileEdge& E, const double4& Sa, const double4& Sb,
                                              const double4& Ka, const double4& Kb, double dtp, bool ownL, bool ownR,
                                              double& lm, EdgeFlux& f, bool& flux, Lam&& lam, Put&& put)
{
    constexpr bool kDip = kModel == kModelDip;
    unsigned bad = 0;
    SideState SL, SR;
    const double2 n = E.n;
    double xL = 1.0, xR = 1.0;
    if (kDip) {
        xL = dip_x(Ka.z, E.phig);
        xR = dip_x(Kb.z, E.phig);
    }
    if (kScheme == SW2D_SCHEME_GODUNOV) {
        if (kDip) {
            SL = godunov_side_dip<D>(Sa.x, Sa.y, Sa.z, Ka.x, Ka.y, xL, n.x, n.y);
            SR = godunov_side_dip<D>(Sb.x, Sb.y, Sb.z, Kb.x, Kb.y, xR, n.x, n.y);
        } else {
            SL = godunov_side<D>(Sa.x, Sa.y, Sa.z, Ka.x, Ka.y, n.x, n.y);
            SR = godunov_side<D>(Sb.x, Sb.y, Sb.z, Kb.x, Kb.y, n.x, n.y);
        }
    } else if (kDip) {
        SL = evr_side_dip<D>(true, Sa.x, Sa.y, Sa.z, Ka.x, Ka.y, xL, Sa.w, E.ga.x, E.ga.y, E.da.x, E.da.y, n.x, n.y, dtp);
        SR = evr_side_dip<D>(false, Sb.x, Sb.y, Sb.z, Kb.x, Kb.y, xR, Sb.w, E.gb.x, E.gb.y, E.db.x, E.db.y, n.x, n.y, dtp);
    } else {
        SL = evr_side<D>(true, Sa.x, Sa.y, Sa.z, Ka.x, Ka.y, Sa.w, E.ga.x, E.ga.y, E.da.x, E.da.y, n.x, n.y, dtp, m.dry);
        SR = evr_side<D>(false, Sb.x, Sb.y, Sb.z, Kb.x, Kb.y, Sb.w, E.gb.x, E.gb.y, E.db.x, E.db.y, n.x, n.y, dtp, m.dry);
    }
    lm = max4(fabs(SL.lm), fabs(SL.lp), fabs(SR.lm), fabs(SR.lp));
    const double lw = lm * E.len;
    const bool wetL = Sa.x > m.h_min, wetR = Sb.x > m.h_min;
    if (ownL) lam(0, wetL ? lw : 0.0);
    if (ownR) lam(1, (wetL || wetR) ? lw : 0.0);
    const double hL = SL.z - Ka.x, hR = SR.z - Kb.x;
    flux = (hL > m.h_min) || (hR > m.h_min);
    if (flux) {
        f = kDip ? hllc_dip<D>(kBlending, Ka.y, Kb.y, E.phig, Ka.z, Kb.z, Ka.x, Kb.x, SL, SR, m.h_min, m.phi_min)
                 : hllc<D>(kBlending, Ka.y, Kb.y, Ka.z, Kb.z, Ka.x, Kb.x, SL, SR, m.h_min, m.phi_min);
        bad |= f.bad;
        if (isnan(f.f1)) bad |= kStatusNanFlux;
        const double nx = n.x, ny = n.y;
        if (ownL) {
            const double c = E.cf.x;
            const double f1 = -c, f2F2 = -c * nx, f2F3 = +c * ny, f2S2 = +c * nx;
            const double f3F2 = -c * ny, f3F3 = -c * nx, f3S2 = +c * ny;
            put(0, make_slot(f1 * f.f1, f2F2 * f.f2 + f2S2 * f.sl + f2F3 * f.f3, f3F2 * f.f2 + f3S2 * f.sl + f3F3 * f.f3));
        }
        if (ownR) {
            const double c = E.cf.y;
            const double f1 = +c, f2F2 = +c * nx, f2F3 = -c * ny, f2S2 = +c * nx;
            const double f3F2 = +c * ny, f3F3 = +c * nx, f3S2 = +c * ny;
            put(1, make_slot(f1 * f.f1, f2F2 * f.f2 + f2S2 * f.sr + f2F3 * f.f3, f3F2 * f.f2 + f3S2 * f.sr + f3F3 * f.f3));
        }
    }
    return bad;
}

// One boundary edge e (hypBoundaryFlux, swSpHyp.cpp:13-135) of a cell staged as {S, K}, as
// edge_boundary computes it; lambda_max and the fluxes are kept for recording.
template <int kScheme, int kModel, class D>
__device__ __forceinline__ unsigned tile_boundary(const DevMesh& m, int e, const double4& S, const double4& K, double t,
                                                  double& lm, double& cfl, double& f1, double& f2, double& f3, Slot& slot)
{
    constexpr bool kDip = kModel == kModelDip;
    const double4 g = ld(&m.bgeo[e]);
    const double phiGb = kDip ? ld(&m.phigb[e]) : 0.0;
    SideState R = kDip ? godunov_side_dip<D>(S.x, S.y, S.z, K.x, K.y, dip_x(K.z, phiGb), g.x, g.y)
                       : godunov_side<D>(S.x, S.y, S.z, K.x, K.y, g.x, g.y);
    lm = (kScheme == SW2D_SCHEME_GODUNOV) ? smax(fabs(R.lp), fabs(R.lm)) : smax(fabs(R.lm), fabs(R.lp));
    cfl = (S.x > m.h_min) ? lm * g.z : 0.0;
    const int k = ld(&m.bbc[e]);
    const long long o0 = ld(&m.bcoff[k]), o1 = ld(&m.bcoff[k + 1]);
    const double v = bc_value(m.bctimes + o0, m.bcvals + o0, o1 - o0, t);
    const unsigned bad = kDip ? boundary_flux_dip(K.y, phiGb, K.z, K.x, R, ld(&m.bctype[k]), v, m.h_min, &f1, &f2, &f3)
                              : boundary_flux(K.y, K.z, K.x, R, ld(&m.bctype[k]), v, m.h_min, &f1, &f2, &f3);
    const double cf = g.w, nx = g.x, ny = g.y;
    const double fa = +cf, f2F2 = +cf * nx, f2F3 = -cf * ny, f2S2 = +cf * nx;
    const double f3F2 = +cf * ny, f3F3 = +cf * nx, f3S2 = +cf * ny;
    const double s2 = 0.0;  // boundary geometric source: never set by hypBoundaryFlux
    slot = make_slot(fa * f1, f2F2 * f2 + f2S2 * s2 + f2F3 * f3, f3F2 * f2 + f3S2 * s2 + f3F3 * f3);
    return bad;
}

}  // namespace sw2d
