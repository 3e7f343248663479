// sw2d_run.cu — many time steps of a small SP or DIP mesh in one launch.
//
// The four-kernel step of a mesh that does not fill the GPU is bound by latency: its kernels take
// 6-9 us each whatever the mesh (graph-launched step: 18 us at 2,000 cells, 20 us at 20,000), most of
// it launch gaps, dependent trips to L2 for tables that never change, and grid-wide reductions.
// k_run keeps the mesh on chip instead.  One CTA per tile of consecutive (Hilbert-ordered) cells,
// all CTAs resident at once (cooperative launch), holds in shared memory the tile's cells, the two
// rings of cells around it, its edges and balance slots for the whole launch, and steps as the
// fused form does (sw2d_tile.cu): slopes of the tile and ring 1, every edge with a cell in the tile,
// the CFL bound, the update of the tile's own cells.  Two exchanges per step remain:
//   * the time step: each CTA publishes its CFL minimum and reads everybody's;
//   * the new states: each CTA publishes its cells and reads those of its rings.
// Both go through L2 as words that carry 32 bits of data and the step's 32-bit epoch: a reader polls
// the word itself, so no fence, counter or barrier is needed, one store-to-load trip each.
//   - A minimum is read by every CTA before any CTA passes two steps further: two slots in turn.
//   - A state is read before its owner can write the next one: the owner first needs the next step's
//     minimum of every CTA, which each publishes after it has read its rings: one slot.
// Every wait is bounded; a wait that runs out sets the status word and ends the launch, and the call
// reports it (the state is then undefined until it is set or restored).  The arithmetic is that of the
// four kernels (sp_phases.cuh, tile_phases.cuh), operand for operand, so the results are the same bits,
// and the four kernels serve wherever this one does not: no memory for the tiles or no room for them on
// chip, a new handle's first steps (run_worth), other handles' calls in progress (RunTurn).
//
// A pair of lanes takes each slope and each internal edge while a tile's edges then still fit one pass
// of the CTA (up to about 20k cells on 148 SMs): one component of the slope, one side's Riemann state.
// Divisions and roots are the forms that keep zeros off the general routine (DivZero).
//
// Measured (B200, us per step, graph of the chained four kernels -> k_run): MUSCL-EVR 500 cells 15.8 -> 7.6,
// 2,000 16.7 -> 8.2, 20,000 18.7 -> 10.7, 40,000 20.8 -> 12.1, 60,000 24.3 -> 15.0; Godunov 5,000 15.9 -> 7.7,
// 20,000 16.1 -> 9.0, 60,000 18.9 -> 12.6; DIP 20,000 20.5 -> 12.3, 60,000 27.4 -> 20.2, its Godunov 20,000
// 15.4 -> 8.8.  A tile of about 450 cells fills the shared memory of an SM, which ends the range.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <string>
#include <vector>

#include "sp_phases.cuh"
#include "sw2d_internal.cuh"
#include "tile_phases.cuh"

namespace sw2d {

struct RunLayout {  // byte offsets of a tile's sections in shared memory (every section 16-byte aligned)
    int st, cst, xy, sl, coff, lam, slot, en, ecf, elen, esl, epg, eg, ell, ent, so, fric, smem;
};

struct RunState {
    TileMesh tm{};
    std::vector<void*> tile_allocs, allocs;
    RunLayout lay{};
    ulonglong2* pk_dt = nullptr;  // [2][tiles] CFL minima, a line each
    ulonglong2* pk_st = nullptr;  // [kRunWords * cells] states {h, q, r}
    unsigned epoch = 0;           // epochs used so far
    bool pairs = false;           // a pair of lanes per edge
    bool ok = false;              // false: the mesh does not fit, the four-kernel step serves
};

namespace {

using ull = unsigned long long;

struct RunArgs {
    ulonglong2* pk_dt;
    ulonglong2* pk_st;
    unsigned epoch;  // the first step's
    int n;           // steps of this launch
    int friction, head_loss, dissip;
    long long polls;
};

// steps of one launch: bounds its duration (about 10 ms), not its results
constexpr int kRunSteps = 1024;
constexpr int kRunThreads = 512;
// A CTA's minimum has a 128-byte line of its own: 148 CTAs exchange in 2,100 cycles, against 6,300 with
// the minima packed (every CTA polls lines that eight others still write).
constexpr int kRunLine = 8;
constexpr int kRunWords = 3;  // ulonglong2 of a cell's state
constexpr long long kRunPolls = 1ll << 22;  // a few seconds of polling

__device__ __forceinline__ void put_words(ulonglong2* p, unsigned epoch, double v)
{
    const ull e = (ull)epoch << 32, b = (ull)__double_as_longlong(v);
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(e | (b & 0xffffffffull)), "l"(e | (b >> 32))
                 : "memory");
}

// the value at p if both its words carry the epoch
__device__ __forceinline__ bool get_words(const ulonglong2* p, unsigned epoch, double& v)
{
    ull a, b;
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
    v = __longlong_as_double((long long)((b << 32) | (a & 0xffffffffull)));
    return (unsigned)(a >> 32) == epoch && (unsigned)(b >> 32) == epoch;
}

// the warp's minimum (no NaN among the values) by integer reductions of order-preserving keys
__device__ __forceinline__ double warp_min(double v)
{
    const ull key = dmin_key((ull)__double_as_longlong(v));
    const unsigned hi = (unsigned)(key >> 32), mh = __reduce_min_sync(0xffffffffu, hi);
    const unsigned ml = __reduce_min_sync(0xffffffffu, hi == mh ? (unsigned)key : 0xffffffffu);
    return __longlong_as_double((long long)dmin_bits((ull)mh << 32 | ml));
}

struct RunStage {
    double4 *st, *cst;
    double2 *xy, *sl;
    int2* coff;
    double* lam;
    Slot* slot;
    double2 *en, *ecf;
    double* elen;
    int2* esl;
    double* epg;
    double4* eg;
    ushort2* ell;
    unsigned *ent, *so;
    double4* fric;
};

__device__ __forceinline__ RunStage run_stage(unsigned char* s, const RunLayout& o)
{
    RunStage v;
    v.st = reinterpret_cast<double4*>(s + o.st);
    v.cst = reinterpret_cast<double4*>(s + o.cst);
    v.xy = reinterpret_cast<double2*>(s + o.xy);
    v.sl = reinterpret_cast<double2*>(s + o.sl);
    v.coff = reinterpret_cast<int2*>(s + o.coff);
    v.lam = reinterpret_cast<double*>(s + o.lam);
    v.slot = reinterpret_cast<Slot*>(s + o.slot);
    v.en = reinterpret_cast<double2*>(s + o.en);
    v.ecf = reinterpret_cast<double2*>(s + o.ecf);
    v.elen = reinterpret_cast<double*>(s + o.elen);
    v.esl = reinterpret_cast<int2*>(s + o.esl);
    v.epg = reinterpret_cast<double*>(s + o.epg);
    v.eg = reinterpret_cast<double4*>(s + o.eg);
    v.ell = reinterpret_cast<ushort2*>(s + o.ell);
    v.ent = reinterpret_cast<unsigned*>(s + o.ent);
    v.so = reinterpret_cast<unsigned*>(s + o.so);
    v.fric = reinterpret_cast<double4*>(s + o.fric);
    return v;
}

// num / den of the limiter, den != 0 of either sign: num is zero wherever the cell itself holds the
// smaller (larger) level, and sw2d_div says what a zero costs
__device__ __forceinline__ double limiter_factor(double num, double den)
{
    const bool z = num == 0.0;
    const double q = (z ? den : num) / den;
    return z ? (den < 0.0 ? -num : num) : q;
}

// the limited slope of staged cell l (slopes_cell, sp_phases.cuh)
__device__ __forceinline__ double2 run_slope(const RunStage& sv, int l, bool plain)
{
    const int k0 = (int)sv.so[l], cnt = (int)sv.so[l + 1] - k0;
    const double zc = sv.st[l].w;
    const double2 xy = sv.xy[l];
    double sx = 0.0, sy = 0.0;
    if (cnt <= kUnrollSlopes) {
        unsigned en[kUnrollSlopes];
        double zj[kUnrollSlopes];
        bool ok = plain;
#pragma unroll
        for (int i = 0; i < kUnrollSlopes; i++)
            if (i < cnt) {
                en[i] = sv.ent[k0 + i];
                zj[i] = sv.st[en[i] & 0xffffu].w;
                ok = ok && div_range_ok(zj[i] - zc);
            }
        if (cnt > 1) {
            double wsum = 0.0;
#pragma unroll
            for (int i = 0; i < kUnrollSlopes; i++)
                if (i < cnt) {
                    const double2 xj = sv.xy[en[i] & 0xffffu];
                    if (ok) {
                        const double4 g = sv.eg[(en[i] >> 16) & 0x7fffu];
                        const double dz = zj[i] - zc;
                        sx += div_known(div_known(dz * (xj.x - xy.x), g.x, g.y), g.x, g.y) * g.y;
                        sy += div_known(div_known(dz * (xj.y - xy.y), g.x, g.y), g.x, g.y) * g.y;
                        wsum += g.y;
                    } else {
                        grad_term(zc, zj[i], xy, xj, sx, sy, wsum);
                    }
                }
            sx = sw2d_div(sx, wsum);
            sy = sw2d_div(sy, wsum);
        }
#pragma unroll
        for (int i = 0; i < kUnrollSlopes; i++)
            if (i < cnt) {
                const double4 g = sv.eg[(en[i] >> 16) & 0x7fffu];
                limit_slope(zc, zj[i], (en[i] >> 31) != 0, make_double2(g.z, g.w), xy, sx, sy);
            }
        return make_double2(sx, sy);
    }
    double wsum = 0.0;
    for (int k = k0; k < k0 + cnt; k++) {
        const unsigned j = sv.ent[k] & 0xffffu;
        grad_term(zc, sv.st[j].w, xy, sv.xy[j], sx, sy, wsum);
    }
    sx /= wsum;
    sy /= wsum;
    for (int k = k0; k < k0 + cnt; k++) {
        const unsigned en = sv.ent[k];
        const double4 g = sv.eg[(en >> 16) & 0x7fffu];
        limit_slope(zc, sv.st[en & 0xffffu].w, (en >> 31) != 0, make_double2(g.z, g.w), xy, sx, sy);
    }
    return make_double2(sx, sy);
}

__device__ __forceinline__ double swap_pair(double v) { return __shfl_xor_sync(0xffffffffu, v, 1); }

// Component p (0: x, 1: y) of the limited slope of staged cell l, by a pair of lanes: each takes its
// component's chain and the two exchange the products of the limiter.  Every lane of the warp calls it.
__device__ __forceinline__ double run_slope_pair(const RunStage& sv, int l, int p, bool plain)
{
    const int k0 = (int)sv.so[l], cnt = (int)sv.so[l + 1] - k0;
    const double zc = sv.st[l].w;
    const double xc = reinterpret_cast<const double*>(&sv.xy[l])[p];
    unsigned en[kUnrollSlopes];
    double zj[kUnrollSlopes];
    double s = 0.0, wsum = 0.0;
    bool ok = plain;
#pragma unroll
    for (int i = 0; i < kUnrollSlopes; i++) {
        en[i] = i < cnt ? sv.ent[k0 + i] : 0u;
        zj[i] = i < cnt ? sv.st[en[i] & 0xffffu].w : zc;
        ok = ok && div_range_ok(zj[i] - zc);
    }
#pragma unroll
    for (int i = 0; i < kUnrollSlopes; i++)
        if (i < cnt) {
            const double2 g = *reinterpret_cast<const double2*>(&sv.eg[(en[i] >> 16) & 0x7fffu]);
            const double v = (zj[i] - zc) * (reinterpret_cast<const double*>(&sv.xy[en[i] & 0xffffu])[p] - xc);
            s += (ok ? div_known(div_known(v, g.x, g.y), g.x, g.y) : v / g.x / g.x) * g.y;
            wsum += g.y;
        }
    s = cnt > 1 ? sw2d_div(s, wsum) : 0.0;
#pragma unroll
    for (int i = 0; i < kUnrollSlopes; i++) {
        const double mp = reinterpret_cast<const double*>(&sv.eg[(en[i] >> 16) & 0x7fffu])[2 + p];
        const double a = (mp - xc) * s, b = swap_pair(a);
        const double rec = zc + (p ? b : a) + (p ? a : b);
        const bool is_r = (en[i] >> 31) != 0;
        const double zL = is_r ? zj[i] : zc, zR = is_r ? zc : zj[i];
        const double fmx = smax(zL, zR), fmn = smin(zL, zR);
        const bool under = rec < fmn;
        if (i < cnt && (under || rec > fmx)) s *= limiter_factor((under ? fmn : fmx) - zc, rec - zc);
    }
    if (cnt > kUnrollSlopes) {  // not a triangle: each lane the whole slope
        const double2 g = run_slope(sv, l, plain);
        s = p ? g.y : g.x;
    }
    return s;
}

// One internal edge by a pair of lanes, as tile_edge: lane p holds side p (0: L, 1: R) of the Riemann
// states, both compute the flux, each writes its own cell's contribution.  Every lane of the warp calls
// it; `own` lanes of edges outside the tile's list write nothing.
template <int kScheme, bool kBlending, int kModel>
__device__ __forceinline__ unsigned run_edge_pair(const DevMesh& m, const RunStage& sv, int j, int p, double dtp, bool own,
                                                  int s0)
{
    constexpr bool kDip = kModel == kModelDip;
    constexpr bool kMuscl = kScheme == SW2D_SCHEME_MUSCL_EVR;
    const ushort2 ll = sv.ell[j];
    const int c = p ? ll.y : ll.x, o = p ? ll.x : ll.y;
    const double2 n = sv.en[j];
    const double4 S = sv.st[c], K = sv.cst[c], Ko = sv.cst[o];
    const double phig = kDip ? sv.epg[j] : 0.0;
    const double x = kDip ? dip_x(K.z, phig) : 1.0;
    SideState A, B;
    if (!kMuscl) {
        A = kDip ? godunov_side_dip<DivZero>(S.x, S.y, S.z, K.x, K.y, x, n.x, n.y) : godunov_side<DivZero>(S.x, S.y, S.z, K.x, K.y, n.x, n.y);
    } else {
        const double2 mp = *(reinterpret_cast<const double2*>(&sv.eg[j]) + 1), xy = sv.xy[c], g = sv.sl[c];
        const double dx = mp.x - xy.x, dy = mp.y - xy.y;
        A = kDip ? evr_side_dip<DivZero>(p == 0, S.x, S.y, S.z, K.x, K.y, x, S.w, g.x, g.y, dx, dy, n.x, n.y, dtp)
                 : evr_side<DivZero>(p == 0, S.x, S.y, S.z, K.x, K.y, S.w, g.x, g.y, dx, dy, n.x, n.y, dtp, m.dry);
    }
    B.z = swap_pair(A.z);
    B.q = swap_pair(A.q);
    B.r = swap_pair(A.r);
    B.lm = swap_pair(A.lm);
    B.lp = swap_pair(A.lp);
    const SideState SL = p ? B : A, SR = p ? A : B;
    const double4 Ka = p ? Ko : K, Kb = p ? K : Ko;
    const int2 sl = sv.esl[j];
    const int at = (p ? sl.y : sl.x) - s0;
    const double lw = max4(fabs(SL.lm), fabs(SL.lp), fabs(SR.lm), fabs(SR.lp)) * sv.elen[j];
    const bool wet = S.x > m.h_min, wet_o = sv.st[o].x > m.h_min;
    if (own) sv.lam[at] = (wet || (p && wet_o)) ? lw : 0.0;
    unsigned bad = 0;
    if ((SL.z - Ka.x > m.h_min) || (SR.z - Kb.x > m.h_min)) {
        const EdgeFlux f = kDip ? hllc_dip<DivZero>(kBlending, Ka.y, Kb.y, phig, Ka.z, Kb.z, Ka.x, Kb.x, SL, SR, m.h_min, m.phi_min)
                                : hllc<DivZero>(kBlending, Ka.y, Kb.y, Ka.z, Kb.z, Ka.x, Kb.x, SL, SR, m.h_min, m.phi_min);
        bad = f.bad;
        if (isnan(f.f1)) bad |= kStatusNanFlux;
        // the factors of tile_edge: L has -w / (A phi) on the fluxes, both + on the bed source
        const double2 cf = sv.ecf[j];
        const double c0 = p ? cf.y : cf.x, cs = p ? c0 : -c0, s2 = p ? f.sr : f.sl;
        const Slot v = make_slot(cs * f.f1, cs * n.x * f.f2 + c0 * n.x * s2 + -cs * n.y * f.f3,
                                 cs * n.y * f.f2 + c0 * n.y * s2 + cs * n.x * f.f3);
        if (own) sv.slot[at] = v;
    }
    return bad;
}

template <int kFriction>
__device__ __forceinline__ void run_sources_h(const DevMesh& m, int c, double dt, double hh, double& qq, double& rr,
                                              const double4* fr, bool head_loss)
{
    if (head_loss) cell_sources<kFriction, true>(m, c, dt, hh, qq, rr, nullptr, fr);
    else cell_sources<kFriction, false>(m, c, dt, hh, qq, rr, nullptr, fr);
}

__device__ __forceinline__ void run_sources(const DevMesh& m, int friction, bool head_loss, int c, double dt, double hh,
                                            double& qq, double& rr, const double4* fr)
{
    switch (friction) {
        case SW2D_FRICTION_CHEZY: run_sources_h<SW2D_FRICTION_CHEZY>(m, c, dt, hh, qq, rr, fr, head_loss); break;
        case SW2D_FRICTION_MANNING: run_sources_h<SW2D_FRICTION_MANNING>(m, c, dt, hh, qq, rr, fr, head_loss); break;
        case SW2D_FRICTION_STRICKLER: run_sources_h<SW2D_FRICTION_STRICKLER>(m, c, dt, hh, qq, rr, fr, head_loss); break;
        default: run_sources_h<SW2D_FRICTION_NONE>(m, c, dt, hh, qq, rr, nullptr, head_loss); break;
    }
}

// kPairs: a pair of lanes per slope and per internal edge (tiles whose edges then still take one pass)
template <int kScheme, bool kBlending, int kModel, bool kPairs>
__global__ void __launch_bounds__(kRunThreads, 1) k_run(DevMesh m, TileMesh tm, RunLayout lay, RunArgs a)
{
    constexpr bool kMuscl = kScheme == SW2D_SCHEME_MUSCL_EVR;
    constexpr bool kDip = kModel == kModelDip;
    constexpr int kThreads = kRunThreads, kWarps = kThreads / 32;
    extern __shared__ __align__(16) unsigned char run_smem[];
    __shared__ double wmin[2][kWarps];
    const RunStage sv = run_stage(run_smem, lay);
    const TileInfo ti = tm.info[blockIdx.x];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    Ctrl* ctrl = m.ctrl;
    double t = ctrl->t, dt = ctrl->dt;
    const double t_max = ctrl->t_max;
    if (!(t < t_max)) {  // the run is over (the same for every CTA)
        if (blockIdx.x == 0 && tid == 0) ctrl->go = 0;
        return;
    }
    const int nt = ti.nt, nf = nt + ti.nh1, nl = nf + ti.nh2, c0 = ti.c0, s0 = ti.s0;
    const int nflux = ti.ne_own + ti.nx_flux, nbe = ti.b1 - ti.b0;
    const bool has_fric = a.friction != SW2D_FRICTION_NONE;

    // ---- the tile, its rings and its edges into shared memory, for the whole launch
    for (int l = tid; l < nl; l += kThreads) {
        const int g = (l < nt) ? c0 + l : ld(&tm.halo[ti.hoff + l - nt]);
        cpa16(reinterpret_cast<double2*>(sv.st + l), reinterpret_cast<const double2*>(m.st + g));
        cpa16(reinterpret_cast<double2*>(sv.st + l) + 1, reinterpret_cast<const double2*>(m.st + g) + 1);
        if (kMuscl) cpa16(sv.xy + l, m.cxy + g);
        if (l < nf) {
            cpa16(reinterpret_cast<double2*>(sv.cst + l), reinterpret_cast<const double2*>(m.cst + g));
            cpa16(reinterpret_cast<double2*>(sv.cst + l) + 1, reinterpret_cast<const double2*>(m.cst + g) + 1);
        }
        if (has_fric && l < nt) {
            cpa16(reinterpret_cast<double2*>(sv.fric + l), reinterpret_cast<const double2*>(m.fric + g));
            cpa16(reinterpret_cast<double2*>(sv.fric + l) + 1, reinterpret_cast<const double2*>(m.fric + g) + 1);
        }
    }
    for (int l = tid; l <= nt; l += kThreads) cpa8(sv.coff + l, m.coff + c0 + l);
    const int ns = ld(&m.coff[c0 + nt].y) - s0;
    for (int k = tid; k < 3 * ns; k += kThreads)
        cpa8(reinterpret_cast<double*>(sv.slot) + k, reinterpret_cast<const double*>(m.slot + s0) + k);
    const int nall = kMuscl ? nflux + ti.nx_slope : nflux;
    for (int j = tid; j < nall; j += kThreads) {
        const int e = (j < ti.ne_own) ? ti.e0 + j : ld(&tm.xe[ti.xoff + j - ti.ne_own]);
        cpa4(sv.ell + j, tm.eloc + ti.loff + j);
        if (kMuscl) {
            cpa16(reinterpret_cast<double2*>(sv.eg + j), reinterpret_cast<const double2*>(m.egeo + e));
            cpa16(reinterpret_cast<double2*>(sv.eg + j) + 1, reinterpret_cast<const double2*>(m.egeo + e) + 1);
        }
        if (j < nflux) {
            cpa16(sv.en + j, m.nxy + e);
            cpa16(sv.ecf + j, m.coef + e);
            cpa8(sv.elen + j, m.len + e);
            cpa8(sv.esl + j, m.eslot + e);
            if (kDip) cpa8(sv.epg + j, m.phig + e);
        }
    }
    if (kMuscl) {
        for (int k = tid; k < ti.nent; k += kThreads) cpa4(sv.ent + k, tm.scsr + ti.soff + k);
        for (int l = tid; l <= nf; l += kThreads) cpa4(sv.so + l, tm.soffs + ti.so_off + l);
    }
    cpa_wait_all();
    __syncthreads();

    int steps = 0, store = 0;
    unsigned bad = 0;
    bool lost = false;  // a wait ran out
    while (steps < a.n && t < t_max) {
        const unsigned epoch = a.epoch + (unsigned)steps;
        if (kMuscl) {
            if (kPairs) {
                for (int i = wid * 32; i < 2 * nf; i += kThreads) {
                    const int l = min((i + lane) >> 1, nf - 1);
                    const double s = run_slope_pair(sv, l, lane & 1, m.geo_plain != 0);
                    if (i + lane < 2 * nf) reinterpret_cast<double*>(&sv.sl[l])[lane & 1] = s;
                }
            } else {
                for (int l = tid; l < nf; l += kThreads) sv.sl[l] = run_slope(sv, l, m.geo_plain != 0);
            }
            __syncthreads();
        }
        // ---- the tile's internal edges, then (from the next warp on) its boundary edges
        const int ni = kPairs ? 2 * nflux : nflux, nw = (ni + 31) & ~31;
        for (int i = tid; i < nw + nbe; i += kThreads) {
            if (i < nw) {
                if (kPairs) {
                    const int j = min(i >> 1, nflux - 1), p = lane & 1;
                    const ushort2 ll = sv.ell[j];
                    bad |= run_edge_pair<kScheme, kBlending, kModel>(m, sv, j, p, dt, i < ni && (p ? ll.y : ll.x) < nt, s0);
                    continue;
                }
                if (i >= ni) continue;
                const ushort2 ll = sv.ell[i];
                TileEdge E;
                E.a = ll.x;
                E.b = ll.y;
                E.n = sv.en[i];
                E.cf = sv.ecf[i];
                E.len = sv.elen[i];
                E.phig = kDip ? sv.epg[i] : 0.0;
                if (kMuscl) {
                    const double4 g = sv.eg[i];
                    const double2 ca = sv.xy[E.a], cb = sv.xy[E.b];
                    E.ga = sv.sl[E.a];
                    E.gb = sv.sl[E.b];
                    E.da = make_double2(g.z - ca.x, g.w - ca.y);
                    E.db = make_double2(g.z - cb.x, g.w - cb.y);
                }
                const int2 sl = sv.esl[i];
                double lm;
                EdgeFlux f;
                bool flux;
                bad |= tile_edge<kScheme, kBlending, kModel, DivZero>(
                    m, E, sv.st[E.a], sv.st[E.b], sv.cst[E.a], sv.cst[E.b], dt, E.a < nt, E.b < nt, lm, f, flux,
                    [&](int side, double v) { sv.lam[(side ? sl.y : sl.x) - s0] = v; },
                    [&](int side, const Slot& v) { sv.slot[(side ? sl.y : sl.x) - s0] = v; });
            } else {
                const int e = ti.b0 + i - nw;
                const int l = ld(&m.bcell[e]) - c0, k = ld(&m.bslot[e]) - s0;
                double lm, cfl, f1, f2, f3;
                Slot v;
                bad |= tile_boundary<kScheme, kModel, DivZero>(m, e, sv.st[l], sv.cst[l], t, lm, cfl, f1, f2, f3, v);
                sv.lam[k] = cfl;
                sv.slot[k] = v;
            }
        }
        __syncthreads();
        // ---- CFL bound of the tile, published; everybody's read (hypComputeTimeStep)
        double best = m.dt_max;
        for (int l = tid; l < nt; l += kThreads) {
            double sw = 0.0;
            for (int k = sv.coff[l].y - s0; k < sv.coff[l + 1].y - s0; k++) sw += sv.lam[k];
            best = min_keep(best, m.cfl_max * (sv.cst[l].w / smax(sw, kSmallReal)));
        }
        best = warp_min(best);
        if (lane == 0) wmin[0][wid] = best;
        __syncthreads();
        ulonglong2* pk = a.pk_dt + kRunLine * (epoch & 1u) * gridDim.x;
        if (wid == 0) {
            best = warp_min(lane < kWarps ? wmin[0][lane] : m.dt_max);
            if (lane == 0) put_words(pk + kRunLine * blockIdx.x, epoch, best);
        }
        best = m.dt_max;
        for (int i = tid; i < (int)gridDim.x; i += kThreads) {
            double v;
            long long polls = 0;
            while (!get_words(pk + kRunLine * i, epoch, v))
                if (++polls > a.polls) {
                    lost = true;
                    break;
                }
            if (!lost) best = min_keep(best, v);
        }
        best = warp_min(best);
        if (lane == 0) wmin[1][wid] = best;
        if (__syncthreads_or(lost)) {
            lost = true;
            break;
        }
        dt = warp_min(lane < kWarps ? wmin[1][lane] : m.dt_max);
        dt = dt_snap<false>(m.dt_map, t, t_max, dt, store);
        // ---- balance and sources of the tile's cells (update_cell), published
        for (int l = tid; l < nt; l += kThreads) {
            const int c = c0 + l;
            const double4 v0 = sv.st[l];
            double hh = v0.x, qq = v0.y, rr = v0.z;
            for (int k = sv.coff[l].y - s0; k < sv.coff[l + 1].y - s0; k++) {
                const Slot v = sv.slot[k];
                hh += v.a * dt;
                qq += v.b * dt;
                rr += v.c * dt;
            }
            if (kDip && a.dissip) {
                const double4 mu = ld(&m.mu[c]);
                momentum_dissipation(mu.x, mu.y, mu.z, mu.w, v0.x, v0.y, v0.z, hh, qq, rr);
            }
            if (fabs(hh) < kSmallReal) hh = 0.;
            if (fabs(qq) < kSmallReal) qq = 0.;
            if (fabs(rr) < kSmallReal) rr = 0.;
            if (m.neg_detect) {
                if (hh < 0) bad |= kStatusNegDepth;
            } else if (hh < 0.) {
                hh = 0.;
                qq = 0.;
                rr = 0.;
            }
            double4 fr = make_double4(0.0, 0.0, 0.0, 0.0);
            if (has_fric) fr = sv.fric[l];
            run_sources(m, a.friction, a.head_loss != 0, c, dt, hh, qq, rr, &fr);
            sv.st[l] = make_double4(hh, qq, rr, hh + sv.cst[l].x);
            ulonglong2* p = a.pk_st + kRunWords * (size_t)c;
            put_words(p, epoch, hh);
            put_words(p + 1, epoch, qq);
            put_words(p + 2, epoch, rr);
        }
        t = t + dt;  // swSp.cpp:592
        steps++;
        if (!(steps < a.n && t < t_max)) break;
        // ---- the rings' new states
        for (int l = nt + tid; l < nl; l += kThreads) {
            const int g = ld(&tm.halo[ti.hoff + l - nt]);
            const ulonglong2* p = a.pk_st + kRunWords * (size_t)g;
            double h, q, r;
            long long polls = 0;
            for (;;) {
                const bool x = get_words(p, epoch, h), y = get_words(p + 1, epoch, q), z = get_words(p + 2, epoch, r);
                if (x && y && z) break;
                if (++polls > a.polls) {
                    lost = true;
                    break;
                }
            }
            // z = h + z_b, as the owner stores it (ring 2 holds no statics: z_b from memory)
            sv.st[l] = make_double4(h, q, r, h + (l < nf ? sv.cst[l].x : ld(&m.zbv[g])));
        }
        if (__syncthreads_or(lost)) {
            lost = true;
            break;
        }
    }
    if (lost) {
        if (tid == 0) atomicOr(&ctrl->status, kStatusRunWait);
        return;
    }
    __syncthreads();
    // ---- the tile's states, balance slots and slopes back to memory
    for (int l = tid; l < nt; l += kThreads) {
        m.st[c0 + l] = sv.st[l];
        if (kMuscl) m.slope[c0 + l] = sv.sl[l];
    }
    for (int k = tid; k < 3 * ns; k += kThreads)
        reinterpret_cast<double*>(m.slot + s0)[k] = reinterpret_cast<const double*>(sv.slot)[k];
    if (bad) atomicOr(&ctrl->status, bad);
    if (blockIdx.x == 0 && tid == 0) {
        ctrl->t = t;
        ctrl->dt = dt;
        ctrl->steps += steps;
        ctrl->store_map = store;
        ctrl->go = 1;
    }
}

RunLayout run_layout(const TileMesh& tm, bool muscl, bool dip, bool friction)
{
    RunLayout o{};
    size_t at = 0;
    auto sec = [&](int* off, size_t bytes) {
        *off = (int)at;
        at += (bytes + 15) & ~(size_t)15;
    };
    const size_t nl = tm.nl_max, nf = tm.nf_max, nt = tm.nt_max, ns = tm.ns_max, ne = tm.ne_max, na = tm.na_max;
    sec(&o.st, 32 * nl);
    sec(&o.cst, 32 * nf);
    sec(&o.xy, muscl ? 16 * nl : 0);
    sec(&o.sl, muscl ? 16 * nf : 0);
    sec(&o.coff, 8 * (nt + 1));
    sec(&o.lam, 8 * ns);
    sec(&o.slot, sizeof(Slot) * ns);
    sec(&o.en, 16 * ne);
    sec(&o.ecf, 16 * ne);
    sec(&o.elen, 8 * ne);
    sec(&o.esl, 8 * ne);
    sec(&o.epg, dip ? 8 * ne : 0);
    // at least one record: the pairs' slopes read the first one where a cell has fewer neighbours
    sec(&o.eg, muscl ? 32 * std::max<size_t>(na, 1) : 0);
    sec(&o.ell, 4 * na);
    sec(&o.ent, muscl ? 4 * (size_t)tm.nent_max : 0);
    sec(&o.so, muscl ? 4 * (nf + 1) : 0);
    sec(&o.fric, friction ? 32 * nt : 0);
    o.smem = (int)at;
    return o;
}

template <int kScheme, bool kBlending, int kModel>
const void* run_fn_t(bool pairs)
{
    return pairs ? reinterpret_cast<const void*>(&k_run<kScheme, kBlending, kModel, true>)
                 : reinterpret_cast<const void*>(&k_run<kScheme, kBlending, kModel, false>);
}

template <int kModel>
const void* run_fn_m(const sw2d_handle* h, bool pairs)
{
    const bool bl = h->p.topo == SW2D_TOPO_BLENDING;
    if (h->p.scheme == SW2D_SCHEME_GODUNOV)
        return bl ? run_fn_t<SW2D_SCHEME_GODUNOV, true, kModel>(pairs) : run_fn_t<SW2D_SCHEME_GODUNOV, false, kModel>(pairs);
    return bl ? run_fn_t<SW2D_SCHEME_MUSCL_EVR, true, kModel>(pairs) : run_fn_t<SW2D_SCHEME_MUSCL_EVR, false, kModel>(pairs);
}

const void* run_fn(const sw2d_handle* h, bool pairs)
{
    return h->model == kModelDip ? run_fn_m<kModelDip>(h, pairs) : run_fn_m<kModelSp>(h, pairs);
}

constexpr int64_t kRunCellsMax = 66000;  // above it no tile fits (see the figures at the top)
// Least cells of a tile: fewer take more SMs (and the exchanges more readers) for a shorter chain per CTA.
// us per step with least tiles of 32 / 64 / 96 / 128 cells: MUSCL-EVR 500 cells 7.3 / 7.4 / 8.0 / 8.3, 2,000
// 7.8 / 7.8 / 8.4 / 9.0, 5,000 8.1 / 8.1 / 8.9 / 9.3; Godunov 2,000 5.9 / 5.8 / 6.2 / 6.2, 5,000 6.2 / 5.9 / 6.5 /
// 6.7.  At 64 up to four meshes of 2,000 cells share the chip.
constexpr int kRunTileLeast = 64;
constexpr int kRunSmemMax = 220 * 1024;

void run_free(RunState* r)
{
    for (void* p : r->tile_allocs) cudaFree(p);
    r->tile_allocs.clear();
    for (void* p : r->allocs) cudaFree(p);
    r->allocs.clear();
}

// The tiles and words of a handle's run kernel; RunState.ok tells whether they fit the chip
int run_build(sw2d_handle* h)
{
    RunState* r = h->run = new RunState();
    if (!h->sms && (cudaDeviceGetAttribute(&h->sms, cudaDevAttrMultiProcessorCount, h->device) != cudaSuccess || h->sms <= 0))
        h->sms = 148;
    int coop = 0;
    CK(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, h->device));
    if (!coop) return SW2D_OK;
    const int tile = (int)std::max<int64_t>(kRunTileLeast, (h->nc + h->sms - 1) / h->sms);
    std::string why;
    const int rc = tiles_make(h, h->h_coff, h->h_cint, h->h_lr, h->h_bcell, tile, true, 1, r->tm, r->tile_allocs, why);
    if (rc) return rc;
    const bool muscl = h->p.scheme == SW2D_SCHEME_MUSCL_EVR;
    r->lay = run_layout(r->tm, muscl, h->model == kModelDip, h->p.friction != SW2D_FRICTION_NONE);
    if (r->lay.smem > kRunSmemMax) return SW2D_OK;
    r->pairs = 2 * r->tm.ne_max <= kRunThreads;
    const void* fn = run_fn(h, r->pairs);
    // the limit belongs to the kernel, not to this handle: always the largest
    CK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kRunSmemMax));
    int per_sm = 0;
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kRunThreads, (size_t)r->lay.smem));
    if (per_sm < 1 || (int64_t)per_sm * h->sms < r->tm.ntiles) return SW2D_OK;
    auto alloc = [&](size_t n, ulonglong2** p) -> int {
        void* q = nullptr;
        CK(device_malloc(&q, n * sizeof(ulonglong2)));
        r->allocs.push_back(q);
        CK(cudaMemsetAsync(q, 0, n * sizeof(ulonglong2), h->stream));
        *p = static_cast<ulonglong2*>(q);
        return SW2D_OK;
    };
    int rc2 = alloc(2 * kRunLine * (size_t)r->tm.ntiles, &r->pk_dt);
    if (!rc2) rc2 = alloc(kRunWords * (size_t)h->nc, &r->pk_st);
    if (rc2) return rc2;
    r->ok = true;
    return SW2D_OK;
}

}  // namespace

// Steps of a new handle that its tiles, made on the host, are worth: 0.1 ms at 500 cells, 0.2 at 2,000,
// 1.3 at 20,000, 3.7 at 60,000, against 9 us a step in the run kernel and 21 launched kernel by kernel, or
// the graph that 32 steps by kernels make.  Until then (or sw2d_prepare_steps, or the option set to 1)
// the step's kernels take them.  First call of a new handle, ms, tiles at once / kernels: 500 cells, 1 step
// 0.14 / 0.06, 20 steps 0.31 / 0.42; 2,000 cells, 20 steps 0.48 / 0.44, 31 steps 0.57 / 0.66; 5,000 cells, 31
// steps 0.78 / 0.65, 64 steps 1.1 / 2.1; 20,000 cells, 31 steps 1.7 / 0.7, 64 steps 2.1 / 2.2; 60,000 cells, 64
// steps 5.1 / 2.7, 256 steps 8.9 / 9.0.
int64_t run_worth(const sw2d_handle* h)
{
    return std::max(std::clamp<int64_t>(h->nc / 80, 8, 32), h->nc / 256);
}

int run_ready(sw2d_handle* h, int64_t steps, bool* ready)
{
    *ready = false;
    if (!h->run_kernel || h->model == kModelDdp || h->fused || h->closure || h->result || h->nc > kRunCellsMax) return SW2D_OK;
    if (h->m.lmax || h->m.lmaxb || h->m.flux || h->m.bflux) return SW2D_OK;  // recorded by the step's kernels
    if (!h->run) {
        if (steps >= 0 && !h->run_eager) {
            h->run_asked += std::min(steps, run_worth(h));
            if (h->run_asked < run_worth(h)) return SW2D_OK;
        }
        // no memory for the tiles (or no kernel to hold them): the step's kernels need none of it and serve
        if (run_build(h) != SW2D_OK) {
            cudaGetLastError();
            h->err.clear();
        }
        if (!h->run->ok) run_free(h->run);
    }
    *ready = h->run->ok;
    return SW2D_OK;
}

// Tiles of the calls in progress on each device.  A tile's CTA takes an SM to itself (128 registers x 512
// threads), so that launches whose tiles outnumber the SMs follow one another, where the step's kernels
// of several streams share them.  Measured (B200, calls of 64 steps, us per step over all threads, run
// kernel / step kernels): 2,000 cells (32 tiles) 4 threads 2.1 / 4.7, 8 threads 2.1 / 3.1; 5,000 cells (79
// tiles) 2 threads 8.2 / 9.1, 4 threads 8.2 / 4.9; 20,000 cells (148) 2 threads 10.2 / 10.4, 4 threads 10.3 /
// 6.2; 60,000 cells 2 threads 17.3 / 14.1.  So the run kernel as long as the calls' tiles take two turns
// of the chip at most, and one for the meshes whose step is no longer bound by latency; beyond, all of
// them step by kernels, since each sees the others (4 threads of 20,000 cells 6.6, 8 threads 4.5).  Meshes
// beyond the run kernel's size do not count: beside one of a million cells a mesh of 5,000 takes 10.7 us a
// step and the large one 298; by kernels 161 and 170.  The results are the same bits either way.
constexpr int kRunDevices = 64;
constexpr int64_t kRunCellsOneTurn = 40000;
std::atomic<int> g_run_tiles[kRunDevices];

RunTurn::RunTurn(const sw2d_handle* h, bool ready)
    : device_(h->device), tiles_(ready && h->device < kRunDevices ? h->run->tm.ntiles : 0), run_(ready)
{
    if (!tiles_) return;
    const int before = g_run_tiles[device_].fetch_add(tiles_);
    if (before > 0) run_ = before + tiles_ <= (h->nc > kRunCellsOneTurn ? 1 : 2) * h->sms;
}

RunTurn::~RunTurn()
{
    if (tiles_) g_run_tiles[device_].fetch_sub(tiles_);
}

int run_steps(sw2d_handle* h, int64_t n)
{
    RunState* r = h->run;
    const void* fn = run_fn(h, r->pairs);
    RunArgs a;
    a.pk_dt = r->pk_dt;
    a.pk_st = r->pk_st;
    a.friction = h->p.friction;
    a.head_loss = h->p.singular_head_loss ? 1 : 0;
    a.dissip = h->dissipation;
    a.polls = h->run_polls >= 0 ? h->run_polls : kRunPolls;
    for (int64_t left = n; left > 0;) {
        const int k = (int)std::min<int64_t>(left, kRunSteps);
        if (r->epoch > 0xffffffffu - (unsigned)k - 2u) {  // the epochs start over
            CK(cudaMemsetAsync(r->pk_dt, 0, 2 * kRunLine * (size_t)r->tm.ntiles * sizeof(ulonglong2), h->stream));
            CK(cudaMemsetAsync(r->pk_st, 0, kRunWords * (size_t)h->nc * sizeof(ulonglong2), h->stream));
            r->epoch = 0;
        }
        a.epoch = r->epoch + 1;
        a.n = k;
        r->epoch += (unsigned)k;
        void* args[] = {&h->m, &r->tm, &r->lay, &a};
        CK(cudaLaunchCooperativeKernel(fn, dim3((unsigned)r->tm.ntiles), dim3((unsigned)kRunThreads), args, (size_t)r->lay.smem,
                                       h->stream));
        left -= k;
    }
    return SW2D_OK;
}

void run_retry(sw2d_handle* h)
{
    if (h->run && !h->run->ok) run_release(h);
}

void run_release(sw2d_handle* h)
{
    if (!h->run) return;
    run_free(h->run);
    delete h->run;
    h->run = nullptr;
}

}  // namespace sw2d
