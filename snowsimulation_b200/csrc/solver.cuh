// solver.cuh -- constraint and integration kernels of the substep.
//
// One thread per particle in sorted order (neighbouring threads share cells, so the
// 27-cell gathers hit L1), fused across the particle sets of a stage, grid-stride over
// the set sizes held on the device.  Each neighbor sum keeps the reference's structure
// (per-cell partial sums added to the running total, cells z-y-x, particles ascending)
// and skips only terms that are exactly zero: a term is evaluated when
// d2 < cut-off, which is equivalent to the reference's distance test d < h (resp.
// d < 2r, d <= 2r) because sqrt is correctly rounded and monotone.
#pragma once
#include "common.cuh"
#include "sort.cuh"

namespace snowb {

struct Sets {
    snowb_particle_data sph, dem, bnd;
};
// compact sorted attribute copies (valid for sorted index j < n of the last sort)
struct Sorted {
    float* invm;     // massInv
    float* contrib;  // contrib
    float* lambda;   // lambda (written by the lambda stage)
    float* mass;     // boundary only: mass
};

// Neighbour lists.  The density+lambda pass records, per water or snow particle, every
// candidate that passed the support test (d < h), in traversal order, tagged with its
// set and its cell (0..26).  The PBF and contact passes of the same sort replay the list
// (their supports are d < h or smaller) instead of re-testing ~300 candidates over 81
// cells, keeping the per-cell partial sums.  A particle with more than NLIST_K entries is
// marked overflowed and its consumers traverse the cells as before.
#ifndef SNOWB_NLIST_K
#define SNOWB_NLIST_K 384
#endif
constexpr uint32_t NLIST_K = SNOWB_NLIST_K;
constexpr uint32_t NL_J_MASK = (1u << 25) - 1u;
constexpr uint32_t NL_OVF = 1u << 31;
// The first density pass of a substep lists, per snow particle, its snow candidates within h plus
// a skin of NL_SKIN h (those beyond h marked NL_FAR; link formation skips them).  While the snow
// keeps its sort (DevState::skin_ok) the iterations' density passes take the snow's own sums from
// these lists, each pair put to the exact test, in place of some 300 candidates in 27 cells, and
// list no own neighbours again (NL_OWN_SKIN): the PBF, contact and friction passes read the same
// lists.  The sums are those of the traversal, term by term: the lists are in traversal order, and
// a kept sort keeps every cell's members.  A pair that comes within h has one end that moved more
// than half the skin: the rank pass marks the 27 cells around such a particle, and in marked cells
// the traversal is taken, as it is for a list that a stale cell range went into (NL_STALE: those
// members' own cells may lie elsewhere).
// Density + lambda pass at rest: 832 -> 577 us at 1.18M particles (the frame 22.9 -> 19.6 ms), 144
// -> 112 us at 153.8k (4.08 -> 3.78 ms).  A resting block's particles move 2e-4 m a substep by
// gravity and 99% of them less than 6e-4 m in all, at h = 0.04; skins of 0.02, 0.03 and 0.045 h
// gave 3.78, 3.77, 3.80 and 19.6, 19.8, 20.0 ms.  Where the snow is sorted at every point (the
// melt, batches in which some scene always is) the lists' extra candidates cost about 0.5%.
constexpr float NL_SKIN = 0.02f;
constexpr uint32_t NL_FAR = 1u << 30;        // in an entry
constexpr uint32_t NL_STALE = 1u << 30;      // in a count of the lists with a skin
constexpr uint32_t NL_OWN_SKIN = 1u << 30;   // in a count of the iteration's lists
struct NList {
    uint32_t* e;       // entry k of slot s at e[k * stride + s]: j | cell << 25 | set << 30
    uint32_t* cnt;     // per slot: own | other << 10 | boundary << 20 (| NL_OVF)
    uint32_t stride;   // 2 * capacity: water slots [0, cap), snow slots [cap, 2 cap)
    uint32_t cap;
    const uint32_t *skin_e, *skin_cnt;   // the substep's snow lists with a skin (null: not used)
    const uint32_t* skin_far;            // per cell: the last substep that marked it
};
struct NLWriter {
    uint32_t* e;
    uint32_t stride, slot, n;
    __device__ __forceinline__ void push(uint32_t j, int cell, int set)
    {
        if (n < NLIST_K) e[(size_t)n * stride + slot] = j | ((uint32_t)cell << 25) | ((uint32_t)set << 30);
        ++n;
    }
};
#define CELL27 ((oz + 1) * 9 + (oy + 1) * 3 + (ox + 1))

// ------------------------------------------------------------ per-cell neighbour sums
// pbf_correction (:883-929)
__device__ __forceinline__ float3 pbf_own_cell(const DevParams& P, const SetView& v, float3 p, GCell g, int ox, int oy,
                                               int oz, uint32_t skip, float li, const float* lam_s, const float* lam_o,
                                               const float* con_s, const float* con_o, float dt)
{
    float3 cs = f3(0.f, 0.f, 0.f);
    uint32_t s, e;
    if (v.range(P, g, ox, oy, oz, s, e))
        for (uint32_t j = s; j < e; ++j) {
            if (j == skip) continue;
            float3 dv = sub3(p, v.pos(j));
            float d2 = dot3(dv, dv);
            if (d2 < P.h2_lt) {
                float d = sqrtf(d2);
                float3 gr = G_spiky_in(P, dv, d);
                float lj = v.attr(lam_s, lam_o, j), cj = v.attr(con_s, con_o, j);
                cs = add3(cs, sc3(cj * lam_scorr(P, li + lj, d, dt), gr));
            }
        }
    return cs;
}
__device__ __forceinline__ float3 acc_pbf_own(const DevParams& P, float3 acc, const SetView& v, float3 p, GCell g,
                                              uint32_t skip, float li, const float* lam_s, const float* lam_o,
                                              const float* con_s, const float* con_o, float dt)
{
    FOR27 acc = add3(acc, pbf_own_cell(P, v, p, g, ox, oy, oz, skip, li, lam_s, lam_o, con_s, con_o, dt));
    return acc;
}
// pbf_correction_boundary (:932-979)
__device__ __forceinline__ float3 pbf_bnd_cell(const DevParams& P, const SetView& v, float3 p, GCell g, int ox, int oy,
                                               int oz, float li, const float* lam_s, const float* lam_o, float dt)
{
    float3 cs = f3(0.f, 0.f, 0.f);
    uint32_t s, e;
    if (v.range(P, g, ox, oy, oz, s, e))
        for (uint32_t j = s; j < e; ++j) {
            float3 dv = sub3(p, v.pos(j));
            float d2 = dot3(dv, dv);
            if (d2 < P.h2_lt) {
                float d = sqrtf(d2);
                float3 gr = G_spiky_in(P, dv, d);
                cs = add3(cs, sc3(lam_scorr(P, li + v.attr(lam_s, lam_o, j), d, dt), gr));
            }
        }
    return cs;
}
__device__ __forceinline__ float3 acc_pbf_bnd(const DevParams& P, float3 acc, const SetView& v, float3 p, GCell g,
                                              float li, const float* lam_s, const float* lam_o, float dt)
{
    FOR27 acc = add3(acc, pbf_bnd_cell(P, v, p, g, ox, oy, oz, li, lam_s, lam_o, dt));
    return acc;
}
// pbf_correction_coupling (:982-1034); reference quirks: the self-skip compares indices of
// two different sets, and s_corr is taken as 0 (it reads an uninitialised value times 0)
__device__ __forceinline__ float3 pbf_cpl_cell(const DevParams& P, const SetView& v, float3 p, GCell g, int ox, int oy,
                                               int oz, uint32_t skip, float li, const float* lam_s, const float* lam_o,
                                               float dt)
{
    const bool ref = P.quirks == SNOWB_QUIRKS_REFERENCE;
    float3 cs = f3(0.f, 0.f, 0.f);
    uint32_t s, e;
    if (v.range(P, g, ox, oy, oz, s, e))
        for (uint32_t j = s; j < e; ++j) {
            if (ref && j == skip) continue;
            float3 dv = sub3(p, v.pos(j));
            float d2 = dot3(dv, dv);
            if (d2 < P.r2_le) {
                float d = sqrtf(d2);
                float3 gr = G_poly6(P, dv, d);
                cs = add3(cs, sc3(lam_scorr_cpl(P, li + v.attr(lam_s, lam_o, j), d, dt), gr));
            }
        }
    return cs;
}
__device__ __forceinline__ float3 acc_pbf_cpl(const DevParams& P, float3 acc, const SetView& v, float3 p, GCell g,
                                              uint32_t skip, float li, const float* lam_s, const float* lam_o,
                                              float dt)
{
    FOR27 acc = add3(acc, pbf_cpl_cell(P, v, p, g, ox, oy, oz, skip, li, lam_s, lam_o, dt));
    return acc;
}
// non-penetration: pbd_distance_correction_contrib (:1470-1527, skip) and
// pbd_distance_correction_coupling_contrib (:1648-1705, no skip)
// per-cell partial of acc_contact (cell at offset ox, oy, oz)
__device__ __forceinline__ float3 contact_cell(const DevParams& P, const SetView& v, float3 p, GCell g, int ox, int oy,
                                               int oz, uint32_t skip, float w0, const float* invm_s,
                                               const float* invm_o)
{
    float3 cs = f3(0.f, 0.f, 0.f);
    uint32_t s, e;
    if (v.range_culled(P, g, ox, oy, oz, p, P.r2_cull, s, e))
        for (uint32_t j = s; j < e; ++j) {
            if (j == skip) continue;
            float3 dv = sub3(p, v.pos(j));
            float d2 = dot3(dv, dv);
            if (d2 < P.r2_lt) {
                float d = sqrtf(d2);
                float w1 = v.attr(invm_s, invm_o, j);
                float ws = w0 + w1;
                float C = d - P.two_r;
                float3 n = div3(dv, d + P.pbd_eps);
                cs = add3(cs, sc3(((-w0) * (1.f / ws)) * C, n));
            }
        }
    return cs;
}
__device__ __forceinline__ float3 acc_contact(const DevParams& P, float3 acc, const SetView& v, float3 p, GCell g,
                                              uint32_t skip, float w0, const float* invm_s, const float* invm_o)
{
    FOR27 acc = add3(acc, contact_cell(P, v, p, g, ox, oy, oz, skip, w0, invm_s, invm_o));
    return acc;
}

// Replays of a recorded neighbour segment [k0, k1) of slot `slot`, per-cell partial sums
// kept (entries of one cell are contiguous and in traversal order).
struct Seg {
    const uint32_t* e;
    uint32_t stride, slot, k0, k1;
    __device__ __forceinline__ uint32_t at(uint32_t k) const { return __ldg(e + (size_t)k * stride + slot); }
};
__device__ __forceinline__ float3 seg_pbf_own(const DevParams& P, float3 acc, const Seg& S, const SetView& v,
                                              float3 p, float li, const float* lam_s, const float* lam_o,
                                              const float* con_s, const float* con_o, float dt)
{
    float3 cs = f3(0.f, 0.f, 0.f);
    uint32_t cur = 0xFFu;
    for (uint32_t k = S.k0; k < S.k1; ++k) {
        const uint32_t en = S.at(k), j = en & NL_J_MASK, cell = (en >> 25) & 31u;
        if (cell != cur) { if (cur != 0xFFu) acc = add3(acc, cs); cs = f3(0.f, 0.f, 0.f); cur = cell; }
        float3 dv = sub3(p, v.pos(j));
        const float d2 = dot3(dv, dv);
        if (!(d2 < P.h2_lt)) continue;   // lists with a skin hold more
        float d = sqrtf(d2);
        float3 gr = G_spiky_in(P, dv, d);
        float lj = v.attr(lam_s, lam_o, j), cj = v.attr(con_s, con_o, j);
        cs = add3(cs, sc3(cj * lam_scorr(P, li + lj, d, dt), gr));
    }
    if (cur != 0xFFu) acc = add3(acc, cs);
    return acc;
}
__device__ __forceinline__ float3 seg_pbf_bnd(const DevParams& P, float3 acc, const Seg& S, const SetView& v,
                                              float3 p, float li, const float* lam_s, const float* lam_o, float dt)
{
    float3 cs = f3(0.f, 0.f, 0.f);
    uint32_t cur = 0xFFu;
    for (uint32_t k = S.k0; k < S.k1; ++k) {
        const uint32_t en = S.at(k), j = en & NL_J_MASK, cell = (en >> 25) & 31u;
        if (cell != cur) { if (cur != 0xFFu) acc = add3(acc, cs); cs = f3(0.f, 0.f, 0.f); cur = cell; }
        float3 dv = sub3(p, v.pos(j));
        float d = sqrtf(dot3(dv, dv));   // a recorded candidate: d < h
        float3 gr = G_spiky_in(P, dv, d);
        cs = add3(cs, sc3(lam_scorr(P, li + v.attr(lam_s, lam_o, j), d, dt), gr));
    }
    if (cur != 0xFFu) acc = add3(acc, cs);
    return acc;
}
__device__ __forceinline__ float3 seg_pbf_cpl(const DevParams& P, float3 acc, const Seg& S, const SetView& v,
                                              float3 p, uint32_t skip, float li, const float* lam_s,
                                              const float* lam_o, float dt)
{
    const bool ref = P.quirks == SNOWB_QUIRKS_REFERENCE;
    float3 cs = f3(0.f, 0.f, 0.f);
    uint32_t cur = 0xFFu;
    for (uint32_t k = S.k0; k < S.k1; ++k) {
        const uint32_t en = S.at(k), j = en & NL_J_MASK, cell = (en >> 25) & 31u;
        if (cell != cur) { if (cur != 0xFFu) acc = add3(acc, cs); cs = f3(0.f, 0.f, 0.f); cur = cell; }
        if (ref && j == skip) continue;
        float3 dv = sub3(p, v.pos(j));
        float d2 = dot3(dv, dv);
        if (d2 < P.r2_le) {
            float d = sqrtf(d2);
            float3 gr = G_poly6(P, dv, d);
            cs = add3(cs, sc3(lam_scorr_cpl(P, li + v.attr(lam_s, lam_o, j), d, dt), gr));
        }
    }
    if (cur != 0xFFu) acc = add3(acc, cs);
    return acc;
}
__device__ __forceinline__ float3 seg_contact(const DevParams& P, float3 acc, const Seg& S, const SetView& v,
                                              float3 p, float w0, const float* invm_s, const float* invm_o)
{
    // entries taken four (then two) at a time: their squared distances screened with packed
    // arithmetic against the slightly larger r2_cull, the exact test and the term for those
    // that pass; per-cell partials closed where the cell changes, entry by entry in order
    const P2 pp = bcast2(p);
    float3 cs = f3(0.f, 0.f, 0.f);
    uint32_t cur = 0xFFu;
    auto one = [&](uint32_t j, uint32_t cell, float3 q, bool pass) {
        if (cell != cur) { if (cur != 0xFFu) acc = add3(acc, cs); cs = f3(0.f, 0.f, 0.f); cur = cell; }
        if (!pass) return;
        float3 dv = sub3(p, q);
        float d2 = dot3(dv, dv);
        if (d2 < P.r2_lt) {
            float d = sqrtf(d2);
            float w1 = v.attr(invm_s, invm_o, j);
            float ws = w0 + w1;
            float C = d - P.two_r;
            float3 n = div3(dv, d + P.pbd_eps);
            cs = add3(cs, sc3(((-w0) * (1.f / ws)) * C, n));
        }
    };
    uint32_t k = S.k0;
    for (; k + 3 < S.k1; k += 4) {
        const uint32_t e0 = S.at(k), e1 = S.at(k + 1), e2 = S.at(k + 2), e3 = S.at(k + 3);
        const uint32_t j0 = e0 & NL_J_MASK, j1 = e1 & NL_J_MASK, j2 = e2 & NL_J_MASK, j3 = e3 & NL_J_MASK;
        const float3 q0 = v.pos(j0), q1 = v.pos(j1), q2 = v.pos(j2), q3 = v.pos(j3);
        const float2 da = d2_pair(pp, make_float4(q0.x, q0.y, q0.z, 0.f), make_float4(q1.x, q1.y, q1.z, 0.f));
        const float2 db = d2_pair(pp, make_float4(q2.x, q2.y, q2.z, 0.f), make_float4(q3.x, q3.y, q3.z, 0.f));
        one(j0, (e0 >> 25) & 31u, q0, da.x < P.r2_cull);
        one(j1, (e1 >> 25) & 31u, q1, da.y < P.r2_cull);
        one(j2, (e2 >> 25) & 31u, q2, db.x < P.r2_cull);
        one(j3, (e3 >> 25) & 31u, q3, db.y < P.r2_cull);
    }
    for (; k + 1 < S.k1; k += 2) {
        const uint32_t e0 = S.at(k), e1 = S.at(k + 1);
        const uint32_t j0 = e0 & NL_J_MASK, j1 = e1 & NL_J_MASK;
        const float3 q0 = v.pos(j0), q1 = v.pos(j1);
        const float2 dd = d2_pair(pp, make_float4(q0.x, q0.y, q0.z, 0.f), make_float4(q1.x, q1.y, q1.z, 0.f));
        one(j0, (e0 >> 25) & 31u, q0, dd.x < P.r2_cull);
        one(j1, (e1 >> 25) & 31u, q1, dd.y < P.r2_cull);
    }
    if (k < S.k1) {
        const uint32_t e0 = S.at(k), j0 = e0 & NL_J_MASK;
        one(j0, (e0 >> 25) & 31u, v.pos(j0), true);
    }
    if (cur != 0xFFu) acc = add3(acc, cs);
    return acc;
}
// segments of slot `slot`; false when the list overflowed (fall back to traversal)
__device__ __forceinline__ bool segments(const NList& L, uint32_t slot, Seg& own, Seg& oth, Seg& bnd)
{
    const uint32_t c = L.cnt[slot];
    if (c & NL_OVF) return false;
    const uint32_t a = c & 1023u, b = (c >> 10) & 1023u, d = (c >> 20) & 1023u;
    own = Seg{L.e, L.stride, slot, 0u, a};
    if (c & NL_OWN_SKIN) own = Seg{L.skin_e, L.stride, slot, 0u, L.skin_cnt[slot] & 1023u};
    oth = Seg{L.e, L.stride, slot, a, a + b};
    bnd = Seg{L.e, L.stride, slot, a + b, a + b + d};
    return true;
}

// ======================================================================== density
// Density and W-weighted sums with an optional lambda gradient sum in the same pass.
// compute_snow_{sph,dem_sph,boundary}_density_d (:2219-2528) and, when LAMBDA is set,
// compute_snow_{sph,dem_sph,boundary}_lambdas_d (:2598-2898): lambda needs the particle's
// own C and neighbour positions only, so both come out of one traversal.  Each quantity
// keeps its own per-cell accumulation in the reference's loop order.
// one candidate of acc_WG
template <bool LAMBDA, bool SKIN = false>
__device__ __forceinline__ void wg_term(const DevParams& P, float& cs, float& cg, float4 q, float3 p, uint32_t j,
                                        bool vol, int mode, float m_self, float m_j, NLWriter* wr, int cell, int set)
{
    float3 dv = sub3(p, xyz(q));
    float d2 = dot3(dv, dv);
    if (d2 < P.h2_lt) {
        if (wr) wr->push(j, cell, set);
        float d = sqrtf(d2);   // d < h: d2 passed the exact support test
        float w = vol ? P.rho0 * q.w : q.w;
        cs += w * W_poly6_in(P, d);
        if (LAMBDA) {
            float sc;
            if (mode == 0) sc = P.inv_rho0;
            else {
                float m = mode == 1 ? m_self : m_j;
                sc = P.inv_rho0 * ((P.rho0 * q.w) / m);
            }
            float3 gc = sc3(sc, G_spiky_in(P, dv, d));
            cg += dot3(gc, gc);
        }
    } else if (SKIN && d2 < P.s2) {
        wr->push(j, cell, 1);   // NL_FAR
    }
}
template <bool LAMBDA, bool SKIN = false>
__device__ __forceinline__ void acc_WG(const DevParams& P, float& rho, float& gs, const SetView& v, float3 p,
                                       const Nbhd& nb, uint32_t skip, bool vol, int mode, float m_self,
                                       const float* mass_s, const float* mass_o, NLWriter* wr = nullptr, int set = 0,
                                       float* dpart = nullptr, uint32_t* dmask = nullptr, bool* stale = nullptr)
{
    const P2 pp = bcast2(p);
    const float cull = SKIN ? P.s2_cull : P.h2_cull;
    FOR27 {
        float cs = 0.f, cg = 0.f;
        uint32_t s, e;
        if (v.range_nb(nb, ox, oy, oz, s, e)) {
            const int cell = CELL27;
            if (SKIN) *stale |= !(s < v.n && __ldg(v.gh + s) == nb.hash(ox, oy, oz));
            if (e <= v.n) {
                // current entries only: the compact sorted copies.  Candidates are screened
                // two at a time with packed arithmetic; ptxas may contract its multiply-adds,
                // so the screen is a superset test against the slightly larger h2_cull, and
                // every candidate that passes goes through the exact scalar test and terms.
                uint32_t j = s;
                for (; j + 1 < e; j += 2) {
                    const float4 q0 = __ldg(v.p4 + j), q1 = __ldg(v.p4 + j + 1);
                    const float2 dd = d2_pair(pp, q0, q1);
                    if (dd.x < cull && j != skip) {
                        const float mj = (LAMBDA && mode == 2) ? __ldg(mass_s + j) : 0.f;
                        wg_term<LAMBDA, SKIN>(P, cs, cg, q0, p, j, vol, mode, m_self, mj, wr, cell, set);
                    }
                    if (dd.y < cull && j + 1 != skip) {
                        const float mj = (LAMBDA && mode == 2) ? __ldg(mass_s + j + 1) : 0.f;
                        wg_term<LAMBDA, SKIN>(P, cs, cg, q1, p, j + 1, vol, mode, m_self, mj, wr, cell, set);
                    }
                }
                if (j < e && j != skip) {
                    const float mj = (LAMBDA && mode == 2) ? __ldg(mass_s + j) : 0.f;
                    wg_term<LAMBDA, SKIN>(P, cs, cg, __ldg(v.p4 + j), p, j, vol, mode, m_self, mj, wr, cell, set);
                }
            } else {
                for (uint32_t j = s; j < e; ++j) {
                    if (j == skip) continue;
                    const float mj = (LAMBDA && mode == 2) ? v.attr(mass_s, mass_o, j) : 0.f;
                    wg_term<LAMBDA, SKIN>(P, cs, cg, v.pw(j), p, j, vol, mode, m_self, mj, wr, cell, set);
                }
            }
        }
        // dpart: keep the cell's density partial aside instead of adding it now (a partial
        // of +0, which adds nothing, is not kept)
        if (dpart) {
            if (cs != 0.f) { dpart[CELL27] = cs; *dmask |= 1u << CELL27; }
        } else {
            rho += cs;
        }
        if (LAMBDA) gs += cg;
    }
}
// the same sums for a snow particle and its own set from its list with a skin, entries taken four
// at a time
__device__ __forceinline__ void acc_skin(const DevParams& P, float& rho, float& gs, const NList& L, uint32_t slot,
                                         uint32_t n, const SetView& v, float3 p)
{
    const Seg S{L.skin_e, L.stride, slot, 0u, n};
    float cs = 0.f, cg = 0.f;
    uint32_t cur = 0u;
    for (uint32_t k = 0u; k < n; k += 4u) {
        uint32_t en[4];
        float4 q[4];
#pragma unroll
        for (uint32_t u = 0u; u < 4u; ++u) en[u] = S.at(umin32(k + u, n - 1u));
#pragma unroll
        for (uint32_t u = 0u; u < 4u; ++u) q[u] = v.pw(en[u] & NL_J_MASK);
#pragma unroll
        for (uint32_t u = 0u; u < 4u; ++u) {
            if (k + u >= n) break;
            const uint32_t cell = (en[u] >> 25) & 31u;
            if (cell != cur) {
                rho += cs; gs += cg;
                cs = cg = 0.f;
                cur = cell;
            }
            wg_term<true>(P, cs, cg, q[u], p, en[u] & NL_J_MASK, false, 0, 0.f, 0.f, nullptr, 0, 0);
        }
    }
    rho += cs;
    gs += cg;
}
// Sums over the boundary set of every boundary particle (own term included): the opening
// terms of its density and lambda sums, the same in every pass of a call since the boundary
// does not move.  The call's first pass over the boundary forms them, the later ones read them
// (by sorted index; DevState::base_ready).
struct BndBase {
    float *rho, *gs;
};
// which of the water (bit 0) and snow (bit 1) sets have an entry, stale ones included, in the
// 27 cells around g; the loads are independent
__device__ __forceinline__ uint32_t occupied27(const DevParams& P, GCell g, const SetView& vs, const SetView& vd)
{
    uint32_t w = 0, s = 0;
#pragma unroll
    for (int oz = -1; oz <= 1; ++oz)
#pragma unroll
        for (int oy = -1; oy <= 1; ++oy)
#pragma unroll
            for (int ox = -1; ox <= 1; ++ox) {
                const uint32_t h = grid_hash(P, g, ox, oy, oz);
                w |= ~__ldg(vs.cs + h);     // SNOWB_EMPTY is all ones
                s |= ~__ldg(vd.cs + h);
            }
    return (w ? 1u : 0u) | (s ? 2u : 0u);
}
// The 27 cell ranges are loaded first (independent loads), then the occupied cells walked: one
// layer of boundary particles fills about 9 of them.
__device__ __forceinline__ void boundary_base(const DevParams& P, const SetView& vb, const Sets& X, const Sorted& sb,
                                              uint32_t i, uint32_t o, float3 p, GCell g, bool ready, const BndBase& base,
                                              float& rho, float& gs)
{
    if (ready) {
        rho = base.rho[i];
        gs = base.gs[i];
        return;
    }
    uint32_t s[27], e[27], m = 0;
#pragma unroll
    for (int c = 0; c < 27; ++c) {
        const uint32_t h = grid_hash(P, g, c % 3 - 1, (c / 3) % 3 - 1, c / 9 - 1);
        s[c] = __ldg(vb.cs + h);
        e[c] = __ldg(vb.ce + h);
        if (s[c] != SNOWB_EMPTY) m |= 1u << c;
    }
    rho = (P.rho0 * X.bnd.volume[o]) * P.W0;
    gs = 0.f;
    while (m) {
        const int c = __ffs(m) - 1;
        m &= m - 1u;
        float cs = 0.f, cg = 0.f;
        for (uint32_t j = s[c]; j < e[c]; ++j)
            if (j != i)
                wg_term<true>(P, cs, cg, vb.pw(j), p, j, true, 2, 0.f, vb.attr(sb.mass, X.bnd.mass, j), nullptr, 0, 0);
        rho += cs;
        gs += cg;
    }
    base.rho[i] = rho;
    base.gs[i] = gs;
}

template <bool LAMBDA>
// with_bnd = 0: water and snow only (the boundary particles' density, C and lambda are then
// left as they were; a later density+lambda pass of the substep rewrites them).  The water
// and snow sums take the boundary's terms either way, through its compact sorted copies.
__global__ void __launch_bounds__(256) k_density(DevParams P, DevState* __restrict__ S, SetView vs, SetView vd,
                                                 SetView vb, Sets X, Sorted ss, Sorted sd, Sorted sb, NList L,
                                                 int with_bnd, BndBase base, float4* __restrict__ skin_p4)
{
    wait_prior();
    const uint32_t ns = S->n_sph, nd = S->n_dem, nb = S->n_b, nbt = with_bnd ? nb : 0u;
    vs.n = ns; vd.n = nd; vb.n = nb;
    const bool ready = S->base_ready != 0u;
    const float3 z = f3(0.f, 0.f, 0.f);
    const bool skin = LAMBDA && S->skin_ok != 0u;
    const uint32_t epoch = S->epoch;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        if (LAMBDA) {
            S->far_move = 0u;   // the lists are new
            if (skin) ++S->skin_passes;
        } else {
            S->skin_ok = 1u;
        }
    }
    GRID_LOOP(t, ns + nd + nbt) {
        float rho, gs = dot3(z, z);
        const snowb_particle_data* D;
        float* lam_s;
        uint32_t o, i;
        if (t < ns + nd) {
            const bool w = t < ns;
            i = w ? t : t - ns;
            const SetView& own = w ? vs : vd;
            const SetView& oth = w ? vd : vs;
            D = w ? &X.sph : &X.dem;
            lam_s = w ? ss.lambda : sd.lambda;
            o = own.gi[i];
            float3 p = xyz(own.p4[i]); GCell g = grid_pos(P, p, own.scene(i));
            const Nbhd nb = make_nbhd(P, g, p, LAMBDA || w ? P.h2_cull : P.s2_cull);
            rho = D->mass[o] * P.W0;
            NLWriter wr{L.e, L.stride, (w ? 0u : L.cap) + i, 0u};
            // the density+lambda pass lists all three sets for the PBF and contact passes; the
            // substep's first density pass lists the snow-snow candidates for link formation
            NLWriter* pw = (LAMBDA || !w) ? &wr : nullptr;
            const uint32_t listed = skin && !w && L.skin_far[nb.hash(0, 0, 0)] != epoch ? L.skin_cnt[wr.slot] : NL_OVF;
            const bool use_skin = !(listed & (NL_OVF | NL_STALE));
            bool stale = false;
            if (use_skin) {
                acc_skin(P, rho, gs, L, wr.slot, listed & 1023u, own, p);
            } else if (LAMBDA || w) {
                if (skin && !w) atomicAdd(&S->skin_walks, 1u);
                acc_WG<LAMBDA>(P, rho, gs, own, p, nb, i, false, 0, 0.f, nullptr, nullptr, pw, 0);
            } else {
                acc_WG<LAMBDA, true>(P, rho, gs, own, p, nb, i, false, 0, 0.f, nullptr, nullptr, pw, 0, nullptr, nullptr,
                                     &stale);
                skin_p4[i] = own.p4[i];
            }
            const uint32_t n_own = wr.n;
            if (!LAMBDA) pw = nullptr;
            acc_WG<LAMBDA>(P, rho, gs, oth, p, nb, SNOWB_UMAX, false, 0, 0.f, nullptr, nullptr, pw, 1);
            const uint32_t n_oth = wr.n - n_own;
            acc_WG<LAMBDA>(P, rho, gs, vb, p, nb, SNOWB_UMAX, true, 1, D->mass[o], nullptr, nullptr, pw, 2);
            if (LAMBDA) {
                const uint32_t n_bnd = wr.n - n_own - n_oth;
                L.cnt[wr.slot] = wr.n > NLIST_K ? NL_OVF : (n_own | (n_oth << 10) | (n_bnd << 20) | (use_skin ? NL_OWN_SKIN : 0u));
                if (wr.n > NLIST_K) atomicAdd(&S->n_nl_ovf, 1u);
            } else if (!w) {
                L.cnt[wr.slot] = n_own > NLIST_K ? NL_OVF : (n_own | (stale ? NL_STALE : 0u));
            }
        } else {
            // boundary: density sums the sets in the order (b, snow, water), lambda (b, water,
            // snow); the sums over the boundary itself open both, and most boundary particles
            // have no other neighbour
            i = t - ns - nd; o = vb.gi[i];
            float3 p = xyz(vb.p4[i]); GCell g = grid_pos(P, p, vb.scene(i));
            boundary_base(P, vb, X, sb, i, o, p, g, ready, base, rho, gs);
            const uint32_t near = occupied27(P, g, vs, vd);
            if (LAMBDA && near) {
                // one traversal per set for both sums: water first (its lambda terms come
                // before the snow's), its density partials kept aside and added after the
                // snow's, cell by cell in order -- the two orders of the separate passes
                const Nbhd nb = make_nbhd(P, g, p, P.h2_cull);
                float wpart[27];
                uint32_t wmask = 0;
                if (near & 1u)
                    acc_WG<true>(P, rho, gs, vs, p, nb, SNOWB_UMAX, false, 0, 0.f, nullptr, nullptr, nullptr, 0, wpart,
                                 &wmask);
                if (near & 2u) acc_WG<true>(P, rho, gs, vd, p, nb, SNOWB_UMAX, false, 0, 0.f, nullptr, nullptr);
                while (wmask) {
                    const int c = __ffs(wmask) - 1;
                    wmask &= wmask - 1u;
                    rho += wpart[c];
                }
            } else if (near) {
                const Nbhd nb = make_nbhd(P, g, p, P.h2_cull);
                float unused = 0.f;
                acc_WG<false>(P, rho, unused, vd, p, nb, SNOWB_UMAX, false, 0, 0.f, nullptr, nullptr);
                acc_WG<false>(P, rho, unused, vs, p, nb, SNOWB_UMAX, false, 0, 0.f, nullptr, nullptr);
            }
            D = &X.bnd; lam_s = sb.lambda;
        }
        D->density[o] = rho;
        float c = (rho / P.rho0) - 1.f;
        c = c > 0.f ? c : 0.f;
        D->C[o] = c;
        if (LAMBDA) {
            float lam = (-c) / (gs + P.eps);
            D->lambda[o] = lam;
            lam_s[i] = lam;
        }
    }
}

constexpr uint32_t DENSITY_WARP_MAX = 40000;
// The same pass with one warp per particle, for sets too small to fill the GPU with threads
// (DENSITY_WARP_MAX): one thread walking 81 cells is a chain of some 160 dependent loads, 80 to
// 120 us whatever the set's size.  Lane c < 27 takes cell c of each set: it marks the
// candidates within the support, the counts' prefix over the lanes places its list entries in
// traversal order, it forms the cell's partial sums in index order, and the partials are added
// in cell order with shuffles -- the operations of the one-thread form in the same order.  A
// warp takes 32 boundary particles: each lane tests whether its particle has water or snow
// around it, and the few that do are taken by the whole warp one after another.
// Density + lambda, both forms, us a launch: 67 -> 18 at 208 particles, 105 -> 33 at 5,096, 119
// -> 55 at 16,380.  Whole frames, one thread against one warp each: 2.66 against 2.03 ms at
// 15.8k particles, 3.24 against 3.03 at 35.7k, 3.32 against 3.80 at 58k; the line lies between.
struct CellHits {
    uint32_t s, e, n, mask;     // range, candidates within the support, which of the first 32
};
__device__ __forceinline__ CellHits cell_hits(const DevParams& P, const SetView& v, float3 p, uint32_t h, bool live,
                                              uint32_t skip)
{
    CellHits c{0u, 0u, 0u, 0u};
    if (!live) return c;
    c.s = __ldg(v.cs + h);
    c.e = __ldg(v.ce + h);
    if (c.s == SNOWB_EMPTY) c.e = c.s = 0u;
    for (uint32_t j0 = c.s; j0 < c.e; j0 += 4u) {
        float d2[4];
#pragma unroll
        for (uint32_t u = 0; u < 4u; ++u) {
            const float3 dv = sub3(p, v.pos(umin32(j0 + u, c.e - 1u)));
            d2[u] = dot3(dv, dv);
        }
#pragma unroll
        for (uint32_t u = 0; u < 4u; ++u)
            if (j0 + u < c.e && d2[u] < P.h2_lt && j0 + u != skip) {
                ++c.n;
                if (j0 + u - c.s < 32u) c.mask |= 1u << (j0 + u - c.s);
            }
    }
    return c;
}
// the cell's partial sums and, with e set, its list entries from position k on
template <bool LAMBDA>
__device__ __forceinline__ void cell_sums(const DevParams& P, const SetView& v, float3 p, const CellHits& c,
                                          uint32_t skip, bool vol, int mode, float m_self, NLWriter* wr, int cell,
                                          int set, float& cs, float& cg)
{
    cs = cg = 0.f;
    uint32_t m = c.mask;
    while (m) {
        const uint32_t j = c.s + (uint32_t)__ffs(m) - 1u;
        m &= m - 1u;
        wg_term<LAMBDA>(P, cs, cg, v.pw(j), p, j, vol, mode, m_self, 0.f, wr, cell, set);
    }
    for (uint32_t j = c.s + 32u; j < c.e; ++j)
        if (j != skip) wg_term<LAMBDA>(P, cs, cg, v.pw(j), p, j, vol, mode, m_self, 0.f, wr, cell, set);
}
// adds the cells' partials in cell order (partials are never negative and the totals never -0,
// so a cell whose partials are both +0 is left out)
__device__ __forceinline__ void warp_ordered_add(float& a, float& b, float pa, float pb)
{
    uint32_t m = __ballot_sync(0xffffffffu, (__float_as_uint(pa) | __float_as_uint(pb)) != 0u);
    while (m) {
        const int k = __ffs(m) - 1;
        m &= m - 1u;
        a += __shfl_sync(0xffffffffu, pa, k);
        b += __shfl_sync(0xffffffffu, pb, k);
    }
}
template <bool LAMBDA>
__global__ void __launch_bounds__(256) k_density_warp(DevParams P, DevState* __restrict__ S, SetView vs, SetView vd,
                                                      SetView vb, Sets X, Sorted ss, Sorted sd, Sorted sb, NList L,
                                                      int with_bnd, BndBase base)
{
    wait_prior();
    const uint32_t ns = S->n_sph, nd = S->n_dem, nb = S->n_b, nbg = with_bnd ? (nb + 31u) / 32u : 0u;
    vs.n = ns; vd.n = nd; vb.n = nb;
    const bool ready = S->base_ready != 0u;
    const uint32_t lane = threadIdx.x & 31u, full = 0xffffffffu;
    const bool cl = lane < 27u;
    const int ox = (int)(lane % 3u) - 1, oy = (int)((lane / 3u) % 3u) - 1, oz = (int)(lane / 9u) - 1;
    if (LAMBDA && blockIdx.x == 0 && threadIdx.x == 0) S->far_move = 0u;   // the lists are new
    const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < ns + nd + nbg; t += nwarps) {
        if (t < ns + nd) {
            const bool w = t < ns;
            const uint32_t i = w ? t : t - ns;
            const SetView& own = w ? vs : vd;
            const SetView& oth = w ? vd : vs;
            const snowb_particle_data& D = w ? X.sph : X.dem;
            const uint32_t o = own.gi[i];
            const float3 p = xyz(own.p4[i]);
            const uint32_t h = grid_hash(P, grid_pos(P, p, own.scene(i)), ox, oy, oz);
            const float mass = D.mass[o];
            const CellHits c0 = cell_hits(P, own, p, h, cl, i), c1 = cell_hits(P, oth, p, h, cl, SNOWB_UMAX),
                           c2 = cell_hits(P, vb, p, h, cl, SNOWB_UMAX);
            // list positions: the lambda pass lists all three sets, the first density pass the
            // snow-snow candidates
            const bool l0 = LAMBDA || !w;
            const uint32_t slot = (w ? 0u : L.cap) + i;
            const uint32_t i0 = l0 ? warp_incl_scan(c0.n) : 0u, n0 = __shfl_sync(full, i0, 31);
            const uint32_t i1 = LAMBDA ? warp_incl_scan(c1.n) : 0u, n1 = __shfl_sync(full, i1, 31);
            const uint32_t i2 = LAMBDA ? warp_incl_scan(c2.n) : 0u, n2 = __shfl_sync(full, i2, 31);
            float rho = mass * P.W0, gs = 0.f, pa, pb;
            NLWriter wr{L.e, L.stride, slot, i0 - c0.n};
            cell_sums<LAMBDA>(P, own, p, c0, i, false, 0, 0.f, l0 ? &wr : nullptr, (int)lane, 0, pa, pb);
            warp_ordered_add(rho, gs, pa, pb);
            wr.n = n0 + i1 - c1.n;
            cell_sums<LAMBDA>(P, oth, p, c1, SNOWB_UMAX, false, 0, 0.f, LAMBDA ? &wr : nullptr, (int)lane, 1, pa, pb);
            warp_ordered_add(rho, gs, pa, pb);
            wr.n = n0 + n1 + i2 - c2.n;
            cell_sums<LAMBDA>(P, vb, p, c2, SNOWB_UMAX, true, 1, mass, LAMBDA ? &wr : nullptr, (int)lane, 2, pa, pb);
            warp_ordered_add(rho, gs, pa, pb);
            if (lane == 0) {
                const uint32_t n = n0 + n1 + n2;
                if (l0) {
                    L.cnt[slot] = n > NLIST_K ? NL_OVF : (n0 | (n1 << 10) | (n2 << 20));
                    if (LAMBDA && n > NLIST_K) atomicAdd(&S->n_nl_ovf, 1u);
                }
                float c = (rho / P.rho0) - 1.f;
                c = c > 0.f ? c : 0.f;
                D.density[o] = rho;
                D.C[o] = c;
                if (LAMBDA) {
                    const float lam = (-c) / (gs + P.eps);
                    D.lambda[o] = lam;
                    (w ? ss.lambda : sd.lambda)[i] = lam;
                }
            }
        } else {
            // a warp's boundary particles lie nbg apart: those with neighbours come in patches
            const uint32_t i = (t - ns - nd) + lane * nbg;
            const bool live = i < nb;
            float3 p = f3(0.f, 0.f, 0.f);
            GCell g{};
            float rho = 0.f, gs = 0.f;
            uint32_t near = 0;
            if (live) {
                p = xyz(vb.p4[i]);
                g = grid_pos(P, p, vb.scene(i));
                boundary_base(P, vb, X, sb, i, vb.gi[i], p, g, ready, base, rho, gs);
                near = occupied27(P, g, vs, vd);
            }
            uint32_t m = __ballot_sync(full, near != 0u);
            while (m) {
                const int k = __ffs(m) - 1;
                m &= m - 1u;
                const float3 q = f3(__shfl_sync(full, p.x, k), __shfl_sync(full, p.y, k), __shfl_sync(full, p.z, k));
                const GCell gk{__shfl_sync(full, g.x, k), __shfl_sync(full, g.y, k), __shfl_sync(full, g.z, k),
                               __shfl_sync(full, g.bx, k), __shfl_sync(full, g.bz, k)};
                const uint32_t h = grid_hash(P, gk, ox, oy, oz);
                float wa, wb, sa, sb2, r = __shfl_sync(full, rho, k), s = __shfl_sync(full, gs, k), none = 0.f;
                cell_sums<LAMBDA>(P, vs, q, cell_hits(P, vs, q, h, cl, SNOWB_UMAX), SNOWB_UMAX, false, 0, 0.f, nullptr,
                                  0, 0, wa, wb);
                cell_sums<LAMBDA>(P, vd, q, cell_hits(P, vd, q, h, cl, SNOWB_UMAX), SNOWB_UMAX, false, 0, 0.f, nullptr,
                                  0, 0, sa, sb2);
                warp_ordered_add(r, none, sa, 0.f);     // density: snow, then water
                warp_ordered_add(r, none, wa, 0.f);
                warp_ordered_add(s, none, wb, 0.f);     // lambda: water, then snow
                warp_ordered_add(s, none, sb2, 0.f);
                if (lane == (uint32_t)k) { rho = r; gs = s; }
            }
            if (live) {
                const uint32_t o = vb.gi[i];
                float c = (rho / P.rho0) - 1.f;
                c = c > 0.f ? c : 0.f;
                X.bnd.density[o] = rho;
                X.bnd.C[o] = c;
                if (LAMBDA) {
                    const float lam = (-c) / (gs + P.eps);
                    X.bnd.lambda[o] = lam;
                    sb.lambda[i] = lam;
                }
            }
        }
    }
}

// ------------------------------------------------- ordered per-cell sums by a warp (small sets)
// The sums of a one-thread neighbour loop -- per cell a partial sum in index order, the partials
// added in cell order -- over the entries j != skip of set v within d2 < cut of p, for sets too
// small to fill the GPU with threads.  Lane c < 27 scans cell c (h: its hash; live: the lane takes
// part), four entries in flight; the counts' prefix over the lanes lists those accepted in
// traversal order, 32 of them at a time are evaluated side by side (terms(j, out) writes one
// addend for each of NA sums), and lane a < NA adds the addends of sum a in order, a partial
// closed where the cell changes.  acc carries on from the sets before.
constexpr uint32_t CELL_LIST = 96;
struct CellBuf {
    uint32_t e[CELL_LIST];           // j | cell << 25
    float t[32 * 3];
};
template <int NA, class F>
__device__ __forceinline__ void warp_cell_sums(const SetView& v, float3 p, uint32_t h, bool live, uint32_t skip, float cut,
                                               CellBuf& W, float& acc, F&& terms)
{
    static_assert(NA == 1 || NA == 3, "addends of a neighbour");
    const uint32_t lane = threadIdx.x & 31u, full = 0xffffffffu;
    uint32_t s = 0, e = 0;
    if (live) {
        s = __ldg(v.cs + h);
        e = __ldg(v.ce + h);
        if (s == SNOWB_EMPTY || e < s) s = e = 0u;
    }
    auto hit = [&](uint32_t j) {
        const float3 r = sub3(p, v.pos(j));
        return dot3(r, r) < cut && j != skip;
    };
    uint32_t n = 0, mask = 0;   // accepted, and which of the first 32 entries
    for (uint32_t k = 0; k < e - s; k += 4u)
#pragma unroll
        for (uint32_t u = 0; u < 4u; ++u)
            if (hit(umin32(s + k + u, e - 1u)) && s + k + u < e) {
                ++n;
                if (k + u < 32u) mask |= 1u << (k + u);
            }
    if (!__any_sync(full, n != 0u)) return;
    const uint32_t first = warp_incl_scan(n) - n, total = __shfl_sync(full, first + n, 31);
    float cs = 0.f;
    uint32_t cur = 0xFFu;
    for (uint32_t w0 = 0; w0 < total; w0 += CELL_LIST) {
        __syncwarp();
        uint32_t at = first, m = mask;
        while (m) {
            const uint32_t j = s + (uint32_t)__ffs(m) - 1u;
            m &= m - 1u;
            if (at - w0 < CELL_LIST) W.e[at - w0] = j | lane << 25;
            ++at;
        }
        for (uint32_t j = s + 32u; j < e; ++j)
            if (hit(j)) {
                if (at - w0 < CELL_LIST) W.e[at - w0] = j | lane << 25;
                ++at;
            }
        __syncwarp();
        const uint32_t held = umin32(total - w0, CELL_LIST);
        for (uint32_t b = 0; b < held; b += 32u) {
            if (b + lane < held) terms(W.e[b + lane] & NL_J_MASK, W.t + lane * NA);
            __syncwarp();
            if (lane < (uint32_t)NA)
                for (uint32_t k = 0; k < umin32(held - b, 32u); ++k) {
                    const uint32_t cell = W.e[b + k] >> 25;
                    if (cell != cur) {
                        if (cur != 0xFFu) acc += cs;
                        cs = 0.f;
                        cur = cell;
                    }
                    cs += W.t[k * NA + lane];
                }
            __syncwarp();
        }
    }
    acc += cs;
}
__device__ __forceinline__ float3 warp_vec3(float acc)
{
    return f3(__shfl_sync(0xffffffffu, acc, 0), __shfl_sync(0xffffffffu, acc, 1), __shfl_sync(0xffffffffu, acc, 2));
}
// lane c < 27: hash of cell c around g
__device__ __forceinline__ uint32_t lane_cell(const DevParams& P, GCell g)
{
    const uint32_t c = threadIdx.x & 31u;
    return c < 27u ? grid_hash(P, g, (int)(c % 3u) - 1, (int)((c / 3u) % 3u) - 1, (int)(c / 9u) - 1) : 0u;
}
#define WARP_LOOP(t, n) \
    for (uint32_t t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < (n); t += (gridDim.x * blockDim.x) >> 5)
constexpr uint32_t SMALL_TPB = 128;
// Where the lines lie, by whole frames (ms, one thread against one warp per particle):
// contacts (by snow particles): 1.651 / 1.538 at 4.8k, 1.848 / 1.753 at 8.6k, 2.046 / 2.073 at
// 14.1k and 2.362 / 2.509 at 23.1k at rest; in the melt, where lists are long, 4.431 / 3.912 at
// 8.6k and 4.432 / 3.952 at 14.1k.  Heat: fixed quirks (27 cells of both sets) 3.238 / 3.061 at
// 24.8k and 3.798 / 3.646 at 35.7k; reference quirks (the own cell) even at 5k, 2.362 / 2.447 at
// 24.8k.  Friction: 1.651 / 1.606 at 4.8k; beyond FRICTION_WARP_MAX the one-thread form's list
// replay is the faster one (2.046 / 2.133 at 14.1k), the traversal it falls back to when the lists
// do not hold is the slower one up to about twice that (eight substeps of 13.8k: 6.20 / 5.57),
// so up to FRICTION_BOTH_MAX both are launched and one returns at once.
constexpr uint32_t CONTACT_WARP_MAX = 16000;
constexpr uint32_t HEAT_WARP_MAX = 40000, HEAT_WARP_MAX_REF = 6000;
constexpr uint32_t FRICTION_WARP_MAX = 9000, FRICTION_BOTH_MAX = 24000;

// ======================================================== applying a correction
// apply_correction (:1342-1380) for one particle: new and predicted position q + sor * corr,
// the correction cleared, the set marked when the particle left its cell.  Passes that
// finish a particle's correction apply it themselves where k_apply would come next; limits
// carry the reference's launch sizes (Q12).
__device__ __forceinline__ uint32_t launch_limit(const DevParams& P, uint32_t n0, uint32_t n)
{
    return P.quirks == SNOWB_QUIRKS_REFERENCE ? umin32(coverage(n0), n) : n;
}
__device__ __forceinline__ float3 apply_one(const DevParams& P, const snowb_particle_data& D, const SortTrack& T,
                                            uint32_t o, float3 q, float3 corr, uint32_t scene)
{
    const float3 np = add3(q, sc3(P.sor, corr));
    st3(D.new_positions, o, np);
    st3(D.predict_positions, o, np);
    st3(D.correction, o, f3(0.f, 0.f, 0.f));
    if (T.key) track_move(P, T, o, np, scene);
    return np;
}

// ==================================================== PBF + water-side contact corrections
// compute_pbf_sph_correction (:3070-3184) fused with compute_sph_dem_distance_correction
// (:2061-2110) and compute_sph_sph_distance_correction (:2164-2217) for water, and
// compute_pbf_new_dem_correction (:3187-3304) for snow.  Each water particle adds its
// terms to its correction in the reference's kernel order.
struct StageFlags {
    int correct_dem, sph_sph, interlink, step_sph, step_dem;
};
// Water sets up to this size run the water terms one warp per particle (k_pbf_water_warp):
// with few particles one thread each leaves the GPU idle while each thread walks its
// neighbours; above it, threads fill the GPU and the warp form's extra work would cost more.
constexpr uint32_t PBF_WARP_MAX_WATER = 65536;
// apply: as in k_pbf_water_warp, for the water particles this pass takes
__global__ void __launch_bounds__(256) k_pbf(DevParams P, DevState* __restrict__ S, SetView vs, SetView vd,
                                             SetView vb, Sets X, Sorted ss, Sorted sd, Sorted sb, float dt,
                                             StageFlags F, NList L, int apply, SortTrack ts)
{
    wait_prior();
    const uint32_t ns = S->n_sph, nd = S->n_dem, nb = S->n_b;
    vs.n = ns; vd.n = nd; vb.n = nb;
    const bool ref = P.quirks == SNOWB_QUIRKS_REFERENCE;
    // the density + lambda pass before this one has formed the boundary sums
    if (blockIdx.x == 0 && threadIdx.x == 0) S->base_ready = 1u;
    // up to PBF_WARP_MAX_WATER water particles the water terms come from k_pbf_water_warp;
    // the snow particles keep the thread mapping t = ns + i of the reference's launch (its
    // float atomics, Q3, follow it)
    GRID_LOOP(t, ns + nd) {
        if (t < ns) {
            if (ns <= PBF_WARP_MAX_WATER) continue;   // k_pbf_water_warp has them
            const uint32_t i = t, o = vs.gi[i];
            float3 p = xyz(vs.p4[i]); GCell g = grid_pos(P, p, vs.scene(i));
            const float li = ss.lambda[i];
            float3 c = f3(0.f, 0.f, 0.f);
            Seg so, sx, sbn;
            const bool lst = segments(L, i, so, sx, sbn);
            if (lst) {
                c = seg_pbf_own(P, c, so, vs, p, li, ss.lambda, X.sph.lambda, ss.contrib, X.sph.contrib, dt);
                c = seg_pbf_cpl(P, c, sx, vd, p, i, li, sd.lambda, X.dem.lambda, dt);
                c = seg_pbf_bnd(P, c, sbn, vb, p, li, sb.lambda, X.bnd.lambda, dt);
            } else {
                c = acc_pbf_own(P, c, vs, p, g, i, li, ss.lambda, X.sph.lambda, ss.contrib, X.sph.contrib, dt);
                c = acc_pbf_cpl(P, c, vd, p, g, i, li, sd.lambda, X.dem.lambda, dt);
                c = acc_pbf_bnd(P, c, vb, p, g, li, sb.lambda, X.bnd.lambda, dt);
            }
            c = sc3(P.inv_rho0, c);
            const float ci = X.sph.contrib[o];
            c = sc3(ci, c);
            if (nan3(c)) c = f3(0.f, 0.f, 0.f);
            float3 acc = add3(ldv3(X.sph.correction, o), c);
            const float3 z = f3(0.f, 0.f, 0.f);
            const float w0 = X.sph.massInv[o];
            // the contact terms are scaled by (1 - contrib): with contrib == 1 they add a
            // zero to a correction that is never -0 here, which leaves it unchanged
            if (F.correct_dem && ci != 1.f) {     // compute_sph_dem_distance_correction
                float3 d = lst ? seg_contact(P, z, sx, vd, p, w0, sd.invm, X.dem.massInv)
                               : acc_contact(P, z, vd, p, g, SNOWB_UMAX, w0, sd.invm, X.dem.massInv);
                d = sc3(1.f - ci, d);
                if (nan3(d)) d = z;
                acc = add3(acc, sc3(P.k_stretch, d));
            }
            if (F.sph_sph && ci != 1.f) {         // compute_sph_sph_distance_correction
                // pbd_sph_sph_distance_correction (:1586-1646) acts only for contrib <= 0.99
                float3 d = ci <= 0.99f ? acc_contact(P, z, vs, p, g, i, w0, ss.invm, X.sph.massInv) : add3(z, z);
                d = sc3(1.f - ci, d);
                if (nan3(d)) d = z;
                acc = add3(acc, d);
            }
            if (apply && i < launch_limit(P, S->n0_sph, ns)) apply_one(P, X.sph, ts, o, p, acc, vs.scene(i));
            else st3(X.sph.correction, o, acc);
        } else {
            const uint32_t i = t - ns;
            const uint32_t o = ref ? vs.gi[i] : vd.gi[i];   // Q3: SPH grid_index in the reference
            // the snow PBF correction is scaled by (1 - contrib): with contrib == 1 it adds a
            // zero (a NaN or infinity becomes zero too) to the +0 the last apply left
            if (X.dem.contrib[o] == 1.f) continue;
            float3 p = xyz(vd.p4[i]); GCell g = grid_pos(P, p, vd.scene(i));
            const float li = X.dem.lambda[o];
            float3 c = f3(0.f, 0.f, 0.f);
            Seg so, sx, sbn;
            if (segments(L, L.cap + i, so, sx, sbn)) {
                c = seg_pbf_cpl(P, c, sx, vs, p, i, li, ss.lambda, X.sph.lambda, dt);
                if (nan3(c)) c = f3(0.f, 0.f, 0.f);
                c = seg_pbf_own(P, c, so, vd, p, li, sd.lambda, X.dem.lambda, sd.contrib, X.dem.contrib, dt);
                if (nan3(c)) c = f3(0.f, 0.f, 0.f);
                c = seg_pbf_bnd(P, c, sbn, vb, p, li, sb.lambda, X.bnd.lambda, dt);
            } else {
                c = acc_pbf_cpl(P, c, vs, p, g, i, li, ss.lambda, X.sph.lambda, dt);
                if (nan3(c)) c = f3(0.f, 0.f, 0.f);
                c = acc_pbf_own(P, c, vd, p, g, i, li, sd.lambda, X.dem.lambda, sd.contrib, X.dem.contrib, dt);
                if (nan3(c)) c = f3(0.f, 0.f, 0.f);
                c = acc_pbf_bnd(P, c, vb, p, g, li, sb.lambda, X.bnd.lambda, dt);
            }
            if (nan3(c)) c = f3(0.f, 0.f, 0.f);
            c = sc3(P.inv_rho0, c);
            c = sc3(1.f - X.dem.contrib[o], c);
            if (nan3(c)) c = f3(0.f, 0.f, 0.f);
            float* q = reinterpret_cast<float*>(X.dem.correction) + 3ull * o;
            if (ref) {   // targets can repeat in the reference's indexing
                atomicAdd(q, c.x); atomicAdd(q + 1, c.y); atomicAdd(q + 2, c.z);
            } else {
                q[0] += c.x; q[1] += c.y; q[2] += c.z;
            }
        }
    }
    (void)nb;
}

// ============================================================ snow-side corrections
// delete_record (:4624-4658): remove the link from both particles' slot lists.
__device__ __forceinline__ void delete_record(const snowb_particle_data& D, uint32_t M, uint32_t i0, uint32_t i1)
{
    for (uint32_t s = i0 * M; s < (i0 + 1) * M; ++s)
        if (atomicCAS(D.connect_record + s, i1, SNOWB_UMAX) == i1) { atomicExch(D.connect_length + s, 0.f); break; }
    for (uint32_t s = i1 * M; s < (i1 + 1) * M; ++s)
        if (atomicCAS(D.connect_record + s, i0, SNOWB_UMAX) == i0) { atomicExch(D.connect_length + s, 0.f); break; }
}
// compute_dem_sph_distance_correction (:2112-2162) and compute_dem_distance_correction
// (:1765-1834) for snow particle o, added to its correction in the reference's kernel
// order (after the PBF pass; the interlink terms of k_link_sum follow).  SUMS: the two
// contact sums are kept apart instead: sums[2o] the water contact (scaled by k_stretch *
// contrib; +0 without correct_dem), sums[2o+1] the snow-then-boundary contact (scaled by
// contrib).  That pass reads no correction, so it can run beside the snow PBF pass, and
// k_link_apply adds both to the correction after the PBF term, in this order.
template <bool SUMS>
__global__ void __launch_bounds__(256) k_dem_corr(DevParams P, const DevState* __restrict__ S, SetView vs, SetView vd,
                                                  SetView vb, Sets X, Sorted ss, Sorted sd, Sorted sb, StageFlags F,
                                                  NList L, float4* __restrict__ sums)
{
    wait_prior();
    const uint32_t ns = S->n_sph, nd = S->n_dem, nb = S->n_b;
    vs.n = ns; vd.n = nd; vb.n = nb;
    const float3 z = f3(0.f, 0.f, 0.f);
    GRID_LOOP(i, nd) {
        const uint32_t o = vd.gi[i];
        float3 p = xyz(vd.p4[i]); GCell g = grid_pos(P, p, vd.scene(i));
        const float w0 = X.dem.massInv[o], ci = X.dem.contrib[o];
        float3 acc = SUMS ? z : ldv3(X.dem.correction, o);
        Seg so, sx, sbn;
        const bool lst = segments(L, L.cap + i, so, sx, sbn);
        if (F.correct_dem) {
            float3 d = lst ? seg_contact(P, z, sx, vs, p, w0, ss.invm, X.sph.massInv)
                           : acc_contact(P, z, vs, p, g, SNOWB_UMAX, w0, ss.invm, X.sph.massInv);
            d = sc3(P.k_stretch * ci, d);
            if (nan3(d)) d = z;
            if (SUMS) sums[2 * (size_t)o] = make_float4(d.x, d.y, d.z, 0.f);
            else acc = add3(acc, d);
        } else if (SUMS) {
            sums[2 * (size_t)o] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        {
            float3 d = lst ? seg_contact(P, z, so, vd, p, w0, sd.invm, X.dem.massInv)
                           : acc_contact(P, z, vd, p, g, i, w0, sd.invm, X.dem.massInv);
            d = lst ? seg_contact(P, d, sbn, vb, p, w0, sb.invm, X.bnd.massInv)
                    : acc_contact(P, d, vb, p, g, SNOWB_UMAX, w0, sb.invm, X.bnd.massInv);
            d = sc3(ci, d);
            if (nan3(d)) d = z;
            if (SUMS) sums[2 * (size_t)o + 1] = make_float4(d.x, d.y, d.z, 0.f);
            else st3(X.dem.correction, o, add3(acc, d));
        }
    }
    (void)ns; (void)nb;
}
// the same with one warp per particle, by traversal (small sets; 28 -> 18 us at 5,096 particles)
template <bool SUMS>
__global__ void __launch_bounds__(SMALL_TPB) k_dem_corr_warp(DevParams P, const DevState* __restrict__ S, SetView vs,
                                                             SetView vd, SetView vb, Sets X, Sorted ss, Sorted sd,
                                                             Sorted sb, StageFlags F, float4* __restrict__ sums)
{
    wait_prior();
    __shared__ CellBuf bufs[SMALL_TPB / 32];
    CellBuf& W = bufs[threadIdx.x >> 5];
    const uint32_t nd = S->n_dem, lane = threadIdx.x & 31u;
    vs.n = S->n_sph; vd.n = nd; vb.n = S->n_b;
    const float3 z = f3(0.f, 0.f, 0.f);
    WARP_LOOP(i, nd) {
        const uint32_t o = vd.gi[i];
        const float3 p = xyz(vd.p4[i]);
        const uint32_t h = lane_cell(P, grid_pos(P, p, vd.scene(i)));
        const float w0 = X.dem.massInv[o], ci = X.dem.contrib[o];
        auto contact = [&](const SetView& v, uint32_t skip, const float* invm_s, const float* invm_o, float& acc) {
            warp_cell_sums<3>(v, p, h, lane < 27u, skip, P.r2_lt, W, acc, [&](uint32_t j, float* out) {
                const float3 dv = sub3(p, v.pos(j));
                const float d = sqrtf(dot3(dv, dv));
                const float ws = w0 + v.attr(invm_s, invm_o, j), C = d - P.two_r;
                const float3 t = sc3(((-w0) * (1.f / ws)) * C, div3(dv, d + P.pbd_eps));
                out[0] = t.x; out[1] = t.y; out[2] = t.z;
            });
        };
        float3 dw = z;
        if (F.correct_dem) {
            float acc = 0.f;
            contact(vs, SNOWB_UMAX, ss.invm, X.sph.massInv, acc);
            dw = sc3(P.k_stretch * ci, warp_vec3(acc));
            if (nan3(dw)) dw = z;
        }
        float acc = 0.f;
        contact(vd, i, sd.invm, X.dem.massInv, acc);
        contact(vb, SNOWB_UMAX, sb.invm, X.bnd.massInv, acc);
        float3 d = sc3(ci, warp_vec3(acc));
        if (nan3(d)) d = z;
        if (lane == 0u) {
            if (SUMS) {
                sums[2 * (size_t)o] = make_float4(dw.x, dw.y, dw.z, 0.f);
                sums[2 * (size_t)o + 1] = make_float4(d.x, d.y, d.z, 0.f);
            } else {
                float3 c = ldv3(X.dem.correction, o);
                if (F.correct_dem) c = add3(c, dw);
                st3(X.dem.correction, o, add3(c, d));
            }
        }
    }
}
// solve_snow_interlink_constraint_d (:4742-4765) with compute_interlink_correction
// (:4661-4739), in two passes.  Each particle's slots are summed in slot order, which one
// thread per particle walking its slots does with about 11 dependent link terms in a row
// (a record load, the partner's position, a square root and four divisions each), so the
// pass waited on memory.  Here k_link_terms evaluates every slot's term with one thread per
// slot, all independent, and k_link_sum adds each particle's terms in slot order to its
// correction, after the contact terms as in the reference.  Both ends of a link hold the
// same length and see the same distance, so whichever end breaks it first (delete_record),
// neither adds a correction; a slot whose record a partner has deleted adds nothing, and a
// zero term added to the sum leaves it unchanged (the sum of nonzero terms is never -0), so
// the result does not depend on which thread deletes first.
__device__ __forceinline__ float3 link_term(const DevParams& P, const snowb_particle_data& D, uint32_t i0, uint32_t i1,
                                           float L, uint32_t n)
{
    const float3 z = f3(0.f, 0.f, 0.f);
    if (i0 == i1 || i0 >= n || i1 >= n || L == 0.f) return z;
    const float3 v = sub3(ldv3(D.predict_positions, i0), ldv3(D.predict_positions, i1));
    const float dist = len3(v);
    if (dist > P.brk * L || dist > P.h) { delete_record(D, P.maxc, i0, i1); return z; }
    const float w0 = D.massInv[i0], w1 = D.massInv[i1];
    const float ws = w0 + w1, C = dist - L;
    const float3 n3 = div3(v, dist + P.pbd_eps);
    const float3 r = sc3(((P.k_ref * -w0) * (1.f / ws)) * C, n3);
    // len3(r) > 1 without the square root: sqrtf is monotone and correctly rounded, and the
    // smallest float whose root rounds above 1 is 1 + 2^-22, so the test is d2 > 1 + 2^-23
    if (dot3(r, r) > 0x1.000002p+0f || nan3(r) || inf3(r)) return z;
    return r;
}
// term of slot s: (x, y, z, 1) for a filled slot, w = 0 for an empty one
__global__ void __launch_bounds__(256) k_link_terms(DevParams P, const DevState* __restrict__ S,
                                                    snowb_particle_data dem, float4* __restrict__ terms)
{
    wait_prior();
    const uint32_t nd = S->n_dem, M = P.maxc;
    // Plain (cached) loads: a record that a partner deletes during the pass is one whose term
    // is zero at both ends, so whether this thread still sees it, or sees its length already
    // zeroed, the term is the same zero.
    GRID_LOOP(s, nd * M) {
        const uint32_t j = dem.connect_record[s];
        float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
        if (j != SNOWB_UMAX) {
            const float3 r = link_term(P, dem, s / M, j, dem.connect_length[s], nd);
            t = make_float4(r.x, r.y, r.z, 1.f);
        }
        terms[s] = t;
    }
}
__global__ void __launch_bounds__(256) k_link_sum(DevParams P, const DevState* __restrict__ S,
                                                  snowb_particle_data dem, const float4* __restrict__ terms)
{
    wait_prior();
    const uint32_t nd = S->n_dem, M = P.maxc;
    const float3 z = f3(0.f, 0.f, 0.f);
    GRID_LOOP(o, nd) {
        float3 d = z;
        for (uint32_t s = M * o; s < M * (o + 1); ++s) {
            const float4 t = __ldg(terms + s);
            if (t.w != 0.f) d = add3(d, xyz(t));
        }
        if (nan3(d)) d = z;
        st3(dem.correction, o, add3(ldv3(dem.correction, o), d));
    }
}

// The friction pass replays the density+lambda pass's neighbour lists when they still hold
// every contact: the friction sort point kept the snow set's sort (same cells, same order)
// and no snow particle moved more than FR_LIST_MOVE since the lists were built.  A pair
// within 2r now was then within 2r + 2 FR_LIST_MOVE = 0.028 m < h of each other (r = 0.01,
// h = 0.04; the bound is checked against the parameters on the host).
constexpr float FR_LIST_MOVE = 0.004f;

// k_link_sum and the snow part of k_apply in one pass over the sorted snow particles (the
// order k_apply takes them in; o = grid_index[i] runs over the same particles as k_link_sum's
// o): the contact sums and the interlink terms join the correction, which is applied to the
// particles within the launch limit and kept for the others, as k_apply leaves it.
__global__ void __launch_bounds__(256) k_link_apply(DevParams P, DevState* __restrict__ S, SetView vd,
                                                    snowb_particle_data dem, const float4* __restrict__ terms,
                                                    const float4* __restrict__ sums, int correct_dem, int apply,
                                                    SortTrack td)
{
    wait_prior();
    const uint32_t nd = S->n_dem, M = P.maxc;
    const uint32_t ld = apply ? launch_limit(P, S->n0_dem, nd) : 0u;
    const float3 z = f3(0.f, 0.f, 0.f);
    GRID_LOOP(i, nd) {
        const uint32_t o = vd.gi[i];
        float3 d = z;
        for (uint32_t s = M * o; s < M * (o + 1); ++s) {
            const float4 t = __ldg(terms + s);
            if (t.w != 0.f) d = add3(d, xyz(t));
        }
        if (nan3(d)) d = z;
        float3 acc = ldv3(dem.correction, o);
        if (sums) {
            if (correct_dem) acc = add3(acc, xyz(__ldg(sums + 2 * (size_t)o)));
            acc = add3(acc, xyz(__ldg(sums + 2 * (size_t)o + 1)));
        }
        acc = add3(acc, d);
        if (i < ld) {
            const float3 q = xyz(vd.p4[i]);
            const float3 np = apply_one(P, dem, td, o, q, acc, vd.scene(i));
            const float3 dp = sub3(np, q);
            if (!(dot3(dp, dp) <= FR_LIST_MOVE * FR_LIST_MOVE)) S->far_move = 1u;
        } else {
            st3(dem.correction, o, acc);
        }
    }
}


// ======================================================================= apply
// apply_correction (:1342-1380); limits carry the reference's launch sizes (Q12).
// ts, td: a particle that leaves its cell marks its set for a full sort at the next sort
// point (key null: not tracked).
__global__ void k_apply(DevParams P, DevState* __restrict__ S, SetView vs, SetView vd, Sets X, int do_sph,
                        int do_dem, SortTrack ts, SortTrack td)
{
    wait_prior();
    const uint32_t ls = do_sph ? launch_limit(P, S->n0_sph, S->n_sph) : 0u;
    const uint32_t ld = do_dem ? launch_limit(P, S->n0_dem, S->n_dem) : 0u;
    GRID_LOOP(t, ls + ld) {
        const bool w = t < ls;
        const uint32_t i = w ? t : t - ls;
        const SetView& v = w ? vs : vd;
        const snowb_particle_data& D = w ? X.sph : X.dem;
        const uint32_t o = v.gi[i];
        const float3 q = xyz(v.p4[i]);
        const float3 np = apply_one(P, D, w ? ts : td, o, q, ldv3(D.correction, o), v.scene(i));
        if (!w) {
            const float3 dp = sub3(np, q);
            if (!(dot3(dp, dp) <= FR_LIST_MOVE * FR_LIST_MOVE)) S->far_move = 1u;
        }
    }
}

// ==================================================================== friction
// compute_friction_correction (:1989-2059) with pbd_friction_correction{,_boundary}
// (:1836-1987); overwrites the correction.
__device__ __forceinline__ float3 friction_term(const DevParams& P, float3 dx, float w0, float w1, float d, float3 v)
{
    float ws = w0 + w1;
    float3 n = div3(v, d + P.pbd_eps);
    float pen = P.two_r - d;
    float3 dxt = sub3(dx, sc3(dot3(dx, n), n));
    float thr = P.mu_s * pen;
    float len = len3(dxt);
    if (len3(dxt) > thr) {
        float c = fminf((P.mu_k * pen) / (len + 0.000001f), 1.f);
        dxt = sc3(c, dxt);
    }
    return sc3(-(w0 / ws), dxt);
}
// Two phases per set: the candidate scan records the contacts (d <= 2r, a few per
// particle) with their cell in shared memory, then the friction terms are evaluated over
// the record with the per-cell partial sums closed where the cell changes (cells without
// contacts add +0 in the traversal, which leaves the sum unchanged).  The lanes of a warp
// then evaluate the costly term together instead of once per lane that found a contact.
// More than FR_K contacts fall back to the single traversal.
constexpr uint32_t FR_K = 16;
// lists: the replay of the neighbour lists is allowed (see FR_LIST_MOVE); each particle
// then takes its snow and boundary contacts from its list entries, in list order, instead
// of traversing the cells (same contacts, same order: the list holds every candidate with
// d < h in traversal order with its cell).
// APPLY: the friction correction is applied at once (the snow part of k_apply, whose
// position it reads is this pass's p: new and predicted positions, a zero correction, the
// moved mark of the set), without k_apply's far-move flag, which the next density+lambda
// pass clears before any friction pass reads it.
// only_lists: k_friction_warp takes the pass unless the lists hold.
__device__ __forceinline__ bool friction_lists(const DevState* S, int lists)
{
    return lists && S->resort[1] == 0u && S->far_move == 0u;
}
template <bool APPLY>
__global__ void __launch_bounds__(256) k_friction(DevParams P, const DevState* __restrict__ S, SetView vd, SetView vb,
                                                  Sets X, Sorted sd, Sorted sb, NList L, int lists, int only_lists,
                                                  SortTrack td)
{
    wait_prior();
    __shared__ uint32_t rec_sh[FR_K * 256];
    uint32_t* const rec = rec_sh + threadIdx.x;     // entry k at rec[k * blockDim.x]
    const uint32_t bd = blockDim.x;
    vd.n = S->n_dem; vb.n = S->n_b;
    const uint32_t ld = launch_limit(P, S->n0_dem, S->n_dem);
    const bool list_ok = friction_lists(S, lists);
    if (only_lists && !list_ok) return;
    GRID_LOOP(i, ld) {
        const uint32_t o = vd.gi[i];
        float3 p = xyz(vd.p4[i]);
        float3 op0 = ldv3(X.dem.positions, o);
        const float w0 = X.dem.massInv[o];
        Seg so, sx, sbn;
        const bool use_list = list_ok && segments(L, L.cap + i, so, sx, sbn);
        const Nbhd nb = use_list ? Nbhd{} : make_nbhd(P, grid_pos(P, p, vd.scene(i)), p, P.r2_cull);
        float3 c = f3(0.f, 0.f, 0.f);
        // snow-snow contacts (current entries screened two at a time with packed arithmetic
        // against the slightly larger r2_cull, then the exact scalar test, as in the density
        // pass)
        const P2 pp = bcast2(p);
        uint32_t n = 0;
        auto record = [&](uint32_t j, uint32_t cell) {
            if (n < FR_K) rec[n * bd] = j | (cell << 25);
            ++n;
        };
        if (use_list) {
            for (uint32_t k = so.k0; k < so.k1; ++k) {
                const uint32_t en = so.at(k), j = en & NL_J_MASK;
                const float3 v = sub3(p, vd.pos(j));
                if (dot3(v, v) < P.r2_le) record(j, (en >> 25) & 31u);
            }
        } else FOR27 {
            uint32_t s, e;
            if (vd.range_nb(nb, ox, oy, oz, s, e)) {
                const uint32_t cell = (uint32_t)CELL27;
                if (e <= vd.n) {
                    uint32_t j = s;
                    for (; j + 1 < e; j += 2) {
                        const float4 q0 = __ldg(vd.p4 + j), q1 = __ldg(vd.p4 + j + 1);
                        const float2 dd = d2_pair(pp, q0, q1);
                        if (dd.x < P.r2_cull && j != i) {
                            const float3 v = sub3(p, xyz(q0));
                            if (dot3(v, v) < P.r2_le) record(j, cell);
                        }
                        if (dd.y < P.r2_cull && j + 1 != i) {
                            const float3 v = sub3(p, xyz(q1));
                            if (dot3(v, v) < P.r2_le) record(j + 1, cell);
                        }
                    }
                    if (j < e && j != i) {
                        const float3 v = sub3(p, vd.pos(j));
                        if (dot3(v, v) < P.r2_le) record(j, cell);
                    }
                } else {
                    for (uint32_t j = s; j < e; ++j) {
                        if (j == i) continue;
                        const float3 v = sub3(p, vd.pos(j));
                        if (dot3(v, v) < P.r2_le) record(j, cell);
                    }
                }
            }
        }
        if (n <= FR_K) {
            float3 cs = f3(0.f, 0.f, 0.f);
            uint32_t cur = 0xFFu;
            for (uint32_t k = 0; k < n; ++k) {
                const uint32_t en = rec[k * bd], j = en & NL_J_MASK, cell = en >> 25;
                if (cell != cur) { if (cur != 0xFFu) c = add3(c, cs); cs = f3(0.f, 0.f, 0.f); cur = cell; }
                const float3 pp1 = vd.pos(j);
                const float3 v = sub3(p, pp1);
                const float d2 = dot3(v, v);
                const float3 op1 = ldv3(X.dem.positions, vd.gi[j]);
                const float3 dx = add3(sub3(p, op0), sub3(pp1, op1));
                cs = add3(cs, friction_term(P, dx, w0, vd.attr(sd.invm, X.dem.massInv, j), sqrtf(d2), v));
            }
            if (cur != 0xFFu) c = add3(c, cs);
        } else {   // more contacts than the record holds: the traversal evaluates them
            const Nbhd nbf = use_list ? make_nbhd(P, grid_pos(P, p, vd.scene(i)), p, P.r2_cull) : nb;
            FOR27 {
                float3 cs = f3(0.f, 0.f, 0.f);
                uint32_t s, e;
                if (vd.range_nb(nbf, ox, oy, oz, s, e))
                    for (uint32_t j = s; j < e; ++j) {
                        if (j == i) continue;
                        float3 pp1 = vd.pos(j);
                        float3 v = sub3(p, pp1);
                        float d2 = dot3(v, v);
                        if (d2 < P.r2_le) {
                            const uint32_t oj = vd.gi[j];
                            float3 op1 = ldv3(X.dem.positions, oj);
                            float3 dx = add3(sub3(p, op0), sub3(pp1, op1));
                            cs = add3(cs, friction_term(P, dx, w0, vd.attr(sd.invm, X.dem.massInv, j), sqrtf(d2), v));
                        }
                    }
                c = add3(c, cs);
            }
        }
        // snow-boundary contacts
        n = 0;
        if (use_list) {
            for (uint32_t k = sbn.k0; k < sbn.k1; ++k) {
                const uint32_t en = sbn.at(k), j = en & NL_J_MASK;
                const float3 v = sub3(p, vb.pos(j));
                if (dot3(v, v) < P.r2_le) record(j, (en >> 25) & 31u);
            }
        } else FOR27 {
            uint32_t s, e;
            if (vb.range_nb(nb, ox, oy, oz, s, e)) {
                const uint32_t cell = (uint32_t)CELL27;
                if (e <= vb.n) {
                    uint32_t j = s;
                    for (; j + 1 < e; j += 2) {
                        const float4 q0 = __ldg(vb.p4 + j), q1 = __ldg(vb.p4 + j + 1);
                        const float2 dd = d2_pair(pp, q0, q1);
                        if (dd.x < P.r2_cull) {
                            const float3 v = sub3(p, xyz(q0));
                            if (dot3(v, v) < P.r2_le) record(j, cell);
                        }
                        if (dd.y < P.r2_cull) {
                            const float3 v = sub3(p, xyz(q1));
                            if (dot3(v, v) < P.r2_le) record(j + 1, cell);
                        }
                    }
                    if (j < e) {
                        const float3 v = sub3(p, vb.pos(j));
                        if (dot3(v, v) < P.r2_le) record(j, cell);
                    }
                } else {
                    for (uint32_t j = s; j < e; ++j) {
                        const float3 v = sub3(p, vb.pos(j));
                        if (dot3(v, v) < P.r2_le) record(j, cell);
                    }
                }
            }
        }
        const float3 dx0 = sub3(p, op0);
        if (n <= FR_K) {
            float3 cs = f3(0.f, 0.f, 0.f);
            uint32_t cur = 0xFFu;
            for (uint32_t k = 0; k < n; ++k) {
                const uint32_t en = rec[k * bd], j = en & NL_J_MASK, cell = en >> 25;
                if (cell != cur) { if (cur != 0xFFu) c = add3(c, cs); cs = f3(0.f, 0.f, 0.f); cur = cell; }
                const float3 v = sub3(p, vb.pos(j));
                const float d2 = dot3(v, v);
                cs = add3(cs, friction_term(P, dx0, w0, vb.attr(sb.invm, X.bnd.massInv, j), sqrtf(d2), v));
            }
            if (cur != 0xFFu) c = add3(c, cs);
        } else {
            const Nbhd nbf = use_list ? make_nbhd(P, grid_pos(P, p, vd.scene(i)), p, P.r2_cull) : nb;
            FOR27 {
                float3 cs = f3(0.f, 0.f, 0.f);
                uint32_t s, e;
                if (vb.range_nb(nbf, ox, oy, oz, s, e))
                    for (uint32_t j = s; j < e; ++j) {
                        float3 v = sub3(p, vb.pos(j));
                        float d2 = dot3(v, v);
                        if (d2 < P.r2_le)
                            cs = add3(cs, friction_term(P, dx0, w0, vb.attr(sb.invm, X.bnd.massInv, j), sqrtf(d2), v));
                    }
                c = add3(c, cs);
            }
        }
        if (nan3(c)) c = f3(0.f, 0.f, 0.f);
        if (APPLY) {
            apply_one(P, X.dem, td, o, p, c, vd.scene(i));
        } else {
            st3(X.dem.correction, o, c);
        }
    }
}

// the same with one warp per particle, by traversal (at 16,380 particles, where the one-thread
// form mostly walked the cells, 55 -> 29 us)
template <bool APPLY>
__global__ void __launch_bounds__(SMALL_TPB) k_friction_warp(DevParams P, const DevState* __restrict__ S, SetView vd,
                                                             SetView vb, Sets X, Sorted sd, Sorted sb, int lists,
                                                             int unless_lists, SortTrack td)
{
    wait_prior();
    if (unless_lists && friction_lists(S, lists)) return;   // k_friction replays them
    __shared__ CellBuf bufs[SMALL_TPB / 32];
    CellBuf& W = bufs[threadIdx.x >> 5];
    vd.n = S->n_dem; vb.n = S->n_b;
    const uint32_t ld = launch_limit(P, S->n0_dem, S->n_dem), lane = threadIdx.x & 31u;
    WARP_LOOP(i, ld) {
        const uint32_t o = vd.gi[i];
        const float3 p = xyz(vd.p4[i]);
        const uint32_t h = lane_cell(P, grid_pos(P, p, vd.scene(i)));
        const float3 op0 = ldv3(X.dem.positions, o), dx0 = sub3(p, op0);
        const float w0 = X.dem.massInv[o];
        float acc = 0.f;
        warp_cell_sums<3>(vd, p, h, lane < 27u, i, P.r2_le, W, acc, [&](uint32_t j, float* out) {
            const float3 pp1 = vd.pos(j), v = sub3(p, pp1);
            const float3 dx = add3(dx0, sub3(pp1, ldv3(X.dem.positions, vd.gi[j])));
            const float3 t = friction_term(P, dx, w0, vd.attr(sd.invm, X.dem.massInv, j), sqrtf(dot3(v, v)), v);
            out[0] = t.x; out[1] = t.y; out[2] = t.z;
        });
        warp_cell_sums<3>(vb, p, h, lane < 27u, SNOWB_UMAX, P.r2_le, W, acc, [&](uint32_t j, float* out) {
            const float3 v = sub3(p, vb.pos(j));
            const float3 t = friction_term(P, dx0, w0, vb.attr(sb.invm, X.bnd.massInv, j), sqrtf(dot3(v, v)), v);
            out[0] = t.x; out[1] = t.y; out[2] = t.z;
        });
        float3 c = warp_vec3(acc);
        if (nan3(c)) c = f3(0.f, 0.f, 0.f);
        if (lane == 0u) {
            if (APPLY) apply_one(P, X.dem, td, o, p, c, vd.scene(i));
            else st3(X.dem.correction, o, c);
        }
    }
}

// =================================================================== integrate
// integrate_pbd_cd_d (:467-540) / integrate_pbd_d (:447-465).  The reference kernel has no
// bounds check, so it runs over its whole launch (clamped to the allocation here).
__device__ __forceinline__ void integrate_one(const DevParams& P, const snowb_particle_data& D, uint32_t i, float dt,
                                              int cd_on)
{
    float3 tv = add3(ldv3(D.velocity, i), f3(dt * P.gx, dt * P.gy, dt * P.gz));
    tv = f3(tv.x * P.damping, tv.y * P.damping, tv.z * P.damping);
    float3 pos = ldv3(D.positions, i);
    if (!cd_on) {
        float3 pp = add3(pos, sc3(dt, tv));
        st3(D.predict_positions, i, pp);
        st3(D.velocity, i, tv);
        st3(D.new_positions, i, pp);
        return;
    }
    float3 tp = add3(pos, sc3(dt, tv));
    if (tp.x + P.r >= P.wx1) { tv.x = -fabsf(tv.x); tv = sc3(P.b_damping, tv); }
    if (tp.x - P.r <= P.wx0) { tv.x = fabsf(tv.x); tv = sc3(P.b_damping, tv); }
    if (tp.z + P.r >= P.wz1) { tv.z = -fabsf(tv.z); tv = sc3(P.b_damping, tv); }
    if (tp.z - P.r <= P.wz0) { tv.z = fabsf(tv.z); tv = sc3(P.b_damping, tv); }
    if (pos.y - P.r <= P.floor_y) {
        pos.y = P.floor_y + P.r;
        reinterpret_cast<float*>(D.positions)[3ull * i + 1] = pos.y;
        tv.y = fabsf(tv.y);
        tv = sc3(P.b_damping, tv);
    }
    if (len3(tv) > P.max_speed) tv = sc3(P.max_speed / len3(tv), tv);
    float3 pp = add3(pos, sc3(dt, tv));
    st3(D.predict_positions, i, pp);
    st3(D.velocity, i, tv);
    st3(D.new_positions, i, pp);
    float c = D.contrib[i];
    if (c < 0.99f) c += P.blending;
    if (c >= 0.99f) c = 1.f;
    D.contrib[i] = c;
}
// ts, td: a particle of the last sort (i < n) that leaves its cell marks its set for a
// full sort at the next sort point (key null: not tracked)
__global__ void k_integrate(DevParams P, const DevState* __restrict__ S, Sets X, uint32_t full, float dt, int cd_on,
                            int do_sph, int do_dem, SortTrack ts, SortTrack td)
{
    wait_prior();
    const bool ref = P.quirks == SNOWB_QUIRKS_REFERENCE;
    const uint32_t ns = S->n_sph, nd = S->n_dem;
    const uint32_t ls = do_sph ? (ref ? umin32(coverage(ns), full) : ns) : 0u;
    const uint32_t ld = do_dem ? (ref ? umin32(coverage(nd), full) : nd) : 0u;
    GRID_LOOP(t, ls + ld) {
        const bool w = t < ls;
        const uint32_t i = w ? t : t - ls;
        const snowb_particle_data& D = w ? X.sph : X.dem;
        integrate_one(P, D, i, dt, cd_on);
        const SortTrack& T = w ? ts : td;
        if (T.key && i < (w ? ns : nd))
            track_move(P, T, i, ldv3(D.predict_positions, i), T.sid ? __ldg(T.sid + i) : 0u);
    }
}

// ==================================================================== finalize
// finalize_correction (:1383-1408)
__global__ void k_finalize(DevParams P, const DevState* __restrict__ S, Sets X, float dt, int do_sph, int do_dem)
{
    wait_prior();
    const uint32_t ls = do_sph ? launch_limit(P, S->n0_sph, S->n_sph) : 0u;
    const uint32_t ld = do_dem ? launch_limit(P, S->n0_dem, S->n_dem) : 0u;
    GRID_LOOP(t, ls + ld) {
        const bool w = t < ls;
        const uint32_t i = w ? t : t - ls;
        const snowb_particle_data& D = w ? X.sph : X.dem;
        float3 np = ldv3(D.new_positions, i);
        float3 diff = sub3(np, ldv3(D.positions, i));
        float3 tv = len3(diff) >= P.min_speed ? div3(diff, dt) : f3(0.f, 0.f, 0.f);
        st3(D.velocity, i, tv);
        st3(D.positions, i, np);
    }
}

// One-thread walk of the 27 cells around p: hit(j, d2) for every member with d2 < lim but skip,
// in cell order, index ascending, close() after each cell that has members in reach.  Current
// ranges are screened two members at a time with packed arithmetic against the slightly larger
// cull, then the exact test (see d2_pair).
template <class H, class C>
__device__ __forceinline__ void walk27(const SetView& v, const Nbhd& nb, float3 p, uint32_t skip, float lim, float cull,
                                       H&& hit, C&& close)
{
    const P2 pp = bcast2(p);
    FOR27 {
        uint32_t s, e;
        if (!v.range_nb(nb, ox, oy, oz, s, e)) continue;
        auto test = [&](uint32_t j, float3 q) {
            const float3 d = sub3(p, q);
            const float d2 = dot3(d, d);
            if (d2 < lim && j != skip) hit(j, d2);
        };
        if (e <= v.n) {
            for (uint32_t j = s; j < e; j += 2u) {
                const bool two = j + 1u < e;
                const float4 q0 = __ldg(v.p4 + j), q1 = __ldg(v.p4 + (two ? j + 1u : j));
                const float2 dd = d2_pair(pp, q0, q1);
                if (dd.x < cull) test(j, xyz(q0));
                if (dd.y < cull && two) test(j + 1u, xyz(q1));
            }
        } else {
            for (uint32_t j = s; j < e; ++j) test(j, v.pos(j));
        }
        close();
    }
}
// Neighbour attributes of heat and XSPH by sorted index, for the one-thread forms: (velocity, or
// (T, 0, 0), mass / density).  A hit then costs one 16-byte load beside its position instead of
// a gather of its index, three to five gathers behind it and a division, all of them once per
// pair (32 scenes of 11,155 particles: heat 336 -> 261 us, XSPH 188 -> 144 us, this pass 4 us).
__global__ void k_pair_attrs(const DevState* __restrict__ S, SetView vs, SetView vd, Sets X, int heat,
                             float4* __restrict__ as, float4* __restrict__ ad)
{
    wait_prior();
    const uint32_t ns = S->n_sph, nd = S->n_dem;
    GRID_LOOP(t, ns + nd) {
        const bool w = t < ns;
        const uint32_t i = w ? t : t - ns, o = w ? vs.gi[i] : vd.gi[i];
        const snowb_particle_data& D = w ? X.sph : X.dem;
        const float r = D.mass[o] / D.density[o];
        const float3 a = heat ? f3(D.T[o], 0.f, 0.f) : ldv3(D.velocity, o);
        (w ? as : ad)[i] = make_float4(a.x, a.y, a.z, r);
    }
}
// ======================================================================== heat
// heat_transfer_cell (:3764-3810) over one cell
__device__ __forceinline__ float heat_cell(const DevParams& P, const SetView& v, const snowb_particle_data& O,
                                           GCell g, int ox, int oy, int oz, uint32_t skip, float3 p, float Ti,
                                           float kk)
{
    float res = 0.f;
    uint32_t s, e;
    if (v.range(P, g, ox, oy, oz, s, e))
        for (uint32_t j = s; j < e; ++j) {
            if (j == skip) continue;
            float3 dv = sub3(p, v.pos(j));
            float d2 = dot3(dv, dv);
            if (d2 < P.h2_lt) {
                const uint32_t oj = v.gi[j];
                res += (((O.mass[oj] / O.density[oj]) * kk) * (O.T[oj] - Ti)) * L_visc(P, sqrtf(d2));
            }
        }
    return res;
}
// dT plus the cells' sums over one set; attr: see k_pair_attrs (fixed quirks)
template <bool REF>
__device__ __forceinline__ float heat_sum(const DevParams& P, float dT, const SetView& v, const snowb_particle_data& O,
                                          const float4* __restrict__ attr, GCell g, uint32_t skip, float3 p, float Ti,
                                          float kk)
{
    if (REF) {
        // Q7: the reference passes the particle's own cell to all 27 calls
        const float s = heat_cell(P, v, O, g, 0, 0, 0, skip, p, Ti, kk);
        for (int k = 0; k < 27; ++k) dT += s;
        return dT;
    }
    const Nbhd nb = make_nbhd(P, g, p, P.h2_cull);
    float cs = 0.f;
    walk27(v, nb, p, skip, P.h2_lt, P.h2_cull, [&](uint32_t j, float d2) {
        float T, r;
        if (j < v.n) {
            const float4 a = __ldg(attr + j);
            T = a.x; r = a.w;
        } else {
            const uint32_t oj = v.gi[j];
            T = O.T[oj]; r = O.mass[oj] / O.density[oj];
        }
        cs += ((r * kk) * (T - Ti)) * L_visc(P, sqrtf(d2));
    }, [&]() { dT += cs; cs = 0.f; });
    return dT;
}
// transfer_heat_sph / transfer_heat_dem (:3812-3937): new_T from T
template <bool REF>   // the reference's quirk mode
__global__ void __launch_bounds__(256) k_heat(DevParams P, const DevState* __restrict__ S, SetView vs, SetView vd,
                                              Sets X, float dt, const float4* __restrict__ as,
                                              const float4* __restrict__ ad)
{
    wait_prior();
    const uint32_t ns = S->n_sph, nd = S->n_dem;
    vs.n = ns; vd.n = nd;
    const float kww = ((4.f * P.k_water) * P.k_water) / (P.k_water + P.k_water);
    const float kss = ((4.f * P.k_snow) * P.k_snow) / (P.k_snow + P.k_snow);
    const float kws = ((4.f * P.k_water) * P.k_snow) / (P.k_water + P.k_snow);
    const float ksw = ((4.f * P.k_snow) * P.k_water) / (P.k_snow + P.k_water);
    GRID_LOOP(t, ns + nd) {
        const bool w = t < ns;
        const uint32_t i = w ? t : t - ns;
        const SetView& own = w ? vs : vd;
        const SetView& oth = w ? vd : vs;
        const snowb_particle_data& A = w ? X.sph : X.dem;
        const snowb_particle_data& B = w ? X.dem : X.sph;
        const uint32_t o = own.gi[i];
        float3 p = xyz(own.p4[i]); GCell g = grid_pos(P, p, own.scene(i));
        const float Ti = A.T[o];
        float dT = 0.f;
        dT = heat_sum<REF>(P, dT, own, A, w ? as : ad, g, i, p, Ti, w ? kww : kss);
        dT = heat_sum<REF>(P, dT, oth, B, w ? ad : as, g, SNOWB_UMAX, p, Ti, w ? kws : ksw);
        dT = dT / ((w ? P.C_water : P.C_snow) * A.density[o]);
        A.new_T[o] = Ti + dT * dt;
    }
}
// the same with one warp per particle (small sets; fixed quirks at 16,380 particles, 27 cells of
// both sets: 141 -> 35 us)
__global__ void __launch_bounds__(SMALL_TPB) k_heat_warp(DevParams P, const DevState* __restrict__ S, SetView vs,
                                                         SetView vd, Sets X, float dt)
{
    wait_prior();
    __shared__ CellBuf bufs[SMALL_TPB / 32];
    CellBuf& W = bufs[threadIdx.x >> 5];
    const uint32_t ns = S->n_sph, nd = S->n_dem, lane = threadIdx.x & 31u;
    vs.n = ns; vd.n = nd;
    const bool ref = P.quirks == SNOWB_QUIRKS_REFERENCE;
    const float kww = ((4.f * P.k_water) * P.k_water) / (P.k_water + P.k_water);
    const float kss = ((4.f * P.k_snow) * P.k_snow) / (P.k_snow + P.k_snow);
    const float kws = ((4.f * P.k_water) * P.k_snow) / (P.k_water + P.k_snow);
    const float ksw = ((4.f * P.k_snow) * P.k_water) / (P.k_snow + P.k_water);
    WARP_LOOP(t, ns + nd) {
        const bool w = t < ns;
        const uint32_t i = w ? t : t - ns;
        const SetView& own = w ? vs : vd;
        const snowb_particle_data& A = w ? X.sph : X.dem;
        const uint32_t o = own.gi[i];
        const float3 p = xyz(own.p4[i]);
        const uint32_t h = lane_cell(P, grid_pos(P, p, own.scene(i)));
        const float Ti = A.T[o];
        float dT = 0.f;   // the sum so far, in lane 0
        auto add = [&](const SetView& v, const snowb_particle_data& O, uint32_t skip, float kk) {
            auto term = [&](uint32_t j, float* out) {
                const float3 dv = sub3(p, v.pos(j));
                const uint32_t oj = v.gi[j];
                out[0] = (((O.mass[oj] / O.density[oj]) * kk) * (O.T[oj] - Ti)) * L_visc(P, sqrtf(dot3(dv, dv)));
            };
            if (ref) {   // Q7: the particle's own cell, 27 times
                float s = 0.f;
                warp_cell_sums<1>(v, p, h, lane == 13u, skip, P.h2_lt, W, s, term);
                for (int k = 0; k < 27; ++k) dT += s;
            } else {
                warp_cell_sums<1>(v, p, h, lane < 27u, skip, P.h2_lt, W, dT, term);
            }
        };
        if (w) {
            add(vs, X.sph, i, kww);
            add(vd, X.dem, SNOWB_UMAX, kws);
        } else {
            add(vd, X.dem, i, kss);
            add(vs, X.sph, SNOWB_UMAX, ksw);
        }
        dT = dT / ((w ? P.C_water : P.C_snow) * A.density[o]);
        if (lane == 0u) A.new_T[o] = Ti + dT * dt;
    }
}
// thrust::copy new_T -> T (:3968-3969) then environmental_heat_transfer (:4847-4859)
__global__ void k_heat_commit(const DevState* __restrict__ S, Sets X, float dTe, int env_sph, int env_dem)
{
    wait_prior();
    const uint32_t ns = S->n_sph, nd = S->n_dem;
    GRID_LOOP(t, ns + nd) {
        const bool w = t < ns;
        const uint32_t i = w ? t : t - ns;
        const snowb_particle_data& D = w ? X.sph : X.dem;
        float T = D.new_T[i];
        if (w ? env_sph : env_dem) T += dTe;
        D.T[i] = T;
    }
}

// ======================================================================== XSPH
// xsph_viscosity_cell{,_coupling} (:3419-3502): sum of (m_j/rho_j) (v_j - v_i) W, and
// xsph_sph_viscosity / xsph_dem_viscosity (:3504-3660), Jacobi: results go to out_vel
// (`limit`, the number of sorted particles processed, carries Q6 for the snow set).
// One warp per particle: lane k < 27 computes the partial sum of cell k (the reference's
// per-cell helper), then the partials are added to the running total in cell order with
// shuffles -- the same operations in the same order as one thread would do, with 27-way
// parallelism for the small sets XSPH works on.
// Most cells hold no neighbour of a given kind, and their partial is +0 in every component.
// Adding +0 leaves a float as it is, except -0, which becomes +0 (round to nearest), and
// doing it again changes nothing; so each run of +0 partials is replaced by one addition
// of +0, and only the other partials are fetched and added, in cell order.  (A NaN in the
// total comes from arithmetic here and is already the canonical NaN that +0 keeps.)
__device__ __forceinline__ float3 warp_ordered_sum(float3 acc, float3 part)
{
    const bool nz = (__float_as_uint(part.x) | __float_as_uint(part.y) | __float_as_uint(part.z)) != 0u;
    uint32_t m = __ballot_sync(0xffffffffu, nz) & ((1u << 27) - 1u);
    const float3 zero = f3(0.f, 0.f, 0.f);
    int next = 0;   // cells before `next` are in the total
    while (m) {
        const int k = __ffs(m) - 1;
        m &= m - 1u;
        if (k > next) acc = add3(acc, zero);   // the +0 partials of cells next .. k-1
        float3 v;
        v.x = __shfl_sync(0xffffffffu, part.x, k);
        v.y = __shfl_sync(0xffffffffu, part.y, k);
        v.z = __shfl_sync(0xffffffffu, part.z, k);
        acc = add3(acc, v);
        next = k + 1;
    }
    if (next < 27) acc = add3(acc, zero);
    return acc;
}

// =============================================== PBF + contact corrections of the water set
// compute_pbf_sph_correction (:3070-3184), compute_sph_dem_distance_correction (:2061-2110)
// and compute_sph_sph_distance_correction (:1586-1646, :2164-2217) for the water particles,
// one warp per particle: lane k < 27 computes the per-cell partial of cell k for each sum
// (own water, coupling to snow, boundary, contacts) and the partials are added in cell
// order with shuffles -- the sums the one-thread loops form, with 27 cells in flight.  The
// water set is small (a few thousand particles at a time), so one thread per particle
// left the GPU nearly idle while each thread walked its neighbours.
// apply: the water part of k_apply follows at once for particles within the launch limit
// (the pass's p is k_apply's sorted position; the correction it would read is acc)
__global__ void __launch_bounds__(256) k_pbf_water_warp(DevParams P, DevState* __restrict__ S, SetView vs,
                                                        SetView vd, SetView vb, Sets X, Sorted ss, Sorted sd,
                                                        Sorted sb, float dt, StageFlags F, int apply, SortTrack ts)
{
    wait_prior();
    const uint32_t ns = S->n_sph;
    if (ns > PBF_WARP_MAX_WATER) return;   // k_pbf runs the water terms one thread each
    vs.n = ns; vd.n = S->n_dem; vb.n = S->n_b;
    const uint32_t lane = threadIdx.x & 31u;
    const bool cl = lane < 27u;
    const int ox = (int)(lane % 3u) - 1, oy = (int)((lane / 3u) % 3u) - 1, oz = (int)(lane / 9u) - 1;
    const float3 z = f3(0.f, 0.f, 0.f);
    const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < ns; i += nwarps) {
        const uint32_t o = vs.gi[i];
        const float3 p = xyz(vs.p4[i]);
        const GCell g = grid_pos(P, p, vs.scene(i));
        const float li = ss.lambda[i];
        float3 c = z;
        c = warp_ordered_sum(c, cl ? pbf_own_cell(P, vs, p, g, ox, oy, oz, i, li, ss.lambda, X.sph.lambda, ss.contrib,
                                                  X.sph.contrib, dt) : z);
        c = warp_ordered_sum(c, cl ? pbf_cpl_cell(P, vd, p, g, ox, oy, oz, i, li, sd.lambda, X.dem.lambda, dt) : z);
        c = warp_ordered_sum(c, cl ? pbf_bnd_cell(P, vb, p, g, ox, oy, oz, li, sb.lambda, X.bnd.lambda, dt) : z);
        c = sc3(P.inv_rho0, c);
        const float ci = X.sph.contrib[o];
        c = sc3(ci, c);
        if (nan3(c)) c = z;
        float3 acc = add3(ldv3(X.sph.correction, o), c);
        const float w0 = X.sph.massInv[o];
        // the contact terms are scaled by (1 - contrib): with contrib == 1 they add a zero to
        // a correction that is never -0 here, which leaves it unchanged
        if (F.correct_dem && ci != 1.f) {     // compute_sph_dem_distance_correction
            float3 d = warp_ordered_sum(z, cl ? contact_cell(P, vd, p, g, ox, oy, oz, SNOWB_UMAX, w0, sd.invm,
                                                             X.dem.massInv) : z);
            d = sc3(1.f - ci, d);
            if (nan3(d)) d = z;
            acc = add3(acc, sc3(P.k_stretch, d));
        }
        if (F.sph_sph && ci != 1.f) {         // compute_sph_sph_distance_correction (contrib <= 0.99 only)
            float3 d = ci <= 0.99f
                ? warp_ordered_sum(z, cl ? contact_cell(P, vs, p, g, ox, oy, oz, i, w0, ss.invm, X.sph.massInv) : z)
                : add3(z, z);
            d = sc3(1.f - ci, d);
            if (nan3(d)) d = z;
            acc = add3(acc, d);
        }
        if (lane == 0) {
            if (apply && i < launch_limit(P, S->n0_sph, ns)) apply_one(P, X.sph, ts, o, p, acc, vs.scene(i));
            else st3(X.sph.correction, o, acc);
        }
    }
}
__device__ __forceinline__ float3 xsph_cell(const DevParams& P, const SetView& v, const snowb_particle_data& O,
                                            const snowb_float3* vel, float3 p, GCell g, int ox, int oy, int oz,
                                            uint32_t skip, float3 vi)
{
    float3 cs = f3(0.f, 0.f, 0.f);
    uint32_t s, e;
    if (v.range(P, g, ox, oy, oz, s, e))
        for (uint32_t j = s; j < e; ++j) {
            if (j == skip) continue;
            float3 dv = sub3(p, v.pos(j));
            float d2 = dot3(dv, dv);
            if (d2 < P.h2_lt) {
                const uint32_t oj = v.gi[j];
                float3 vij = sub3(ldv3(vel, oj), vi);
                float a = O.mass[oj] / O.density[oj];
                float wgt = W_poly6(P, sqrtf(d2));
                cs = add3(cs, f3((a * vij.x) * wgt, (a * vij.y) * wgt, (a * vij.z) * wgt));
            }
        }
    return cs;
}
__global__ void __launch_bounds__(256) k_xsph_warp(DevParams P, const DevState* __restrict__ S, SetView vown,
                                                   SetView voth, snowb_particle_data A, snowb_particle_data B,
                                                   int own_is_sph, float visc, snowb_float3* __restrict__ out_vel)
{
    wait_prior();
    const uint32_t ns = S->n_sph, nd = S->n_dem;
    vown.n = own_is_sph ? ns : nd;
    voth.n = own_is_sph ? nd : ns;
    const uint32_t limit = own_is_sph ? ns
                         : (P.quirks == SNOWB_QUIRKS_REFERENCE ? umin32(coverage(ns), nd) : nd);
    const int lane = threadIdx.x & 31;
    const int ox = lane % 3 - 1, oy = (lane / 3) % 3 - 1, oz = lane / 9 - 1;
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t i = warp; i < limit; i += nwarps) {
        const uint32_t o = vown.gi[i];
        const float3 p = xyz(vown.p4[i]);
        const GCell g = grid_pos(P, p, vown.scene(i));
        const float3 vi = ldv3(A.velocity, o);
        const float3 z = f3(0.f, 0.f, 0.f);
        float3 part = lane < 27 ? xsph_cell(P, vown, A, A.velocity, p, g, ox, oy, oz, i, vi) : z;
        float3 c = warp_ordered_sum(z, part);
        part = lane < 27 ? xsph_cell(P, voth, B, B.velocity, p, g, ox, oy, oz, SNOWB_UMAX, vi) : z;
        c = warp_ordered_sum(c, part);
        c = sc3(visc, c);
        if (lane == 0) st3(out_vel, o, add3(vi, c));
    }
}
// write the Jacobi results back (only the processed particles)
// The same sums with one thread per particle, for sets large enough to fill the GPU with
// threads (the warp form's 27-way split then costs more than it hides): the cell partials
// are added in the same cell order as warp_ordered_sum adds them, cells out of reach left out
// (they would add 0).
__device__ __forceinline__ float3 xsph_sum(const DevParams& P, float3 c, const SetView& v, const snowb_particle_data& O,
                                           const float4* __restrict__ attr, const Nbhd& nb, float3 p, uint32_t skip,
                                           float3 vi)
{
    float3 cs = f3(0.f, 0.f, 0.f);
    walk27(v, nb, p, skip, P.h2_lt, P.h2_cull, [&](uint32_t j, float d2) {
        float3 vj;
        float a;
        if (j < v.n) {
            const float4 q = __ldg(attr + j);
            vj = xyz(q); a = q.w;
        } else {
            const uint32_t oj = v.gi[j];
            vj = ldv3(O.velocity, oj); a = O.mass[oj] / O.density[oj];
        }
        const float3 vij = sub3(vj, vi);
        const float wgt = W_poly6(P, sqrtf(d2));
        cs = add3(cs, f3((a * vij.x) * wgt, (a * vij.y) * wgt, (a * vij.z) * wgt));
    }, [&]() { c = add3(c, cs); cs = f3(0.f, 0.f, 0.f); });
    return c;
}
__global__ void __launch_bounds__(256) k_xsph_thread(DevParams P, const DevState* __restrict__ S, SetView vown,
                                                     SetView voth, snowb_particle_data A, snowb_particle_data B,
                                                     const float4* __restrict__ attr_own,
                                                     const float4* __restrict__ attr_oth, int own_is_sph, float visc,
                                                     snowb_float3* __restrict__ out_vel)
{
    wait_prior();
    const uint32_t ns = S->n_sph, nd = S->n_dem;
    vown.n = own_is_sph ? ns : nd;
    voth.n = own_is_sph ? nd : ns;
    const uint32_t limit = own_is_sph ? ns
                         : (P.quirks == SNOWB_QUIRKS_REFERENCE ? umin32(coverage(ns), nd) : nd);
    GRID_LOOP(i, limit) {
        const uint32_t o = vown.gi[i];
        const float3 p = xyz(vown.p4[i]);
        const Nbhd nb = make_nbhd(P, grid_pos(P, p, vown.scene(i)), p, P.h2_cull);
        const float3 vi = ldv3(A.velocity, o);
        float3 c = f3(0.f, 0.f, 0.f);
        c = xsph_sum(P, c, vown, A, attr_own, nb, p, i, vi);
        c = xsph_sum(P, c, voth, B, attr_oth, nb, p, SNOWB_UMAX, vi);
        c = sc3(visc, c);
        st3(out_vel, o, add3(vi, c));
    }
}
// Sets processed by XSPH above this many particles take the one-thread form.
constexpr uint32_t XSPH_WARP_MAX = 65536;
// attr: the set's neighbour attributes that a later XSPH pass reads (or null)
__global__ void k_xsph_commit(DevParams P, const DevState* __restrict__ S, SetView vown, int own_is_sph,
                              const snowb_float3* __restrict__ in_vel, snowb_float3* __restrict__ vel,
                              float4* __restrict__ attr)
{
    wait_prior();
    const uint32_t ns = S->n_sph, nd = S->n_dem;
    const uint32_t limit = own_is_sph ? ns
                         : (P.quirks == SNOWB_QUIRKS_REFERENCE ? umin32(coverage(ns), nd) : nd);
    GRID_LOOP(i, limit) {
        const uint32_t o = vown.gi[i];
        const float3 v = ldv3(in_vel, o);
        st3(vel, o, v);
        if (attr) attr[i] = make_float4(v.x, v.y, v.z, attr[i].w);
    }
}

// ===================================================================== misc
// compute_boundary_volume_d (:303-346) with sph_boundary_volume (:159-192); reads the
// caller's sorted positions directly (one-time setup).
__global__ void k_boundary_volume(DevParams P, snowb_cell_data cd, const float* __restrict__ mass,
                                  float* __restrict__ volume, uint32_t n, const uint32_t* __restrict__ sid_o)
{
    wait_prior();
    GRID_LOOP(i, n) {
        const uint32_t o = cd.grid_index[i];
        float3 p = ldv3(cd.sorted_pos, i);
        float rho = mass[o] * P.W0;
        GCell g = grid_pos(P, p, sid_o ? sid_o[o] : 0u);
        FOR27 {
            float cs = 0.f;
            uint32_t h = grid_hash(P, g, ox, oy, oz);
            uint32_t s = cd.cell_start[h];
            if (s != SNOWB_EMPTY) {
                uint32_t e = cd.cell_end[h];
                for (uint32_t j = s; j < e; ++j) {
                    if (j == i) continue;
                    float3 dv = sub3(p, ldv3(cd.sorted_pos, j));
                    float d2 = dot3(dv, dv);
                    if (d2 < P.h2_lt) cs += mass[cd.grid_index[j]] * W_poly6(P, sqrtf(d2));
                }
            }
            rho += cs;
        }
        volume[o] = mass[o] / rho;
    }
}
// compact sorted view of the boundary set: p4 = (pos, volume), invm/mass by sorted index
__global__ void k_boundary_prep(snowb_cell_data cd, const float* __restrict__ volume, const float* __restrict__ invm,
                                const float* __restrict__ mass, uint32_t n, float4* __restrict__ p4,
                                float* __restrict__ invm_s, float* __restrict__ mass_s,
                                const uint32_t* __restrict__ sid_o, uint32_t* __restrict__ sid_s)
{
    wait_prior();
    GRID_LOOP(i, n) {
        const uint32_t o = cd.grid_index[i];
        float3 q = ldv3(cd.sorted_pos, i);
        p4[i] = make_float4(q.x, q.y, q.z, volume[o]);
        invm_s[i] = invm[o];
        mass_s[i] = mass[o];
        if (sid_s) sid_s[i] = sid_o[o];
    }
}
__global__ void k_set_state(DevState* S, uint32_t ns, uint32_t nd, uint32_t nb)
{
    wait_prior();
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        S->n_sph = ns; S->n_dem = nd; S->n_b = nb;
        S->n0_sph = ns; S->n0_dem = nd;
        S->n_freeze = 0; S->n_melt = 0; S->changed = 0; S->new_sph = ns; S->new_dem = nd;
        // the caller may have changed the tail slots between calls: the first compaction
        // of a call cleans the tail as the reference's does every substep
        S->tail_dirty = 1u;
        // ... and the particles: the first sort point of a call sorts both sets in full
        for (int k = 0; k < 2; ++k) { S->moved[k] = 1u; S->table_any[k] = 1u; S->sorts_full[k] = 0u; S->sorts_kept[k] = 0u; }
        S->skin_passes = S->skin_walks = S->skin_marks = 0u;
        for (int c = 0; c < 8; ++c) S->sc_count[c] = 0u;
        S->clean_hi[0] = SNOWB_UMAX; S->clean_hi[1] = SNOWB_UMAX;
        S->base_ready = 0u;   // ... and the boundary
    }
}
// batched runs: every live slot's scene id must name a scene of the batch
__global__ void k_check_scenes(DevParams P, DevState* S, const uint32_t* __restrict__ sph,
                               const uint32_t* __restrict__ dem, const uint32_t* __restrict__ bnd)
{
    wait_prior();
    const uint32_t ns = S->n_sph, nd = S->n_dem, nb = S->n_b;
    const uint32_t n = ns > nd ? (ns > nb ? ns : nb) : (nd > nb ? nd : nb);
    GRID_LOOP(i, n) {
        bool bad = (i < ns && sph[i] > P.scene_mask) || (i < nd && dem[i] > P.scene_mask) ||
                   (i < nb && bnd[i] > P.scene_mask);
        if (bad) atomicOr(&S->err, SNOWB_DEVERR_SCENE);
    }
}

// FP64 heat-energy and momentum partial sums (deterministic two-level reduction)
__global__ void k_energy_partial(const snowb_particle_data sph, uint32_t ns, const snowb_particle_data dem,
                                 uint32_t nd, double Cw, double Cs, double* __restrict__ part)
{
    wait_prior();
    __shared__ double sm[4][256];
    double a[4] = {0, 0, 0, 0};
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < ns + nd; t += gridDim.x * blockDim.x) {
        const bool w = t < ns;
        const uint32_t i = w ? t : t - ns;
        const snowb_particle_data& D = w ? sph : dem;
        double m = (double)D.mass[i];
        float3 v = ldv3(D.velocity, i);
        a[0] += m * (w ? Cw : Cs) * (double)D.T[i];
        a[1] += m * (double)v.x; a[2] += m * (double)v.y; a[3] += m * (double)v.z;
    }
    for (int k = 0; k < 4; ++k) sm[k][threadIdx.x] = a[k];
    __syncthreads();
    for (int st = 128; st > 0; st >>= 1) {
        if ((int)threadIdx.x < st)
            for (int k = 0; k < 4; ++k) sm[k][threadIdx.x] += sm[k][threadIdx.x + st];
        __syncthreads();
    }
    if (threadIdx.x == 0)
        for (int k = 0; k < 4; ++k) part[4 * blockIdx.x + k] = sm[k][0];
}
__global__ void k_energy_final(const double* __restrict__ part, int nblocks, double* __restrict__ out)
{
    wait_prior();
    if (threadIdx.x < 4) {
        double s = 0;
        for (int b = 0; b < nblocks; ++b) s += part[4 * b + threadIdx.x];
        out[threadIdx.x] = s;
    }
}

}  // namespace snowb
