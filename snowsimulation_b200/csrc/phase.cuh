// phase.cuh -- freezing/melting with compaction (cuda_simulation.cu:3974-4125, :4387-4622)
// and interlink formation (:4127-4292, :4768-4816).
//
// Phase change.  The reference claims target slots with atomicAdd, so their order is
// scheduling dependent (Q8); here a particle's target is its rank among the particles
// changing phase (ascending index).  Compaction always runs in the reference; when no
// particle changed phase it is an identity, so every compaction kernel returns early
// unless DevState::changed is set (no host round trip is needed).
//
// Interlink formation.  The reference lets every snow particle claim slots with atomics
// while others read the same slots (Q10), so the topology depends on scheduling.  Here
// the pass is the sequential reference procedure applied in one fixed order: hash cells
// are grouped into 2x2x2 super-cells, each super-cell gets a colour 0..7 from the parity
// of its coordinates, colours run in turn, and inside a colour each super-cell walks its
// particles in ascending sorted index.  A particle only edits its own slots and those of
// neighbours within h, i.e. in adjacent cells; same-coloured super-cells are at least
// three cells apart, so they never touch the same particle and run in parallel, one
// block per super-cell (one thread above SNOWB_MAXC_FAST slots).  A prefilter marks the particles that can change anything:
// links are never removed during the pass and counts only grow, so a particle whose
// count already reaches its cap, or whose candidates are all linked already, is a no-op.
#pragma once
#include "common.cuh"
#include "sort.cuh"

namespace snowb {

#define SNOWB_MAXC_FAST 32   // interlink slots kept in registers (maximum_connection <= 32)

// copy_particle_info (:3974-4002): every per-particle field, then the link slots
__device__ __forceinline__ void copy_fields(const snowb_particle_data& s, const snowb_particle_data& d, uint32_t i,
                                            uint32_t t)
{
    st3(d.positions, t, ldv3(s.positions, i));
    st3(d.predict_positions, t, ldv3(s.predict_positions, i));
    st3(d.new_positions, t, ldv3(s.new_positions, i));
    st3(d.velocity, t, ldv3(s.velocity, i));
    st3(d.force, t, ldv3(s.force, i));
    st3(d.correction, t, ldv3(s.correction, i));
    d.mass[t] = s.mass[i];
    d.massInv[t] = s.massInv[i];
    d.contrib[t] = s.contrib[i];
    d.density[t] = s.density[i];
    d.C[t] = s.C[i];
    d.lambda[t] = s.lambda[i];
    d.T[t] = s.T[i];
    d.new_T[t] = s.new_T[i];
    d.trackId[t] = s.trackId[i];
    d.iter_end[t] = s.iter_end[i];
}
__device__ __forceinline__ void copy_info(const snowb_particle_data& s, const snowb_particle_data& d, uint32_t i,
                                          uint32_t t, uint32_t M)
{
    copy_fields(s, d, i, t);
    for (uint32_t c = 0; c < M; ++c) {
        d.connect_record[t * M + c] = s.connect_record[i * M + c];
        d.connect_length[t * M + c] = s.connect_length[i * M + c];
    }
}
__device__ __forceinline__ void reset_records(const snowb_particle_data& d, uint32_t t, uint32_t M)
{
    for (uint32_t c = 0; c < M; ++c) {
        d.connect_record[t * M + c] = SNOWB_UMAX;
        d.connect_length[t * M + c] = 0.f;
    }
    d.iter_end[t] = M * t;
}

// freeze / melt predicates (:4425, :4396)
// commit: the heat pass's commit (k_heat_commit: T from new_T, plus the environment
// term) first, each particle its own, so the flags read the committed temperature
__global__ void k_phase_flags(DevParams P, const DevState* __restrict__ S, snowb_particle_data sph,
                              snowb_particle_data dem, int freeze, int melt, uint32_t* __restrict__ fl_s,
                              uint32_t* __restrict__ fl_d, int commit, float dTe, int env_sph, int env_dem)
{
    wait_prior();
    const uint32_t ns = S->n_sph, nd = S->n_dem;
    GRID_LOOP(t, ns + nd) {
        const bool w = t < ns;
        const uint32_t i = w ? t : t - ns;
        const snowb_particle_data& D = w ? sph : dem;
        float T;
        if (commit) {
            T = D.new_T[i];
            if (w ? env_sph : env_dem) T += dTe;
            D.T[i] = T;
        } else {
            T = D.T[i];
        }
        if (w) fl_s[i] = (freeze && T <= P.Tf && sph.contrib[i] >= 0.99f) ? 1u : 0u;
        else fl_d[i] = (melt && T > P.Tf && dem.contrib[i] >= 0.99f) ? 1u : 0u;
    }
}
// scene ids of batched runs travel with the particles (null pointers: one scene)
struct SceneIds {
    uint32_t *sph, *dem, *buf;
};
// freezing (:4416-4449) and melting (:4387-4414) with ranked targets, and the phase-change
// flag: every block derives it from the counts, block 0 stores it for the later passes
__global__ void k_phase_move(DevParams P, DevState* __restrict__ S, snowb_particle_data sph,
                             snowb_particle_data dem, const uint32_t* __restrict__ fl_s,
                             const uint32_t* __restrict__ rk_s, const uint32_t* __restrict__ fl_d,
                             const uint32_t* __restrict__ rk_d, SceneIds sc)
{
    wait_prior();
    const bool changed = (S->n_freeze + S->n_melt) != 0u;
    if (blockIdx.x == 0 && threadIdx.x == 0) S->changed = changed ? 1u : 0u;
    if (!changed) return;
    const uint32_t ns = S->n_sph, nd = S->n_dem, M = P.maxc;
    GRID_LOOP(t, ns + nd) {
        if (t < ns) {
            if (!fl_s[t]) continue;
            const uint32_t i = t, tg = nd + rk_s[i];
            sph.contrib[i] = 0.f;
            copy_info(sph, dem, i, tg, M);
            if (sc.sph) sc.dem[tg] = sc.sph[i];
            sph.predicate[i] = 0; sph.trackId[i] = 0;
            dem.predicate[tg] = 1;
            reset_records(dem, tg, M);
        } else {
            const uint32_t i = t - ns;
            if (!fl_d[i]) continue;
            const uint32_t tg = ns + rk_d[i];
            dem.contrib[i] = 0.f;
            copy_info(dem, sph, i, tg, M);
            if (sc.sph) sc.sph[tg] = sc.dem[i];
            dem.predicate[i] = 0; dem.trackId[i] = 0;
            sph.predicate[tg] = 1;
        }
    }
}
// Compaction moves the kept particles to their ranks (scan_index).  A kept particle with
// no removed one before it stays where it is, and copying it out and back, as the
// reference's copy_to_target and scatter do for every slot, leaves it unchanged; so both
// passes move only the particles whose slot changes (the phase-change buffer, scratch the
// reference overwrites at every compaction, holds only those).  Threads k < full take a
// particle's fields, the others one link slot each (coalesced over the slot arrays).
__device__ __forceinline__ bool compaction_moves(const snowb_particle_data& d, uint32_t i)
{
    return d.predicate[i] == 1 && d.scan_index[i] != i;
}
// The two sets' compactions, side by side in the same launches: the water set through the
// caller's phase-change buffer, the snow set through the library's.
struct CompactSide {
    snowb_particle_data d, buf;
    uint32_t *sid, *sid_buf;      // scene ids (batched runs) or null
    const uint32_t* removed;      // the number of particles the set loses (none: no particle moves)
    int rebase;
};
struct CompactPair {
    CompactSide a[2];
};
// copy_to_target (:4451-4460) into the phase-change buffer
__global__ void k_copy_to_buffer(DevParams P, const DevState* __restrict__ S, const __grid_constant__ CompactPair Q,
                                 uint32_t full)
{
    wait_prior();
    if (S->changed == 0) return;
    const uint32_t M = P.maxc;
#pragma unroll 1
    for (int set = 0; set < 2; ++set) {
        const CompactSide& A = Q.a[set];
        GRID_LOOP(k, *A.removed ? full * (M + 1) : 0u) {
            if (k < full) {
                if (!compaction_moves(A.d, k)) continue;
                copy_fields(A.d, A.buf, k, k);
                if (A.sid) A.sid_buf[k] = A.sid[k];
            } else {
                const uint32_t s = k - full;
                if (!compaction_moves(A.d, s / M)) continue;
                A.buf.connect_record[s] = A.d.connect_record[s];
                A.buf.connect_length[s] = A.d.connect_length[s];
            }
        }
    }
}
// scatter (:4462-4480).  rebase (fixed quirks, snow set): a moved particle keeps its link
// count, iter_end = t*M + count; the reference copies iter_end verbatim (Q13).  A particle
// that stays keeps its iter_end either way.
__global__ void k_scatter_set(DevParams P, DevState* S, const __grid_constant__ CompactPair Q, uint32_t full)
{
    wait_prior();
    if (S->changed == 0) return;
    const uint32_t M = P.maxc;
#pragma unroll 1
    for (int set = 0; set < 2; ++set) {
        const CompactSide& A = Q.a[set];
        // with nothing removed every kept particle stays: only new_index is written
        GRID_LOOP(k, *A.removed ? full * (M + 1) : full) {
            if (k < full) {
                const uint32_t i = k;
                if (A.d.predicate[i] == 1) {
                    const uint32_t t = A.d.scan_index[i];
                    if (t >= full) { atomicOr(&S->err, SNOWB_DEVERR_SCATTER); continue; }
                    if (t != i) {
                        copy_fields(A.buf, A.d, i, t);
                        if (A.rebase) A.d.iter_end[t] = M * t + (A.buf.iter_end[i] - M * i);
                        if (A.sid) A.sid[t] = A.sid_buf[i];
                    }
                    A.d.new_index[i] = t;
                } else A.d.new_index[i] = SNOWB_UMAX;
            } else {
                const uint32_t s = k - full, i = s / M;
                if (A.d.predicate[i] != 1) continue;
                const uint32_t t = A.d.scan_index[i];
                if (t >= full || t == i) continue;
                const uint32_t q = t * M + (s - i * M);
                A.d.connect_record[q] = A.buf.connect_record[s];
                A.d.connect_length[q] = A.buf.connect_length[s];
            }
        }
    }
}
// setSize / new_end (:4545-4551), predicate fill (:4555-4556), clean_tail (:4482-4493).
// The reference compacts every substep; without a phase change that is an identity except
// that it zeroes scan_index in the tail and, if a link pass wrote into tail slots, resets
// them (`full_clean`), which is what this kernel does in that case.
// The tail clean only has to reach the slots that can differ from a clean slot: those that
// held a particle before this compaction (below the set's size plus the particles it
// gained) and those not known clean since the last clean (DevState::clean_hi; a call's
// first compaction and any link pass that wrote past a set's end, tail_dirty, clean the
// whole tail).  A slot at or above both already holds what the clean writes.
// records: also the record update below (update_record_index; its slots, below the new
// snow size, are none of the tail slots this pass cleans), in the same launch
__device__ __forceinline__ void update_record(const DevParams& P, const DevState* S, const snowb_particle_data& dem,
                                              uint32_t s, bool moved, uint32_t nd_old, uint32_t nd);
__global__ void k_compact_finish(DevParams P, DevState* S, snowb_particle_data sph, snowb_particle_data dem,
                                 uint32_t full, int records)
{
    wait_prior();
    const bool full_clean = S->changed || S->tail_dirty;
    const uint32_t sn = S->new_sph, dn = S->new_dem, M = P.maxc;
    const uint32_t hs = S->tail_dirty ? full : umin32(full, umax32(S->clean_hi[0], S->n_sph + S->n_melt));
    const uint32_t hd = S->tail_dirty ? full : umin32(full, umax32(S->clean_hi[1], S->n_dem + S->n_freeze));
    const bool moved = S->changed != 0;
    const uint32_t nd_old = S->n_dem, nd_rec = moved ? S->new_dem : S->n_dem;
    const uint32_t nrec = records && full_clean ? M * nd_rec : 0u;
    GRID_LOOP(t, 2 * full + nrec) {
        if (t >= 2 * full) {
            update_record(P, S, dem, t - 2 * full, moved, nd_old, nd_rec);
            continue;
        }
        const bool w = t < full;
        const uint32_t i = w ? t : t - full;
        const snowb_particle_data& d = w ? sph : dem;
        const uint32_t n = w ? sn : dn;
        if (i < n) {
            if (full_clean) d.predicate[i] = 1;
        } else {
            d.scan_index[i] = 0;
            if (full_clean && i < (w ? hs : hd)) {
                d.predicate[i] = 0; d.trackId[i] = 0;
                reset_records(d, i, M);
            }
        }
        if (i == 0 && full_clean) *d.new_end = n;
    }
}
// The compaction's last launch: the new sizes (a compacted set is sorted in full next),
// the clean mark of the tails, and the tail flag cleared.
__global__ void k_commit_sizes(DevState* S)
{
    wait_prior();
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        // after a clean every slot past the new sizes is clean
        if (S->changed || S->tail_dirty) { S->clean_hi[0] = S->new_sph; S->clean_hi[1] = S->new_dem; }
        if (S->changed) {
            S->n_sph = S->new_sph; S->n_dem = S->new_dem;
            S->moved[0] = 1u; S->moved[1] = 1u;
        }
        S->tail_dirty = 0;
    }
}
// update_record_index (:4114-4125), after the compaction, with shuffle_useless_record
// (:4068-4111) folded in: the reference clears, before the compaction, each link to a
// partner that left the snow set (its record, its length, one off the owner's count).  The
// link's slot moves with its owner and the partner's new index is then empty, so the same
// slot is cleared here at the owner's new place; the count's decrement commutes with the
// compaction's copy or rebase of it.
__device__ __forceinline__ void update_record(const DevParams& P, const DevState* S, const snowb_particle_data& dem,
                                              uint32_t s, bool moved, uint32_t nd_old, uint32_t nd)
{
    const uint32_t r = dem.connect_record[s];
    if (r == SNOWB_UMAX) return;
    if (moved) {
        const uint32_t nr = dem.new_index[r];
        if (r < nd_old && nr == SNOWB_UMAX) {
            dem.connect_length[s] = 0.f;
            atomicSub(dem.iter_end + s / P.maxc, 1u);
        }
        dem.connect_record[s] = nr;
    } else {
        // without a phase change the reference's new_index is the identity below n, empty above
        dem.connect_record[s] = r < nd ? r : SNOWB_UMAX;
    }
}

// ======================================================================= links
__device__ __forceinline__ uint32_t link_tolerance(const DevParams& P, float T, int dynamic)
{
    uint32_t tol = dynamic ? __float2uint_rz(((T - P.Tf) / (P.Th - P.Tf)) * (float)P.maxc) : P.maxc;
    return tol < P.maxc ? tol : P.maxc;
}
// Prefilter: can particle (sorted) i change any record in this pass?  During the pass
// links are only added and counts only grow, so i is a no-op if its count already reaches
// its cap, if it has no free slot, or if every candidate (d < h) is either linked to it
// already or has no room (count at the cap or no free slot): an attempt on a full
// partner claims a slot of i and releases it again.  A candidate that is i itself (a
// stale cell range can hold it) keeps i active.
__device__ __forceinline__ bool has_free_slot(const uint32_t* rec, uint32_t o, uint32_t M)
{
    for (uint32_t q = M * o; q < M * (o + 1); ++q)
        if (rec[q] == SNOWB_UMAX) return true;
    return false;
}
// Super-cells holding an active particle, listed per colour by the prefilter so that a
// colour pass visits only those (same-coloured super-cells are independent, so their order
// does not matter; inside one the particles are still taken in ascending sorted index).
// flag null: no list, the colour pass visits every super-cell of its colour.
struct SCList {
    uint32_t* flag;     // per super-cell (colour c, index t at c * per + t): listed
    uint32_t* list;     // colour c's listed indices t at list[c * per + k], k < count[c]
    uint32_t* count;    // DevState::sc_count
    uint32_t per;       // super-cells per colour
};
// colour and index within the colour of the super-cell holding hash cell h (the layout of
// k_link_colour_warp: super-cell (sx, sy, sz) = cell / 2, colour = parities of sx, sy, sz)
__device__ __forceinline__ void supercell_of(const DevParams& P, uint32_t h, uint32_t& colour, uint32_t& t)
{
    const uint32_t x = h % P.gsx, y = (h / P.gsx) % P.gsy, z = h / (P.gsx * P.gsy);
    const uint32_t sx = x >> 1, sy = y >> 1, sz = z >> 1;
    colour = (sx & 1u) | ((sy & 1u) << 1) | ((sz & 1u) << 2);
    t = (sx >> 1) + (P.gsx >> 2) * ((sy >> 1) + (P.gsy >> 2) * (sz >> 1));
}
__device__ __forceinline__ void list_supercell(const DevParams& P, const SCList& sc, uint32_t h)
{
    uint32_t colour, t;
    supercell_of(P, h, colour, t);
    if (atomicCAS(sc.flag + colour * sc.per + t, 0u, 1u) == 0u)
        sc.list[colour * sc.per + atomicAdd(sc.count + colour, 1u)] = t;
}

// the particles of hash cell h in the current sort: their number and first sorted index (a stale
// range does not begin with an entry of its own cell)
__device__ __forceinline__ uint32_t current_range(const SetView& v, uint32_t h, uint32_t& b)
{
    b = v.cs[h];
    return b != SNOWB_EMPTY && b < v.n && v.gh[b] == h ? v.ce[h] - b : 0u;
}
// L: the snow-snow candidate lists of the substep's first density pass (L.cnt null: none),
// replayed instead of the traversal while no phase change re-sorted the sets.
constexpr uint32_t LF_G = 4;
__global__ void __launch_bounds__(256) k_link_filter(DevParams P, DevState* S, SetView vd,
                                                     snowb_particle_data dem, int dynamic,
                                                     uint8_t* __restrict__ active, NList L, SCList sc)
{
    wait_prior();
    const uint32_t nd = S->n_dem, M = P.maxc;
    vd.n = nd;
    const bool lists = L.cnt != nullptr && S->changed == 0;
    GRID_LOOP(i, nd) {
        const uint32_t o = vd.gi[i];
        const float3 p = vd.pos(i);
        const uint32_t count = dem.iter_end[o] - o * M;
        uint8_t act = 0;
        // With dynamic caps, adjust_connections (:4768-4808) can leave iter_end below the
        // particle's first slot (it decrements for every slot past the cap, empty ones
        // included), so count wraps round; links that partners add during the pass then
        // bring it back below the cap.  Such a particle is kept: the pass decides.
        if (dem.iter_end[o] < o * M) {
            active[i] = 1;
            atomicAdd(&S->n_active, 1u);
            if (sc.flag) list_supercell(P, sc, vd.gh[i]);
            continue;
        }
        // a particle at its cap stays inactive: its slots are not even read
        const bool below = count < link_tolerance(P, dem.T[o], dynamic);
        // own slots in registers (M <= SNOWB_MAXC_FAST), else read from memory
        uint32_t r[SNOWB_MAXC_FAST];
        const bool fast = M <= SNOWB_MAXC_FAST;
#pragma unroll
        for (int k = 0; k < SNOWB_MAXC_FAST; ++k)
            r[k] = below && fast && (uint32_t)k < M ? dem.connect_record[M * o + k] : 0u;
        const uint32_t lc = lists ? L.cnt[L.cap + i] : NL_OVF;
        // a free slot of o: from the registers (slots k >= M hold 0, never empty)
        bool own_free = false;
        if (below) {
            if (fast) {
#pragma unroll
                for (int k = 0; k < SNOWB_MAXC_FAST; ++k) own_free |= r[k] == SNOWB_UMAX;
            } else {
                own_free = has_free_slot(dem.connect_record, o, M);
            }
        }
        if (!(lc & NL_OVF) && own_free) {
            // the same scan over the listed candidates (cells in order, d < h, j != i), taken
            // LF_G at a time: entries, partners' original indices and counts are loaded for
            // the group (all in range: listed entries are current sorted indices), then the
            // candidates are examined in order
            uint32_t skip_cell = 0xFFu;
            const uint32_t nl = lc & 1023u;
            for (uint32_t k0 = 0; k0 < nl && !act; k0 += LF_G) {
                uint32_t en[LF_G], o1[LF_G], ie[LF_G];
#pragma unroll
                for (uint32_t u = 0; u < LF_G; ++u)
                    en[u] = k0 + u < nl ? L.e[(size_t)(k0 + u) * L.stride + L.cap + i] : 0u;
#pragma unroll
                for (uint32_t u = 0; u < LF_G; ++u) o1[u] = k0 + u < nl ? vd.gi[en[u] & NL_J_MASK] : 0u;
#pragma unroll
                for (uint32_t u = 0; u < LF_G; ++u) ie[u] = k0 + u < nl ? dem.iter_end[o1[u]] : 0u;
#pragma unroll
                for (uint32_t u = 0; u < LF_G; ++u) {
                    if (k0 + u >= nl || act) break;
                    const uint32_t cell = (en[u] >> 25) & 31u;
                    if (cell == skip_cell || (en[u] & NL_FAR)) continue;
                    if (o1[u] == o) { act = 1; break; }
                    bool found = false;
                    if (fast) {
#pragma unroll
                        for (int q = 0; q < SNOWB_MAXC_FAST; ++q) found |= (uint32_t)q < M && r[q] == o1[u];
                    } else {
                        for (uint32_t q = M * o; q < M * (o + 1); ++q)
                            if (dem.connect_record[q] == o1[u]) { found = true; break; }
                    }
                    if (found) { skip_cell = cell; continue; }
                    if (ie[u] < (o1[u] + 1) * M && has_free_slot(dem.connect_record, o1[u], M)) act = 1;
                }
            }
        } else if ((lc & NL_OVF) && own_free) {
            const GCell g = grid_pos(P, p, vd.scene(i));
            FOR27 {
                uint32_t s, e;
                if (!vd.range(P, g, ox, oy, oz, s, e)) continue;
                for (uint32_t j = s; j < e && !act; ++j) {
                    if (j == i) continue;
                    float3 dv = sub3(p, vd.pos(j));
                    if (dot3(dv, dv) < P.h2_lt) {
                        const uint32_t o1 = vd.gi[j];
                        if (o1 == o) { act = 1; break; }
                        bool found = false;
                        if (fast) {
#pragma unroll
                            for (int k = 0; k < SNOWB_MAXC_FAST; ++k) found |= (uint32_t)k < M && r[k] == o1;
                        } else {
                            for (uint32_t q = M * o; q < M * (o + 1); ++q)
                                if (dem.connect_record[q] == o1) { found = true; break; }
                        }
                        // a linked candidate ends the reference's scan of this cell, and it
                        // stays linked, so nothing after it in the cell is reached
                        if (found) break;
                        if (dem.iter_end[o1] < (o1 + 1) * M && has_free_slot(dem.connect_record, o1, M)) act = 1;
                    }
                }
                if (act) break;
            }
        }
        active[i] = act;
        if (act) {
            atomicAdd(&S->n_active, 1u);
            if (sc.flag) list_supercell(P, sc, vd.gh[i]);
        }
    }
}
// A particle's links by one warp.  The sequential rule of link_particle, for up to 32
// candidates in traversal order (lane k holds candidate k), resolved at once:
//  - a candidate that o is already linked to ends its cell, so it and the later candidates
//    of its cell drop out;
//  - of the rest, those whose partner has room (count below the cap and a free slot) are
//    linked in order, each into o's next free slot, until o's count reaches its cap or its
//    slots run out; a partner without room changes nothing.
// A link changes only o and its own partner, so the partners' counts and slots are all read
// before the first link, eight slot rows in flight at a time, and the links are written side
// by side: a chunk costs a few dependent memory round trips, where taking the candidates one
// after another cost two for each.  A particle that meets itself or the same partner twice in
// a chunk (stale cell ranges) takes the candidates one by one.
struct LinkState {
    uint32_t o, base, tol, count, skip_cell;
    uint32_t rk;   // lane k < M holds slot k of particle o, the others LINK_NO_SLOT
};
constexpr uint32_t LINK_NO_SLOT = SNOWB_UMAX - 1u;   // no particle index and not an empty slot
// which lanes' candidates (o1, of a cell) o is already linked to or meets after such a one in
// its cell; carries the last ended cell over
__device__ __forceinline__ bool link_ended(uint32_t rk, uint32_t& skip_cell, bool in, uint32_t o1, uint32_t cell,
                                           uint32_t& dupm)
{
    const uint32_t full = 0xffffffffu, lane = threadIdx.x & 31u;
    in = in && cell != skip_cell;
    bool dup = false;
#pragma unroll
    for (int q = 0; q < SNOWB_MAXC_FAST; ++q) dup |= __shfl_sync(full, rk, q) == o1;
    dupm = __ballot_sync(full, in && dup);
    const uint32_t same = __match_any_sync(full, in ? cell : 0x100u + lane);
    if (dupm) skip_cell = __shfl_sync(full, cell, 31 - __clz(dupm));
    return !in || dup || (same & dupm & ((1u << lane) - 1u)) != 0u;
}
struct LinkMap {
    uint32_t slot[32], partner[32];                // by rank of the link: o's slot, the partner
};
// false: nothing later can change anything (cap reached or no free slot)
__device__ __forceinline__ bool link_chunk(const DevParams& P, const snowb_particle_data& d, DevState* S, uint32_t n,
                                           LinkState& L, LinkMap& map, bool in, uint32_t o1, uint32_t cell, float dist)
{
    const uint32_t lane = threadIdx.x & 31u, M = P.maxc, full = 0xffffffffu, below = (1u << lane) - 1u;
    if (!(L.count < L.tol)) return false;
    uint32_t freem = __ballot_sync(full, L.rk == SNOWB_UMAX);
    if (!freem) return false;
    const uint32_t b1 = o1 * M;
    const uint32_t ie = in ? d.iter_end[o1] : 0u;
    uint32_t dupm;
    const bool elig = !link_ended(L.rk, L.skip_cell, in, o1, cell, dupm);   // every lane takes part
    const uint32_t twin = __match_any_sync(full, elig ? o1 : 0x80000000u | lane);
    if (__any_sync(full, elig && (o1 == L.o || (twin & (twin - 1u))))) {
        uint32_t m = __ballot_sync(full, elig);
        uint32_t dead = 0xFFu;   // a cell that a link made in this chunk ended
        while (m) {
            const int k = __ffs(m) - 1;
            m &= m - 1u;
            if (!(L.count < L.tol)) return false;
            const uint32_t p1 = __shfl_sync(full, o1, k), pc = __shfl_sync(full, cell, k);
            const float pd = __shfl_sync(full, dist, k);
            if (pc == dead) continue;
            if (__any_sync(full, L.rk == p1)) {
                dead = pc;
                if (!dupm || pc > L.skip_cell) L.skip_cell = pc;   // the last ended cell carries over
                continue;
            }
            freem = __ballot_sync(full, L.rk == SNOWB_UMAX);
            if (!freem) return false;
            const int fk = __ffs(freem) - 1;
            if (lane == 0) d.connect_record[L.base + fk] = p1;   // claim
            if (lane == (uint32_t)fk) L.rk = p1;
            __syncwarp();
            const uint32_t c1 = p1 * M;
            bool valid = false;
            if (d.iter_end[p1] < c1 + M) {
                const uint32_t q = lane < M ? d.connect_record[c1 + lane] : 0u;
                const uint32_t pm = __ballot_sync(full, lane < M && q == SNOWB_UMAX);
                __syncwarp();
                if (pm) {
                    const int pk = __ffs(pm) - 1;
                    if (lane == 0) {
                        d.connect_record[c1 + pk] = L.o;
                        d.connect_length[c1 + pk] = pd;
                        d.iter_end[p1]++;
                        if (p1 >= n) atomicOr(&S->tail_dirty, 1u);
                    }
                    if (p1 == L.o) {                     // self link (stale cell range)
                        ++L.count;
                        if (lane == (uint32_t)pk) L.rk = L.o;
                    }
                    valid = true;
                }
            }
            __syncwarp();
            if (valid) {
                ++L.count;
                if (lane == 0) {
                    d.connect_length[L.base + fk] = pd;
                    d.iter_end[L.o] = L.base + L.count;
                    atomicAdd(&S->n_links, 1u);
                }
            } else {
                if (lane == 0) d.connect_record[L.base + fk] = SNOWB_UMAX;
                if (lane == (uint32_t)fk) L.rk = SNOWB_UMAX;
            }
            __syncwarp();
        }
        return true;
    }
    const uint32_t most = umin32(L.tol - L.count, (uint32_t)__popc(freem));
    uint32_t need = __ballot_sync(full, elig && ie < b1 + M), okm = 0;
    int pk = 0;   // this lane's candidate: the partner's first free slot
    while (need && (uint32_t)__popc(okm) < most) {
        int k[8];
        uint32_t q[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            k[u] = need ? __ffs(need) - 1 : -1;
            need &= need - 1u;
            const uint32_t row = __shfl_sync(full, b1, k[u] < 0 ? 0 : k[u]);
            q[u] = k[u] >= 0 && lane < M ? d.connect_record[row + lane] : 0u;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const uint32_t pm = __ballot_sync(full, q[u] == SNOWB_UMAX);
            if (pm) okm |= 1u << k[u];
            if (lane == (uint32_t)k[u]) pk = __ffs(pm) - 1;
        }
    }
    // the r-th candidate with room takes the r-th free slot
    const uint32_t made = umin32(most, (uint32_t)__popc(okm)), r = __popc(okm & below), fr = __popc(freem & below);
    const bool link = (okm >> lane & 1u) && r < made, gets = (freem >> lane & 1u) && fr < made;
    __syncwarp();
    if (link) map.partner[r] = o1;
    if (gets) map.slot[fr] = lane;
    __syncwarp();
    if (gets) L.rk = map.partner[fr];
    if (link) {
        const uint32_t fk = map.slot[r];
        d.connect_record[L.base + fk] = o1;
        d.connect_length[L.base + fk] = dist;
        d.connect_record[b1 + pk] = L.o;
        d.connect_length[b1 + pk] = dist;
        d.iter_end[o1] = ie + 1u;
        if (o1 >= n) atomicOr(&S->tail_dirty, 1u);
    }
    L.count += made;
    if (made && lane == 0) {
        d.iter_end[L.o] = L.base + L.count;
        atomicAdd(&S->n_links, made);
    }
    __syncwarp();
    return made < most;
}
// The candidates of sorted particle i (d < h, traversal order) handed to use(in, j, cell, d2)
// in chunks of a warp's width, by the 27-cell traversal: lane c < 27 loads cell c's range, the
// ranges are walked end to end in cell order, 4 x 32 entries in flight, and those within the
// support are packed in shared memory into full chunks.  use returns false to stop.
struct LinkGather {
    uint32_t e[64];                         // sorted index | cell << 25
    float d2[64];
    uint32_t first[27], begin[27];          // flattened position and sorted index of each cell's first member
};
template <class F>
__device__ __forceinline__ void link_candidates(const DevParams& P, const SetView& vd, uint32_t i, LinkGather& W, F&& use)
{
    const uint32_t lane = threadIdx.x & 31u, full = 0xffffffffu;
    const float3 p = vd.pos(i);
    const GCell g = grid_pos(P, p, vd.scene(i));
    uint32_t s = 0, cnt = 0;
    if (lane < 27u) {
        uint32_t e;
        if (vd.range(P, g, (int)(lane % 3u) - 1, (int)((lane / 3u) % 3u) - 1, (int)(lane / 9u) - 1, s, e))
            cnt = e > s ? e - s : 0u;
    }
    const uint32_t incl = warp_incl_scan(cnt);
    __syncwarp();
    if (lane < 27u) { W.first[lane] = incl - cnt; W.begin[lane] = s; }
    const uint32_t total = __shfl_sync(full, incl, 26);
    __syncwarp();
    uint32_t held = 0, cell = 0;
    bool more = true;
    for (uint32_t f0 = 0; f0 < total && more; f0 += 128u) {
        uint32_t en[4];
        float d2[4];
        bool in[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const uint32_t f = f0 + 32u * u + lane;
            in[u] = f < total;
            if (in[u]) {
                // the last cell that starts at or before f (a lane's f grows)
                while (cell < 26u && W.first[cell + 1u] <= f) ++cell;
                const uint32_t j = W.begin[cell] + (f - W.first[cell]);
                in[u] = j != i;
                en[u] = j | cell << 25;
                const float3 dv = sub3(p, vd.pos(j));
                d2[u] = dot3(dv, dv);
            }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const bool pass = more && in[u] && d2[u] < P.h2_lt;
            const uint32_t m = __ballot_sync(full, pass);
            if (pass) {
                const uint32_t at = held + __popc(m & ((1u << lane) - 1u));
                W.e[at] = en[u];
                W.d2[at] = d2[u];
            }
            held += __popc(m);
            __syncwarp();
            if (held >= 32u) {
                const uint32_t ce = W.e[lane], te = W.e[32u + lane];
                const float cd = W.d2[lane], td = W.d2[32u + lane];
                __syncwarp();
                held -= 32u;
                if (lane < held) { W.e[lane] = te; W.d2[lane] = td; }
                __syncwarp();
                more = use(true, ce & NL_J_MASK, ce >> 25, cd);
            }
        }
    }
    if (held && more) {
        const bool in = lane < held;
        const uint32_t ce = in ? W.e[lane] : 0u;
        use(in, ce & NL_J_MASK, ce >> 25, in ? W.d2[lane] : 0.f);
    }
    __syncwarp();
}
// k_link_filter with one warp per particle (small sets, maximum_connection <= SNOWB_MAXC_FAST): 32
// candidates at a time, each lane looking at its own partner (57 -> 16 us at 5,096 particles)
constexpr uint32_t LINK_TPB = 256;
__global__ void __launch_bounds__(128) k_link_filter_warp(DevParams P, DevState* S, SetView vd, snowb_particle_data dem,
                                                          int dynamic, uint8_t* __restrict__ active, NList L, SCList sc)
{
    wait_prior();
    __shared__ LinkGather gather[4];
    const uint32_t nd = S->n_dem, M = P.maxc, lane = threadIdx.x & 31u, full = 0xffffffffu;
    vd.n = nd;
    const bool lists = L.cnt != nullptr && S->changed == 0;
    WARP_LOOP(i, nd) {
        const uint32_t o = vd.gi[i], end = dem.iter_end[o];
        const uint32_t rk = lane < M ? dem.connect_record[o * M + lane] : LINK_NO_SLOT;
        bool act = end < o * M;     // a count below zero (dynamic caps): the pass decides
        if (!act && end - o * M < link_tolerance(P, dem.T[o], dynamic) && __any_sync(full, rk == SNOWB_UMAX)) {
            uint32_t skip_cell = 0xFFu;
            // false once a candidate that can change something is found
            auto look = [&](bool in, uint32_t o1, uint32_t cell) {
                const bool room = in && dem.iter_end[o1] < (o1 + 1u) * M;
                const bool before = in && cell != skip_cell;
                uint32_t dupm;
                const bool open = !link_ended(rk, skip_cell, in, o1, cell, dupm);
                // itself (stale cell range), unless an earlier linked candidate ended its cell
                const uint32_t same = __match_any_sync(full, before ? cell : 0x100u + lane);
                bool may = before && o1 == o && !(same & dupm & ((1u << lane) - 1u));
                if (open && room) may = may || has_free_slot(dem.connect_record, o1, M);
                act = __any_sync(full, may);
                return !act;
            };
            const uint32_t lc = lists ? L.cnt[L.cap + i] : NL_OVF;
            if (!(lc & NL_OVF)) {
                const uint32_t nl = lc & 1023u;
                bool more = true;
                for (uint32_t k0 = 0; k0 < nl && more; k0 += 32u) {
                    const bool in = k0 + lane < nl;
                    const uint32_t en = in ? L.e[(size_t)(k0 + lane) * L.stride + L.cap + i] : 0u;
                    more = look(in && !(en & NL_FAR), in ? vd.gi[en & NL_J_MASK] : 0u, (en >> 25) & 31u);
                }
            } else {
                link_candidates(P, vd, i, gather[threadIdx.x >> 5], [&](bool in, uint32_t j, uint32_t cell, float) {
                    return look(in, in ? vd.gi[j] : 0u, cell);
                });
            }
        }
        if (lane == 0u) {
            active[i] = act ? 1 : 0;
            if (act) {
                atomicAdd(&S->n_active, 1u);
                if (sc.flag) list_supercell(P, sc, vd.gh[i]);
            }
        }
    }
}
// One colour: a block takes a super-cell.  Its active particles link one after another in
// ascending sorted index, each by warp 0 (link_chunk); what a particle's links are chosen from
// -- its candidates -- never changes in the pass, so the block's warps fetch the candidates of
// LINK_BATCH active particles side by side into shared memory first.  They also leave out what
// can no longer link when the batch begins: links are only added and counts only grow in the
// pass, so a candidate that is linked already (with the rest of its cell) or whose count has
// reached the cap stays without effect.  A particle left without candidates costs nothing in
// the chain; the others' own slots, the partners' counts and slots and the writes remain.  (A
// particle with more than LINK_CAND of them has all candidates fetched in its turn.)
// README-scale set-up (every particle active, 64 to a super-cell): a colour takes about 180 us,
// 934 us with one warp per super-cell taking candidates one at a time; 415 us with link_chunk
// but the candidates fetched in the same warp's chain.
// L: the snow-snow candidate lists of the substep's first density pass (L.cnt null: none);
// they are valid while no phase change re-sorted the sets.
constexpr uint32_t LINK_BATCH = 32, LINK_CAND = 64;
__global__ void __launch_bounds__(LINK_TPB, 3) k_link_colour_warp(DevParams P, DevState* S, SetView vd,
                                                               snowb_particle_data dem,
                                                               const uint8_t* __restrict__ active, uint32_t colour,
                                                               int dynamic, NList L, SCList sc)
{
    wait_prior();
    __shared__ uint32_t c_e[LINK_BATCH][LINK_CAND];     // partner | cell << 25
    __shared__ float c_d[LINK_BATCH][LINK_CAND];        // distance
    __shared__ uint32_t a_i[LINK_BATCH], a_o[LINK_BATCH], a_tol[LINK_BATCH], a_n[LINK_BATCH];
    __shared__ LinkGather gather[LINK_TPB / 32];
    __shared__ LinkMap map;
    __shared__ uint32_t st[8], bs[8], s_total, s_next, s_held;
    vd.n = S->n_dem;
    const bool lists = L.cnt != nullptr && S->changed == 0;
    const uint32_t qx = P.gsx >> 2, qy = P.gsy >> 2, qz = P.gsz >> 2, M = P.maxc, full = 0xffffffffu;
    // the listed super-cells of this colour, or all of them
    const uint32_t total = sc.flag ? sc.count[colour] : qx * qy * qz;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    for (uint32_t w = blockIdx.x; w < total; w += gridDim.x) {
        const uint32_t t = sc.flag ? sc.list[colour * sc.per + w] : w;
        const uint32_t sx = 2u * (t % qx) + (colour & 1u);
        const uint32_t sy = 2u * ((t / qx) % qy) + ((colour >> 1) & 1u);
        const uint32_t sz = 2u * (t / (qx * qy)) + ((colour >> 2) & 1u);
        // The 8 cells (dz, dy, dx) in hash order -- ascending sorted index -- with lane c
        // loading cell c's range; the super-cell's particles are then taken in that order
        // (cell by cell, ascending index), as the cell-by-cell loops would.
        if (warp == 0) {
            uint32_t cb = 0, cn = 0;
            if (lane < 8u) {
                const uint32_t dz = lane >> 2, dy = (lane >> 1) & 1u, dx = lane & 1u;
                const uint32_t h = ((2u * sz + dz) * P.gsy + (2u * sy + dy)) * P.gsx + (2u * sx + dx);
                cn = current_range(vd, h, cb);
            }
            const uint32_t incl = warp_incl_scan(cn);
            if (lane < 8u) { st[lane] = incl - cn; bs[lane] = cb; }   // first flattened position of each cell
            if (lane == 7u) s_total = incl;
            if (lane == 0u) s_next = 0u;
        }
        __syncthreads();
        const uint32_t total_p = s_total;
        for (;;) {
            // warp 0: the next LINK_BATCH active particles
            if (warp == 0) {
                uint32_t held = 0, f0 = s_next;
                while (held < LINK_BATCH && f0 < total_p) {
                    const uint32_t f = f0 + lane;
                    uint32_t i = 0;
                    bool act = false;
                    if (f < total_p) {
                        // the last cell starting at or before f holds it (empty cells start
                        // where the next one does)
                        uint32_t c = 0;
#pragma unroll
                        for (uint32_t r = 1; r < 8u; ++r)
                            if (st[r] <= f) c = r;
                        i = bs[c] + (f - st[c]);
                        act = active[i] != 0;
                    }
                    const uint32_t am = __ballot_sync(full, act);
                    const uint32_t at = held + __popc(am & ((1u << lane) - 1u));
                    if (act && at < LINK_BATCH) a_i[at] = i;
                    const uint32_t over = __ballot_sync(full, act && at >= LINK_BATCH);
                    held = umin32(held + __popc(am), LINK_BATCH);
                    f0 += over ? (uint32_t)__ffs(over) - 1u : 32u;   // the first left out opens the next batch
                }
                if (lane == 0u) { s_next = f0; s_held = held; }
            }
            __syncthreads();
            const uint32_t held = s_held;
            if (held == 0u) break;
            for (uint32_t a = warp; a < held; a += nwarps) {
                const uint32_t i = a_i[a];
                const uint32_t o = vd.gi[i], tol = link_tolerance(P, dem.T[o], dynamic);
                const uint32_t rk = lane < M ? dem.connect_record[o * M + lane] : LINK_NO_SLOT;
                const uint32_t lc = lists ? L.cnt[L.cap + i] : NL_OVF;
                uint32_t got = 0, skip_cell = 0xFFu;
                auto keep = [&](bool in, uint32_t o1, uint32_t cell, float dist) {
                    const bool room = in && dem.iter_end[o1] < (o1 + 1u) * M;
                    uint32_t dupm;
                    in = !link_ended(rk, skip_cell, in, o1, cell, dupm) && room;
                    const uint32_t m = __ballot_sync(full, in), k = got + __popc(m & ((1u << lane) - 1u));
                    if (in && k < LINK_CAND) { c_e[a][k] = o1 | cell << 25; c_d[a][k] = dist; }
                    got += __popc(m);
                    return got <= LINK_CAND;
                };
                const uint32_t end = dem.iter_end[o];
                if ((end >= o * M && end - o * M >= tol) || !__any_sync(full, rk == SNOWB_UMAX)) {
                    // at its cap (a count below zero, which dynamic caps can leave, may rise
                    // past zero in this pass) or out of slots
                } else if (!(lc & NL_OVF)) {
                    const float3 p = vd.pos(i);
                    const uint32_t nl = lc & 1023u;
                    bool more = true;
                    for (uint32_t k0 = 0; k0 < nl && more; k0 += 32u) {
                        const bool in = k0 + lane < nl;
                        const uint32_t en = in ? L.e[(size_t)(k0 + lane) * L.stride + L.cap + i] : 0u, j = en & NL_J_MASK;
                        more = keep(in && !(en & NL_FAR), in ? vd.gi[j] : 0u, (en >> 25) & 31u,
                                    in ? len3(sub3(p, vd.pos(j))) : 0.f);
                    }
                } else {
                    link_candidates(P, vd, i, gather[warp], [&](bool in, uint32_t j, uint32_t cell, float d2) {
                        return keep(in, in ? vd.gi[j] : 0u, cell, sqrtf(d2));
                    });
                }
                if (lane == 0u) { a_o[a] = o; a_tol[a] = tol; a_n[a] = got; }
            }
            __syncthreads();
            if (warp == 0)
                for (uint32_t a = 0; a < held; ++a) {
                    const uint32_t o = a_o[a], got = a_n[a];
                    if (got == 0u) continue;
                    LinkState l{o, o * M, a_tol[a], dem.iter_end[o] - o * M, 0xFFu,
                                lane < M ? dem.connect_record[o * M + lane] : LINK_NO_SLOT};
                    if (got <= LINK_CAND) {
                        bool more = true;
                        for (uint32_t k0 = 0; k0 < got && more; k0 += 32u) {
                            const uint32_t k = k0 + lane;
                            const bool in = k < got;
                            const uint32_t en = in ? c_e[a][k] : 0u;
                            more = link_chunk(P, dem, S, vd.n, l, map, in, en & NL_J_MASK, en >> 25, in ? c_d[a][k] : 0.f);
                        }
                    } else if (lists && !(L.cnt[L.cap + a_i[a]] & NL_OVF)) {
                        const uint32_t i = a_i[a];
                        const float3 p = vd.pos(i);
                        const uint32_t nl = L.cnt[L.cap + i] & 1023u;
                        bool more = true;
                        for (uint32_t k0 = 0; k0 < nl && more; k0 += 32u) {
                            const uint32_t k = k0 + lane;
                            const bool in = k < nl;
                            const uint32_t en = in ? L.e[(size_t)k * L.stride + L.cap + i] : 0u, j = en & NL_J_MASK;
                            more = link_chunk(P, dem, S, vd.n, l, map, in && !(en & NL_FAR), in ? vd.gi[j] : 0u,
                                              (en >> 25) & 31u, in ? len3(sub3(p, vd.pos(j))) : 0.f);
                        }
                    } else {
                        link_candidates(P, vd, a_i[a], gather[0], [&](bool in, uint32_t j, uint32_t cell, float d2) {
                            return link_chunk(P, dem, S, vd.n, l, map, in, in ? vd.gi[j] : 0u, cell, sqrtf(d2));
                        });
                    }
                }
            __syncthreads();
        }
        if (sc.flag && threadIdx.x == 0) sc.flag[colour * sc.per + t] = 0u;   // ready for the next pass
        __syncthreads();
    }
}
// connect_and_record_cell (:4127-4252) + connect_and_record_d (:4255-4284) for one particle, the
// sequential rule as it stands with every access in memory (maximum_connection > SNOWB_MAXC_FAST)
__device__ void link_particle(const DevParams& P, const SetView& vd, const snowb_particle_data& d, uint32_t i,
                              int dynamic, DevState* S)
{
    const uint32_t M = P.maxc;
    const float3 p = vd.pos(i);
    const uint32_t o = vd.gi[i];
    const GCell g = grid_pos(P, p, vd.scene(i));
    const float T = d.T[o];
    FOR27 {
        uint32_t s, e;
        if (!vd.range(P, g, ox, oy, oz, s, e)) continue;
        for (uint32_t j = s; j < e; ++j) {
            if (j == i) continue;
            const uint32_t o1 = vd.gi[j];
            const float dist = len3(sub3(p, vd.pos(j)));
            const uint32_t count = d.iter_end[o] - o * M;
            const uint32_t tol = link_tolerance(P, T, dynamic);
            if (dist < P.h && count < tol) {
                bool dup = false;
                for (uint32_t q = M * o; q < M * (o + 1); ++q)
                    if (d.connect_record[q] == o1) { dup = true; break; }
                if (dup) break;   // the reference returns from the cell helper
                for (uint32_t q = M * o; q < M * (o + 1); ++q) {
                    if (d.connect_record[q] == SNOWB_UMAX) {
                        d.connect_record[q] = o1;
                        bool valid = false;
                        if (d.iter_end[o1] < (o1 + 1) * M)
                            for (uint32_t r = o1 * M; r < (o1 + 1) * M; ++r)
                                if (d.connect_record[r] == SNOWB_UMAX) {
                                    d.connect_record[r] = o;
                                    d.connect_length[r] = dist;
                                    d.iter_end[o1]++;
                                    if (o1 >= vd.n) atomicOr(&S->tail_dirty, 1u);
                                    valid = true;
                                    break;
                                }
                        if (valid) { d.connect_length[q] = dist; d.iter_end[o]++; atomicAdd(&S->n_links, 1u); }
                        else d.connect_record[q] = SNOWB_UMAX;
                        break;
                    }
                }
            }
        }
    }
}
// Link formation's copy of the snow set's sorted view (the arrays its passes read: the
// sorted copies, grid index and hash, and the cell table), taken after the sort point before it, so that the first iteration's sort point may rewrite the
// set's view while link formation runs.  `full` entries of the particle arrays (the
// caller's arrays hold that many), `ncells` of the cell table.
__global__ void k_copy_link_view(SetView v, uint32_t full, uint32_t ncells, float4* __restrict__ p4,
                                 snowb_float3* __restrict__ sp, uint32_t* __restrict__ gi,
                                 uint32_t* __restrict__ gh, uint32_t* __restrict__ sid, uint32_t* __restrict__ cs,
                                 uint32_t* __restrict__ ce)
{
    wait_prior();
    const uint32_t m = full > ncells ? full : ncells;
    GRID_LOOP(k, m) {
        if (k < full) {
            p4[k] = v.p4[k];
            sp[k] = v.sp[k];
            gi[k] = v.gi[k];
            gh[k] = v.gh[k];
            if (v.sid) sid[k] = v.sid[k];
        }
        if (k < ncells) { cs[k] = v.cs[k]; ce[k] = v.ce[k]; }
    }
}
// one colour: one thread per super-cell of that colour (maximum_connection > SNOWB_MAXC_FAST)
__global__ void k_link_colour(DevParams P, DevState* S, SetView vd, snowb_particle_data dem,
                              const uint8_t* __restrict__ active, uint32_t colour, int dynamic)
{
    wait_prior();
    vd.n = S->n_dem;
    const uint32_t qx = P.gsx >> 2, qy = P.gsy >> 2, qz = P.gsz >> 2;
    const uint32_t total = qx * qy * qz;
    GRID_LOOP(t, total) {
        const uint32_t sx = 2u * (t % qx) + (colour & 1u);
        const uint32_t sy = 2u * ((t / qx) % qy) + ((colour >> 1) & 1u);
        const uint32_t sz = 2u * (t / (qx * qy)) + ((colour >> 2) & 1u);
        for (uint32_t dz = 0; dz < 2; ++dz)
            for (uint32_t dy = 0; dy < 2; ++dy)
                for (uint32_t dx = 0; dx < 2; ++dx) {
                    const uint32_t h = ((2u * sz + dz) * P.gsy + (2u * sy + dy)) * P.gsx + (2u * sx + dx);
                    uint32_t b = 0;
                    const uint32_t n = current_range(vd, h, b);
                    for (uint32_t i = b; i < b + n; ++i)
                        if (active[i]) link_particle(P, vd, dem, i, dynamic, S);
                }
    }
}
// adjust_connections_d (:4768-4808) in ascending index order (single thread).  The
// reference indexes the partner's slots with an empty record once the count exceeds the
// cap (an out-of-bounds read); that partner loop is skipped here.
__global__ void k_adjust_links(DevParams P, DevState* S, snowb_particle_data d, uint32_t full)
{
    wait_prior();
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    const uint32_t n = S->n_dem, M = P.maxc;
    for (uint32_t i = 0; i < n; ++i) {
        uint32_t cm = __float2uint_rz(((d.T[i] - P.Tf) / (P.Th - P.Tf)) * (float)M);
        if (cm > M) cm = M;
        uint32_t count = 0;
        for (uint32_t s = M * i; s < M * (i + 1); ++s) {
            count = d.connect_record[s] != SNOWB_UMAX ? count + 1 : count;
            if (count > cm) {
                const uint32_t j = d.connect_record[s];
                d.connect_record[s] = SNOWB_UMAX;
                d.connect_length[s] = 0.f;
                d.iter_end[i]--;
                if (j == SNOWB_UMAX || j >= full) continue;
                if (j >= n) S->tail_dirty = 1u;
                for (uint32_t q = M * j; q < M * (j + 1); ++q)
                    if (d.connect_record[q] == i) {
                        d.connect_record[q] = SNOWB_UMAX; d.connect_length[q] = 0.f; d.iter_end[j]--;
                    }
            }
        }
    }
}

}  // namespace snowb
