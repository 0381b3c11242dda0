// sort.cuh -- neighbor structure: cell hashing, a stable counting sort of cell hashes,
// and the cell table (cuda_simulation.cu:194-301, :359-420, :1455-1468).
//
// The reference sorts (hash, index) pairs with thrust::sort_by_key, which is stable.
// This is a counting sort over the num_cells cell keys that yields the same
// permutation:
//   1. hash + count: each particle's cell key, and an (unordered) slot in its cell
//      from an atomic counter;
//   2. exclusive scan of the per-cell counts of the occupied scan chunks; the same pass
//      re-zeroes the counters and clears cell_start over the range the reference clears;
//   3. scatter each particle into its cell's range (unordered inside the cell);
//   4. rank inside the cell by original index (cells hold a handful of particles),
//      which restores the stable order, then write every output of the reference's
//      reorder pass (grid_hash, grid_index, cell_start/cell_end of occupied cells,
//      sorted_pos) plus the compact float4 copy used by the neighbor loops.
#pragma once
#include "common.cuh"

namespace snowb {

constexpr int SCAN_TPB = 256;                 // threads per scan block
constexpr int SCAN_ITEMS = 4;                 // entries per thread
constexpr int SCAN_CHUNK = SCAN_TPB * SCAN_ITEMS;

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v)
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}
__device__ __forceinline__ uint32_t warp_sum(uint32_t v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Block-wide exclusive scan of one value per thread (blockDim.x == SCAN_TPB).
__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t* sm, uint32_t& total)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t inc = warp_incl_scan(v);
    if (lane == 31) sm[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = lane < SCAN_TPB / 32 ? sm[lane] : 0u;
        uint32_t wi = warp_incl_scan(w);
        if (lane < SCAN_TPB / 32) sm[lane] = wi - w;
        if (lane == SCAN_TPB / 32 - 1) sm[SCAN_TPB / 32] = wi;
    }
    __syncthreads();
    uint32_t r = sm[warp] + inc - v;
    total = sm[SCAN_TPB / 32];
    __syncthreads();
    return r;
}

// Sum of the first `count` block sums, computed by every thread of warp 0.
__device__ __forceinline__ uint32_t prefix_of_blocks(const uint32_t* bsum, uint32_t count)
{
    uint32_t s = 0;
    for (uint32_t k = threadIdx.x & 31; k < count; k += 32) s += bsum[k];
    return warp_sum(s);
}

// One or two sets sorted by the same four launches (the water and the snow set of a sort
// point): the particle passes run over both sets' particles end to end, the scan over both
// cell tables.  Two chains of launches on two streams, forked and joined at each sort point, were
// 56 launches and 32 event calls a substep; these are 32 launches at its eight sort points
// (issuing a substep: 330 -> 230 us of host time; one substep of 208 particles 512 -> 480 us).
struct SortSide {
    const snowb_float3* pos;
    const float *w, *invm, *contrib;      // mass, massInv, contrib by original index
    const uint32_t* n;                    // set size (device)
    uint32_t *key, *slot, *tmp, *cnt, *off;
    uint32_t* bsum;                       // particles per scan chunk; zero between sorts
    uint32_t* dirty;                      // per scan chunk: its part of cell_start may hold entries
    const uint32_t* sid_o;                // scene ids by original index (batched runs) or null
    uint32_t* sid_s;
    snowb_cell_data cd;
    float4* p4;
    float *invm_s, *contrib_s;
};
struct SortPair {
    SortSide a[2];
    int on[2];                            // set k is sorted
    // A sort point of the substep decides for itself (S set): the hash pass turns a set's moved
    // flag into the decision (DevState::resort, read by the later passes; the scan pass clears the
    // flag); a set that keeps its last sort only has its gathered outputs refreshed.  The first
    // sort point of a substep also opens it (begin).  S null: both sets sort in full.
    DevState* S;
    int begin;
    uint32_t ncells;
    int clear_all;
    const float4* skin_p4;                // see NL_SKIN
    uint32_t* skin_far;
    __device__ __forceinline__ bool sorts(int k) const { return on[k] && (!S || S->resort[k] != 0u); }
    __device__ __forceinline__ uint32_t size(int k) const { return on[k] ? *a[k].n : 0u; }
};

// ------------------------------------------------------------------ 1. hash + count
// Hash of pos[o] (calcHashD :194-212) and its cell's and scan chunk's counts (one chunk atomic
// per chunk and warp), which the cell scan needs; the scatter pass re-zeroes the chunk counts.
// substep start: launch sizes, phase-change and link counters
__device__ __forceinline__ void begin_substep(DevState* S)
{
    S->n0_sph = S->n_sph; S->n0_dem = S->n_dem;
    S->n_freeze = 0; S->n_melt = 0; S->changed = 0; S->n_active = 0; S->n_links = 0; S->n_nl_ovf = 0;
    S->skin_ok = 0; ++S->epoch;
    for (int c = 0; c < 8; ++c) S->sc_count[c] = 0u;
}
__global__ void k_sort_hash(DevParams P, const __grid_constant__ SortPair Q)
{
    wait_prior();
    uint32_t m[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) m[k] = !Q.on[k] ? 0u : (Q.S ? Q.S->moved[k] : 1u);
    if (Q.S && blockIdx.x == 0 && threadIdx.x == 0) {
        if (Q.begin) begin_substep(Q.S);
#pragma unroll
        for (int k = 0; k < 2; ++k)
            if (Q.on[k]) {
                Q.S->resort[k] = m[k];
                if (m[k]) ++Q.S->sorts_full[k];
                else ++Q.S->sorts_kept[k];
            }
    }
    if (Q.S && m[1] && blockIdx.x == 0 && threadIdx.x == 0) Q.S->skin_ok = 0u;   // the lists hold sorted indices
    const uint32_t n0 = m[0] ? Q.size(0) : 0u, n = n0 + (m[1] ? Q.size(1) : 0u);
    const uint32_t lane = threadIdx.x & 31u;
    // whole warps iterate together so the chunk counts can be aggregated with warp votes
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t base = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < n; base += stride) {
        const uint32_t t = base + lane;
        const int k = t < n0 ? 0 : 1;
        const SortSide& A = Q.a[k];
        const uint32_t o = k ? t - n0 : t;
        const bool live = t < n;
        uint32_t chunk = 0xFFFFFFFFu;
        if (live) {
            const uint32_t h = grid_hash(P, grid_pos(P, ldv3(A.pos, o), A.sid_o ? A.sid_o[o] : 0u), 0, 0, 0);
            A.key[o] = h;
            A.slot[o] = atomicAdd(A.cnt + h, 1u);
            chunk = h / (uint32_t)SCAN_CHUNK;
        }
        const uint32_t peers = __match_any_sync(0xffffffffu, chunk | (uint32_t)k << 30);
        if (live && lane == (uint32_t)(__ffs(peers) - 1)) atomicAdd(A.bsum + chunk, (uint32_t)__popc(peers));
    }
}
// sort_particles path: keys and values already in (grid_hash, grid_index).
__global__ void k_key_count(const uint32_t* __restrict__ keys, const uint32_t* __restrict__ vals, uint32_t n,
                            uint32_t ncells, uint32_t* __restrict__ key_o, uint32_t* __restrict__ val_o,
                            uint32_t* __restrict__ slot_o, uint32_t* __restrict__ cnt, uint32_t* err)
{
    wait_prior();
    GRID_LOOP(i, n) {
        uint32_t h = keys[i];
        if (h >= ncells) { atomicOr(err, 2u); h = ncells - 1; }
        key_o[i] = h;
        val_o[i] = vals[i];
        slot_o[i] = atomicAdd(cnt + h, 1u);
    }
}

// ------------------------------------------------------------------ 2. scan of counts
__global__ void k_block_sums(const uint32_t* __restrict__ cnt, uint32_t ncells, uint32_t* __restrict__ bsum)
{
    wait_prior();
    __shared__ uint32_t sm[SCAN_TPB / 32];
    const uint32_t base = blockIdx.x * SCAN_CHUNK + threadIdx.x * SCAN_ITEMS;
    uint32_t s = 0;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k)
        if (base + k < ncells) s += cnt[base + k];
    s = warp_sum(s);
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x < 32) {
        uint32_t v = threadIdx.x < SCAN_TPB / 32 ? sm[threadIdx.x] : 0u;
        v = warp_sum(v);
        if (threadIdx.x == 0) bsum[blockIdx.x] = v;
    }
}

// off[c] = exclusive prefix of cnt (c <= ncells), cnt re-zeroed, for the scan chunk `chunk`; bsum:
// the counts of the chunks, of which the block's threads sum those before it side by side, in the
// same steps as the scan; cells from `clear` on keep their cell_start (null: none is cleared)
struct ScanShared {
    uint32_t scan[SCAN_TPB / 32 + 1], before[SCAN_TPB / 32];
};
__device__ __forceinline__ void scan_chunk(uint32_t* __restrict__ cnt, uint32_t ncells, uint32_t* __restrict__ off,
                                           uint32_t* __restrict__ cell_start, uint32_t clear, uint32_t chunk,
                                           const uint32_t* bsum, ScanShared& sm)
{
    const uint32_t base = chunk * SCAN_CHUNK + threadIdx.x * SCAN_ITEMS;
    uint32_t before = 0;
    for (uint32_t c = threadIdx.x; c < chunk; c += SCAN_TPB) before += bsum[c];
    uint32_t v[SCAN_ITEMS], t = 0;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        v[k] = base + k < ncells ? cnt[base + k] : 0u;
        t += v[k];
    }
    before = warp_sum(before);
    if ((threadIdx.x & 31) == 0) sm.before[threadIdx.x >> 5] = before;
    uint32_t total;
    uint32_t ex = block_excl_scan(t, sm.scan, total);   // its barriers cover sm.before too
#pragma unroll
    for (int w = 0; w < SCAN_TPB / 32; ++w) ex += sm.before[w];
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        const uint32_t c = base + k;
        if (c < ncells) {
            off[c] = ex;
            cnt[c] = 0u;
            if (cell_start && c < clear) cell_start[c] = SNOWB_EMPTY;
            // the chunk's end: the next chunk, if it is walked, writes the same value
            if (c == ncells - 1 || (k == SCAN_ITEMS - 1 && threadIdx.x == SCAN_TPB - 1)) off[c + 1] = ex + v[k];
        }
        ex += v[k];
    }
}
// sort_particles path: every chunk, no cell table
__global__ void k_cell_scan(uint32_t* __restrict__ cnt, const uint32_t* __restrict__ bsum, uint32_t ncells,
                            uint32_t* __restrict__ off)
{
    wait_prior();
    __shared__ ScanShared sm;
    scan_chunk(cnt, ncells, off, nullptr, 0u, blockIdx.x, bsum, sm);
}
// A block takes a scan chunk of a set.  A chunk without particles only has its part of
// cell_start cleared, if entries may be left there (dirty); its offsets are not written, and no
// pass reads them: most chunks of a batch's wide grid, or above a scene, are empty (32 scenes,
// 8,192 chunks, where every block also summed all earlier chunks: 79 us a set, 27 us both).
// cell_start is cleared for c < clear (min(n, ncells) reproduces the reference's partial memset, Q1).
__global__ void __launch_bounds__(SCAN_TPB) k_sort_scan(const __grid_constant__ SortPair Q, uint32_t chunks)
{
    wait_prior();
    __shared__ ScanShared sm;
    const int k = blockIdx.x < chunks ? 0 : 1;
    const uint32_t chunk = blockIdx.x - (k ? chunks : 0u);
    const SortSide& A = Q.a[k];
    if (Q.S && Q.on[k] && chunk == 0 && threadIdx.x == 0) Q.S->moved[k] = 0u;   // the hash pass has read it
    if (!Q.sorts(k)) return;
    const uint32_t here = A.bsum[chunk], begin = chunk * SCAN_CHUNK, end = umin32(begin + SCAN_CHUNK, Q.ncells);
    const uint32_t clear = Q.clear_all ? Q.ncells : umin32(Q.size(k), Q.ncells);
    const bool dirty = !Q.S || Q.S->table_any[k] != 0u || A.dirty[chunk] != 0u;
    if (here == 0u) {
        if (dirty)
            for (uint32_t c = begin + threadIdx.x; c < umin32(end, clear); c += SCAN_TPB) A.cd.cell_start[c] = SNOWB_EMPTY;
        __syncthreads();
        if (threadIdx.x == 0) A.dirty[chunk] = dirty && end > clear ? 1u : 0u;
        return;
    }
    if (threadIdx.x == 0) A.dirty[chunk] = 1u;
    scan_chunk(A.cnt, Q.ncells, A.off, A.cd.cell_start, clear, chunk, A.bsum, sm);
}

// ------------------------------------------------------------------ 3. scatter
__global__ void k_scatter(const uint32_t* __restrict__ key_o, const uint32_t* __restrict__ slot_o,
                          const uint32_t* __restrict__ off, uint32_t* __restrict__ tmp, uint32_t n)
{
    wait_prior();
    GRID_LOOP(o, n) tmp[off[key_o[o]] + slot_o[o]] = o;
}
__global__ void k_sort_scatter(const __grid_constant__ SortPair Q, uint32_t chunks)
{
    wait_prior();
    const bool s0 = Q.sorts(0), s1 = Q.sorts(1);
    if (Q.S && blockIdx.x == 0 && threadIdx.x == 0) {   // the scan pass has cleared what was left in the tables
        if (s0) Q.S->table_any[0] = 0u;
        if (s1) Q.S->table_any[1] = 0u;
    }
    const uint32_t n0 = s0 ? Q.size(0) : 0u, n = n0 + (s1 ? Q.size(1) : 0u);
    GRID_LOOP(t, n) {
        const int k = t < n0 ? 0 : 1;
        const SortSide& A = Q.a[k];
        const uint32_t o = k ? t - n0 : t;
        A.tmp[A.off[A.key[o]] + A.slot[o]] = o;
    }
    GRID_LOOP(c, chunks) {
        if (s0) Q.a[0].bsum[c] = 0u;
        if (s1) Q.a[1].bsum[c] = 0u;
    }
}

// rank of element o among the (unordered) members of its cell, by ascending o
__device__ __forceinline__ uint32_t stable_rank(const uint32_t* __restrict__ tmp, uint32_t b, uint32_t e, uint32_t o)
{
    uint32_t r = 0;
    for (uint32_t k = b; k < e; ++k) r += tmp[k] < o;
    return r;
}

// ------------------------------------------------------------------ 4. rank + outputs
// Fused path (sort_and_reorder :398-420 with hash = cell of pos).  Also gathers the
// compact sorted attributes: p4 = (pos, w[o]), invm_s, contrib_s.  A set that keeps its last
// sort (no particle left its cell, same set size): grid_hash, grid_index and the cell table are
// already what this sort would write, so only the gathered outputs are refreshed, sorted slot
// by sorted slot.
__global__ void k_sort_rank(DevParams P, const __grid_constant__ SortPair Q)
{
    wait_prior();
    const bool s0 = Q.sorts(0), s1 = Q.sorts(1);
    const uint32_t n0 = Q.size(0), n = n0 + Q.size(1);
    const bool skin = Q.S && Q.on[1] && !s1 && Q.S->skin_ok != 0u;
    GRID_LOOP(t, n) {
        const int k = t < n0 ? 0 : 1;
        const SortSide& A = Q.a[k];
        uint32_t o, p;
        if (k ? s1 : s0) {
            o = k ? t - n0 : t;
            const uint32_t h = A.key[o], b = A.off[h], e = A.off[h + 1], r = stable_rank(A.tmp, b, e, o);
            p = b + r;
            A.cd.grid_index[p] = o;
            A.cd.grid_hash[p] = h;
            if (r == 0) { A.cd.cell_start[h] = b; A.cd.cell_end[h] = e; }
        } else {
            p = k ? t - n0 : t;
            o = A.cd.grid_index[p];
        }
        const float3 q = ldv3(A.pos, o);
        if (k && skin) {
            const float3 d = sub3(q, xyz(Q.skin_p4[p]));
            if (!(dot3(d, d) <= P.skin_move2)) {   // the lists of the cells around are not to be used
                const Nbhd nb = make_nbhd(P, grid_pos(P, q, A.sid_o ? A.sid_o[o] : 0u), q, 0.f);
                const uint32_t now = Q.S->epoch;
                FOR27 Q.skin_far[nb.hash(ox, oy, oz)] = now;
                atomicAdd(&Q.S->skin_marks, 1u);
            }
        }
        st3(A.cd.sorted_pos, p, q);
        A.p4[p] = make_float4(q.x, q.y, q.z, A.w[o]);
        A.invm_s[p] = A.invm[o];
        A.contrib_s[p] = A.contrib[o];
        if (A.sid_s) A.sid_s[p] = A.sid_o[o];
    }
}
// A set whose particles all kept their cells since its last sort sorts to the same
// permutation and cell table, so only the gathered outputs change: the kernels that move
// particles compare each new cell with the particle's key at the last sort and mark the
// set when one differs.
struct SortTrack {
    const uint32_t* key;        // cell key per original index at the set's last sort (null: no tracking)
    const uint32_t* sid;        // scene id per original index (batched runs) or null
    uint32_t* moved;            // &DevState::moved[set]
};
__device__ __forceinline__ void track_move(const DevParams& P, const SortTrack& T, uint32_t o, float3 q,
                                           uint32_t scene)
{
    if (grid_hash(P, grid_pos(P, q, scene), 0, 0, 0) != __ldg(T.key + o)) *T.moved = 1u;
}
// sort_particles path: write the sorted keys and values only.
__global__ void k_rank_pairs(const uint32_t* __restrict__ key_o, const uint32_t* __restrict__ val_o,
                             const uint32_t* __restrict__ off, const uint32_t* __restrict__ tmp,
                             uint32_t* __restrict__ keys, uint32_t* __restrict__ vals, uint32_t n)
{
    wait_prior();
    GRID_LOOP(i, n) {
        const uint32_t h = key_o[i], b = off[h], e = off[h + 1];
        const uint32_t p = b + stable_rank(tmp, b, e, i);
        keys[p] = h;
        vals[p] = val_o[i];
    }
}

// calcHashD (:194-212) alone
__global__ void k_calc_hash(DevParams P, snowb_cell_data cd, const snowb_float3* __restrict__ pos, uint32_t n,
                            const uint32_t* __restrict__ sid_o)
{
    wait_prior();
    GRID_LOOP(i, n) {
        float3 p = ldv3(pos, i);
        cd.grid_hash[i] = grid_hash(P, grid_pos(P, p, sid_o ? sid_o[i] : 0u), 0, 0, 0);
        cd.grid_index[i] = i;
    }
}
// reorderDataAndFindCellStartD (:242-301) alone; cell_start cleared beforehand
__global__ void k_reorder(snowb_cell_data cd, const snowb_float3* __restrict__ pos, uint32_t n)
{
    wait_prior();
    GRID_LOOP(i, n) {
        const uint32_t h = cd.grid_hash[i];
        if (i == 0 || h != cd.grid_hash[i - 1]) {
            cd.cell_start[h] = i;
            if (i > 0) cd.cell_end[cd.grid_hash[i - 1]] = i;
        }
        if (i == n - 1) cd.cell_end[h] = i + 1;
        st3(cd.sorted_pos, i, ldv3(pos, cd.grid_index[i]));
    }
}
// ------------------------------------------------------------------ generic scan
// Exclusive scans of two arrays in[0, n) into out, totals into *total, by the same two launches
// (blocks [0, blocks) take the first array, the rest the second).
struct ScanSide {
    const uint32_t* in;
    const uint32_t* n_ptr;     // null: n
    uint32_t n;
    uint32_t *bsum, *out, *total;
};
struct ScanPair {
    ScanSide a[2];
};
__global__ void k_scan_sums(const __grid_constant__ ScanPair Q, uint32_t blocks)
{
    wait_prior();
    const int k = blockIdx.x < blocks ? 0 : 1;
    const ScanSide& A = Q.a[k];
    const uint32_t b = blockIdx.x - (k ? blocks : 0u), n = A.n_ptr ? *A.n_ptr : A.n;
    __shared__ uint32_t sm[SCAN_TPB / 32];
    const uint32_t base = b * SCAN_CHUNK + threadIdx.x * SCAN_ITEMS;
    if (b * SCAN_CHUNK >= n && b != 0) { if (threadIdx.x == 0) A.bsum[b] = 0; return; }
    uint32_t s = 0;
#pragma unroll
    for (int k2 = 0; k2 < SCAN_ITEMS; ++k2)
        if (base + k2 < n) s += A.in[base + k2];
    s = warp_sum(s);
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x < 32) {
        uint32_t v = threadIdx.x < SCAN_TPB / 32 ? sm[threadIdx.x] : 0u;
        v = warp_sum(v);
        if (threadIdx.x == 0) A.bsum[b] = v;
    }
}
__global__ void k_scan_apply(const __grid_constant__ ScanPair Q, uint32_t blocks)
{
    wait_prior();
    const int k = blockIdx.x < blocks ? 0 : 1;
    const ScanSide& A = Q.a[k];
    const uint32_t b = blockIdx.x - (k ? blocks : 0u), n = A.n_ptr ? *A.n_ptr : A.n;
    if (n == 0) { if (b == 0 && threadIdx.x == 0) *A.total = 0; return; }
    if (b >= (n + SCAN_CHUNK - 1) / SCAN_CHUNK) return;
    __shared__ uint32_t sm[SCAN_TPB / 32 + 1];
    __shared__ uint32_t s_prefix;
    if (threadIdx.x < 32) {
        uint32_t p = prefix_of_blocks(A.bsum, b);
        if (threadIdx.x == 0) s_prefix = p;
    }
    const uint32_t base = b * SCAN_CHUNK + threadIdx.x * SCAN_ITEMS;
    uint32_t v[SCAN_ITEMS], t = 0;
#pragma unroll
    for (int k2 = 0; k2 < SCAN_ITEMS; ++k2) {
        v[k2] = base + k2 < n ? A.in[base + k2] : 0u;
        t += v[k2];
    }
    uint32_t tot;
    __syncthreads();
    uint32_t ex = block_excl_scan(t, sm, tot) + s_prefix;
#pragma unroll
    for (int k2 = 0; k2 < SCAN_ITEMS; ++k2) {
        if (base + k2 < n) {
            A.out[base + k2] = ex;
            if (base + k2 == n - 1) *A.total = ex + v[k2];
        }
        ex += v[k2];
    }
}

}  // namespace snowb
