// adjoint.cuh -- reverse-mode kernels of the substep (the project's adjoint; the reference
// has none).
//
// The adjoint differentiates the substep as the forward kernels compute it in the fixed
// quirk mode, with every discrete decision of the forward pass held fixed: neighbour sets
// (support tests d < h, d < 2r, d <= 2r), interlink topology (records snapshotted at each
// iteration) and link-breaking masks, the C > 0 clamp, the friction static/kinetic branch,
// wall reflections, the floor clamp and the speed clamp.  No particle changes phase inside
// a differentiated substep and every contrib is 1 (the fields the adjoint assumes).
//
// All adjoint and field arrays are in original index order (like the caller's state); the
// gathers run over the sorted views of the positions being differentiated, over the
// neighbours of the forward loops.  Every kernel is a gather: a particle accumulates every
// term in which it takes part, from its own constraint and from its neighbours', so no
// atomics are needed except for the scalar parameter gradients.
//
// The neighbour passes run one warp per particle (warp_neighbors) where one thread each leaves most
// of the GPU idle while it walks up to 81 cells one candidate after another (9,216 particles, us a
// launch: fields 90 -> 43, lambda adjoint 99 -> 19, positions 130 -> 43, friction 81 -> 25, XSPH
// 79 -> 20, heat 94 -> 31), and one thread per particle above ADJ_WARP_MAX.
//
// Notation: r = x_i - x_j, d = |r|.  For a radial vector function F(r) = f(d) r its
// Jacobian is J = f I + (f'(d)/d) r r^T (symmetric, even in r).
#pragma once
#include "common.cuh"
#include "solver.cuh"

namespace snowb {

// fields and their adjoints, one block per particle set (water, snow, boundary)
struct AdjField {
    float *rho, *C, *S, *lam;     // density, constraint, gradient-square sum, lambda
    float *lamb, *rhob, *Sb;      // adjoints of lambda, rho, S
};
// reverse-pass arrays of the water and snow sets (float3 arrays as snowb_float3)
struct AdjSet {
    snowb_float3* xb;     // adjoint of the positions being differentiated
    snowb_float3* u;      // sor * adjoint of the corrected positions (input of the constraint reverse)
    snowb_float3* x0b;    // adjoint of the substep-start positions after integration (friction, finalize)
    const snowb_float3* x0p;   // those positions (tape)
};
// scalar parameter gradients, accumulated in double
struct AdjParams {
    double* g;   // [0] k_refreezing (interlink), [1] k_stretch, [2] k_water, [3] k_snow
};

__device__ __forceinline__ float3 mv3(float a, float3 x, float b, float3 r, float rx)
{
    // (a I + b r r^T) x with rx = r . x
    return f3(a * x.x + b * r.x * rx, a * x.y + b * r.y * rx, a * x.z + b * r.z * rx);
}
// J_spiky(r) y
__device__ __forceinline__ float3 jv_spiky(const DevParams& P, float3 r, float d, float3 y)
{
    const float q = P.h - d, de = d + P.keps;
    const float f = P.spiky_G * (q * q / de);
    const float fp = P.spiky_G * (-2.f * q / de - (q * q) / (de * de));
    const float b = d > 0.f ? fp / d : 0.f;
    return mv3(f, y, b, r, dot3(r, y));
}
// J_poly6-gradient(r) y   (G_poly6 = pG (h^2-d^2)^2 r)
__device__ __forceinline__ float3 jv_gpoly6(const DevParams& P, float3 r, float d, float3 y)
{
    const float q = P.h * P.h - d * d;
    const float f = P.poly6_G * q * q;
    const float b = -4.f * P.poly6_G * q;   // f'(d)/d
    return mv3(f, y, b, r, dot3(r, y));
}
// contact direction phi(r) = (d - 2r)/(d + eps) r and its Jacobian
__device__ __forceinline__ float3 phi_contact(const DevParams& P, float3 r, float d)
{
    return sc3((d - P.two_r) / (d + P.pbd_eps), r);
}
__device__ __forceinline__ float3 jv_contact(const DevParams& P, float3 r, float d, float3 y, float L)
{
    // L = rest length (2r for contact, the link length for interlinks)
    const float de = d + P.pbd_eps;
    const float f = (d - L) / de;
    const float fp = (P.pbd_eps + L) / (de * de);
    const float b = d > 0.f ? fp / d : 0.f;
    return mv3(f, y, b, r, dot3(r, y));
}
// 2 J_spiky(r) G_spiky(r) = d/dr |G_spiky(r)|^2
__device__ __forceinline__ float3 grad_gsq(const DevParams& P, float3 r, float d)
{
    const float3 G = G_spiky(P, r, d);
    return sc3(2.f, jv_spiky(P, r, d, G));
}

// ------------------------------------------------------- a particle's neighbours by a warp
// Ordered sums over the entries j != skip of set v within d2 < cut of p.  Lane c < 27 scans cell c
// (h: its hash), four entries in flight; the counts' prefix over the lanes lists those accepted
// in shared memory in traversal order (cells z-y-x, index ascending), and 32 of them at a time
// are evaluated side by side: terms(j, out) writes M addends for each of NA sums, sum-major.
// Lane a < NA then adds the addends of sum a to its `acc`, neighbour by neighbour in order -- the
// additions that one thread walking the cells makes, so the sums round alike, while the costly
// terms run with full warps although a cell accepts few of its entries.  An absent addend is 0.
// (Views of a full sort: every range is current.)
constexpr uint32_t ADJ_TPB = 128, ADJ_LIST = 96, ADJ_TERMS = 24;
struct AdjBuf {
    uint32_t j[ADJ_LIST];
    float t[32 * (ADJ_TERMS + 1)];    // a lane's addends; an odd row keeps the lanes off each other's banks
};
template <int NA, int M, class F>
__device__ __forceinline__ void warp_neighbors(const SetView& v, float3 p, uint32_t h, uint32_t skip, float cut,
                                               AdjBuf& W, float& acc, F&& terms)
{
    static_assert(NA * M <= (int)ADJ_TERMS, "addends of a neighbour");
    constexpr int ROW = (NA * M) | 1;
    const uint32_t lane = threadIdx.x & 31u, full = 0xffffffffu;
    uint32_t s = 0, e = 0;
    if (lane < 27u) {
        s = __ldg(v.cs + h);
        e = __ldg(v.ce + h);
        if (s == SNOWB_EMPTY) s = e = 0u;
    }
    auto hit = [&](uint32_t j) {
        const float3 r = sub3(p, xyz(__ldg(v.p4 + j)));
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
    const uint32_t first = warp_incl_scan(n) - n, total = __shfl_sync(full, first + n, 31);
    for (uint32_t w0 = 0; w0 < total; w0 += ADJ_LIST) {
        __syncwarp();
        uint32_t at = first, m = mask;
        while (m) {
            const uint32_t j = s + (uint32_t)__ffs(m) - 1u;
            m &= m - 1u;
            if (at - w0 < ADJ_LIST) W.j[at - w0] = j;
            ++at;
        }
        for (uint32_t j = s + 32u; j < e; ++j)
            if (hit(j)) {
                if (at - w0 < ADJ_LIST) W.j[at - w0] = j;
                ++at;
            }
        __syncwarp();
        const uint32_t held = umin32(total - w0, ADJ_LIST);
        for (uint32_t b = 0; b < held; b += 32u) {
            if (b + lane < held) terms(W.j[b + lane], W.t + lane * ROW);
            __syncwarp();
            if (lane < (uint32_t)NA)
                for (uint32_t k = 0; k < umin32(held - b, 32u); ++k)
#pragma unroll
                    for (int q = 0; q < M; ++q) acc += W.t[k * ROW + lane * M + q];
            __syncwarp();
        }
    }
}
// The passes below are written once for both forms: WARP, a particle to a warp, lane a < NA holding
// sum a; else a particle to a thread, which holds all sums and walks the cells itself.  Either way
// a sum's addends are added neighbour by neighbour in traversal order.
template <bool WARP, int NA>
struct AdjSums {
    float v[WARP ? 1 : NA];
    __device__ __forceinline__ AdjSums()
    {
#pragma unroll
        for (int a = 0; a < (WARP ? 1 : NA); ++a) v[a] = 0.f;
    }
    __device__ __forceinline__ void start(int a, float x)
    {
        if (!WARP) v[WARP ? 0 : a] = x;
        else if ((threadIdx.x & 31u) == (uint32_t)a) v[0] = x;
    }
    // sum a, for every lane
    __device__ __forceinline__ float of(int a) const { return WARP ? __shfl_sync(0xffffffffu, v[0], a) : v[WARP ? 0 : a]; }
    __device__ __forceinline__ float3 of3(int a) const { return f3(of(a), of(a + 1), of(a + 2)); }
};
// where a particle looks for neighbours: its cell, and a lane's own one of the 27 around it
template <bool WARP>
struct AdjCell {
    GCell g;
    uint32_t h;
    __device__ __forceinline__ AdjCell(const DevParams& P, float3 p) : g(grid_pos(P, p)), h(WARP ? lane_cell(P, g) : 0u) {}
};
template <int M, bool WARP, int NA, class F>
__device__ __forceinline__ void adj_neighbors(const DevParams& P, const SetView& v, float3 p, const AdjCell<WARP>& c,
                                              uint32_t skip, float cut, AdjBuf& W, AdjSums<WARP, NA>& sums, F&& terms)
{
    if constexpr (WARP) {
        warp_neighbors<NA, M>(v, p, c.h, skip, cut, W, sums.v[0], terms);
    } else {
        FOR27 {
            uint32_t s, e;
            if (!v.range(P, c.g, ox, oy, oz, s, e)) continue;
            for (uint32_t j = s; j < e; ++j) {
                const float3 r = sub3(p, xyz(__ldg(v.p4 + j)));
                if (j == skip || !(dot3(r, r) < cut)) continue;
                float out[NA * M];
                terms(j, out);
#pragma unroll
                for (int a = 0; a < NA; ++a)
#pragma unroll
                    for (int q = 0; q < M; ++q) sums.v[a] += out[a * M + q];
            }
        }
    }
}
// particles t < n of such a pass; the thread that writes a particle's results
#define ADJ_LOOP(WARP, t, n)                                                                      \
    for (uint32_t t = (blockIdx.x * blockDim.x + threadIdx.x) >> ((WARP) ? 5 : 0); t < (n);        \
         t += (gridDim.x * blockDim.x) >> ((WARP) ? 5 : 0))
#define ADJ_LEAD(WARP) (!(WARP) || (threadIdx.x & 31u) == 0u)
// Up to so many particles (water + snow) the passes run one warp each, above it one thread each.
// One warp | one thread, us a launch, at 9.2k, 47.9k, 83.5k and 153.8k particles: fields 43 | 102,
// 91 | 138, 148 | 148, 244 | 156; positions 43 | 122, 134 | 181, 220 | 201, 390 | 283; friction
// 25 | 84, 90 | 104, 150 | 116, 274 | 199; XSPH 20 | 83, 60 | 127, 94 | 124, 165 | 139; heat 30 | 95,
// 118 | 130, 200 | 136, 363 | 192 (the lambda adjoint, fewer neighbours, stays with one warp).  A
// gradient of three substeps meets at 75k: 17.1 | 17.8 ms at 70.2k, 18.4 | 17.8 at 83.5k, and
// 26.2 | 22.2 at 153.8k.
constexpr uint32_t ADJ_WARP_MAX = 75000;
// addend q of the three sums from a on (M addends each)
template <int M>
__device__ __forceinline__ void put3(float* out, int a, int q, float3 x)
{
    out[a * M + q] = x.x;
    out[(a + 1) * M + q] = x.y;
    out[(a + 2) * M + q] = x.z;
}
// A warp takes 32 boundary particles (nbg apart: those with neighbours come in patches): lane by
// lane they are looked over (near(i): is anything around?), and those with something around are
// taken by the whole warp, one after another (take(i), every lane).
template <class N, class T>
__device__ __forceinline__ void boundary_patch(uint32_t t, uint32_t nb, N&& near, T&& take)
{
    const uint32_t nbg = (nb + 31u) / 32u, i = t + (threadIdx.x & 31u) * nbg;
    uint32_t m = __ballot_sync(0xffffffffu, i < nb && near(i));
    while (m) {
        const uint32_t k = (uint32_t)__ffs(m) - 1u;
        m &= m - 1u;
        take(t + k * nbg);
    }
}

// ---------------------------------------------------------------- fields at positions
// density, C, gradient-square sum and lambda of every particle of the three sets (the
// quantities of k_density<true>, fixed quirks), stored in original order.
__device__ __forceinline__ void field_store(const DevParams& P, const AdjField& F, uint32_t o, float rho, float S)
{
    const float C = (rho / P.rho0) - 1.f > 0.f ? (rho / P.rho0) - 1.f : 0.f;
    F.rho[o] = rho;
    F.C[o] = C;
    F.S[o] = S;
    F.lam[o] = -C / (S + P.eps);
}
// a particle's density (sum 0) and gradient-square (sum 1) terms from the entries of set v (vol:
// the boundary, whose lambda denominator scales with the volume over m_of(j))
template <bool WARP, class F>
__device__ __forceinline__ void field_terms(const DevParams& P, const SetView& v, float3 p, const AdjCell<WARP>& c,
                                            uint32_t skip, bool vol, AdjBuf& W, AdjSums<WARP, 2>& acc, F&& m_of)
{
    adj_neighbors<1>(P, v, p, c, skip, P.h2_lt, W, acc, [&](uint32_t j, float* out) {
        const float4 q = __ldg(v.p4 + j);
        const float3 r = sub3(p, xyz(q));
        const float d = sqrtf(dot3(r, r));
        out[0] = (vol ? P.rho0 * q.w : q.w) * W_poly6(P, d);
        const float sc = vol ? P.inv_rho0 * ((P.rho0 * q.w) / m_of(j)) : P.inv_rho0;
        const float3 G = G_spiky(P, r, d);
        out[1] = (sc * sc) * dot3(G, G);
    });
}
// the sums of a boundary particle without water or snow around it: the boundary does not move,
// so they are the same in every pass of a backward call (by sorted index)
__global__ void __launch_bounds__(ADJ_TPB) ka_boundary_base(DevParams P, uint32_t nb, SetView vb, Sets X, float* rho0,
                                                            float* S0)
{
    wait_prior();
    __shared__ AdjBuf bufs[ADJ_TPB / 32];
    AdjBuf& W = bufs[threadIdx.x >> 5];
    const uint32_t lane = threadIdx.x & 31u;
    vb.n = nb;
    WARP_LOOP(i, nb) {
        const float3 p = xyz(vb.p4[i]);
        AdjSums<true, 2> acc;
        acc.start(0, (P.rho0 * X.bnd.volume[vb.gi[i]]) * P.W0);
        field_terms(P, vb, p, AdjCell<true>(P, p), i, true, W, acc, [&](uint32_t j) { return X.bnd.mass[vb.gi[j]]; });
        if (lane == 0u) rho0[i] = acc.v[0];
        if (lane == 1u) S0[i] = acc.v[0];
    }
}
// first: the particles (water, snow, boundary in that order) before it are not taken; the one-thread
// form takes the water and snow, and the boundary comes from the other form
template <bool WARP>
__global__ void __launch_bounds__(ADJ_TPB) ka_fields(DevParams P, uint32_t nw, uint32_t ns, uint32_t nb, SetView vw,
                                                     SetView vs, SetView vb, Sets X, AdjField fw, AdjField fs,
                                                     AdjField fb, const float* __restrict__ rho0,
                                                     const float* __restrict__ S0, uint32_t first)
{
    wait_prior();
    __shared__ AdjBuf bufs[WARP ? ADJ_TPB / 32 : 1];
    AdjBuf& W = bufs[WARP ? threadIdx.x >> 5 : 0];
    vw.n = nw; vs.n = ns; vb.n = nb;
    ADJ_LOOP(WARP, t0, nw + ns + (WARP ? (nb + 31u) / 32u : 0u) - first) {
        const uint32_t t = t0 + first;
        if (t < nw + ns) {
            const bool w = t < nw;
            const uint32_t i = w ? t : t - nw;
            const SetView& own = w ? vw : vs;
            const uint32_t o = own.gi[i];
            const float3 p = xyz(own.p4[i]);
            const AdjCell<WARP> c(P, p);
            const float mi = (w ? X.sph.mass : X.dem.mass)[o];
            auto m_of = [&](uint32_t) { return mi; };
            AdjSums<WARP, 2> acc;
            acc.start(0, mi * P.W0);
            field_terms(P, vw, p, c, w ? i : SNOWB_UMAX, false, W, acc, m_of);
            field_terms(P, vs, p, c, w ? SNOWB_UMAX : i, false, W, acc, m_of);
            field_terms(P, vb, p, c, SNOWB_UMAX, true, W, acc, m_of);
            const float rho = acc.of(0), S = acc.of(1);
            if (ADJ_LEAD(WARP)) field_store(P, w ? fw : fs, o, rho, S);
        } else if constexpr (WARP) {
            boundary_patch(
                t - nw - ns, nb,
                [&](uint32_t i) {
                    const bool near = occupied27(P, grid_pos(P, xyz(vb.p4[i])), vw, vs) != 0u;
                    if (!near) field_store(P, fb, vb.gi[i], rho0[i], S0[i]);
                    return near;
                },
                [&](uint32_t i) {
                    const float3 p = xyz(vb.p4[i]);
                    const uint32_t o = vb.gi[i];
                    const AdjCell<true> c(P, p);
                    auto m_of = [&](uint32_t j) { return X.bnd.mass[vb.gi[j]]; };
                    AdjSums<true, 2> acc;
                    acc.start(0, (P.rho0 * X.bnd.volume[o]) * P.W0);
                    field_terms(P, vw, p, c, SNOWB_UMAX, false, W, acc, m_of);
                    field_terms(P, vs, p, c, SNOWB_UMAX, false, W, acc, m_of);
                    field_terms(P, vb, p, c, i, true, W, acc, m_of);
                    const float rho = acc.of(0), S = acc.of(1);
                    if (ADJ_LEAD(true)) field_store(P, fb, o, rho, S);
                });
        }
    }
}

// ------------------------------------------------- lambda adjoint from the PBF terms
// lambda-bar of every particle from u (sor times the adjoint of the corrected water
// positions), then C-, S- and rho-bar (rho-bar is added to, so other terms at the same
// positions can be accumulated first).
__device__ __forceinline__ void lambar_store(const DevParams& P, const AdjField& F, uint32_t o, float lb)
{
    const float den = F.S[o] + P.eps;
    const float Cb = -lb / den;
    F.lamb[o] = lb;
    F.Sb[o] = lb * F.C[o] / (den * den);
    if ((F.rho[o] / P.rho0) - 1.f > 0.f) F.rhob[o] += Cb * P.inv_rho0;
}
// snow (snow: the coupling's support) and boundary particles take part in the water's PBF sums
__device__ __forceinline__ float lambar_of_water(const DevParams& P, const SetView& vw, float3 p, bool snow,
                                                 const float* contrib, const snowb_float3* u, AdjBuf& W)
{
    float acc = 0.f;
    warp_neighbors<1, 1>(vw, p, lane_cell(P, grid_pos(P, p)), SNOWB_UMAX, snow ? P.r2_le : P.h2_lt, W, acc,
                         [&](uint32_t j, float* out) {
        const float3 r = sub3(p, xyz(__ldg(vw.p4 + j)));   // r = x_i - x_k, the water term uses -r
        const float d = sqrtf(dot3(r, r));
        const uint32_t ok = vw.gi[j];
        out[0] = -(contrib[ok] * dot3(ldv3(u, ok), snow ? G_poly6(P, r, d) : G_spiky(P, r, d)));
    });
    return acc;   // in lane 0
}
__global__ void __launch_bounds__(ADJ_TPB) ka_pbf_lambar(DevParams P, uint32_t nw, uint32_t ns, uint32_t nb, SetView vw,
                                                         SetView vs, SetView vb, Sets X, AdjField fw, AdjField fs,
                                                         AdjField fb, AdjSet aw)
{
    wait_prior();
    __shared__ AdjBuf bufs[ADJ_TPB / 32];
    AdjBuf& W = bufs[threadIdx.x >> 5];
    vw.n = nw; vs.n = ns; vb.n = nb;
    const uint32_t lane = threadIdx.x & 31u;
    WARP_LOOP(t, nw + ns + (nb + 31u) / 32u) {
        if (t < nw) {
            const uint32_t o = vw.gi[t];
            const float3 p = xyz(vw.p4[t]);
            const uint32_t h = lane_cell(P, grid_pos(P, p));
            const float ci = X.sph.contrib[o];
            const float3 ui = ldv3(aw.u, o);
            float acc = 0.f;
            warp_neighbors<1, 1>(vw, p, h, t, P.h2_lt, W, acc, [&](uint32_t j, float* out) {
                const float3 r = sub3(p, xyz(__ldg(vw.p4 + j)));
                const uint32_t oj = vw.gi[j];
                out[0] = (ci * X.sph.contrib[oj]) * dot3(sub3(ui, ldv3(aw.u, oj)), G_spiky(P, r, sqrtf(dot3(r, r))));
            });
            warp_neighbors<1, 1>(vs, p, h, SNOWB_UMAX, P.r2_le, W, acc, [&](uint32_t j, float* out) {
                const float3 r = sub3(p, xyz(__ldg(vs.p4 + j)));
                out[0] = ci * dot3(ui, G_poly6(P, r, sqrtf(dot3(r, r))));
            });
            warp_neighbors<1, 1>(vb, p, h, SNOWB_UMAX, P.h2_lt, W, acc, [&](uint32_t j, float* out) {
                const float3 r = sub3(p, xyz(__ldg(vb.p4 + j)));
                out[0] = ci * dot3(ui, G_spiky(P, r, sqrtf(dot3(r, r))));
            });
            if (lane == 0u) lambar_store(P, fw, o, acc * P.inv_rho0);
        } else if (t < nw + ns) {
            const uint32_t i = t - nw;
            const float acc = lambar_of_water(P, vw, xyz(vs.p4[i]), true, X.sph.contrib, aw.u, W);
            if (lane == 0u) lambar_store(P, fs, vs.gi[i], acc * P.inv_rho0);
        } else {
            boundary_patch(
                t - nw - ns, nb,
                [&](uint32_t i) {
                    const bool near = (occupied27(P, grid_pos(P, xyz(vb.p4[i])), vw, vw) & 1u) != 0u;
                    if (!near) lambar_store(P, fb, vb.gi[i], 0.f);
                    return near;
                },
                [&](uint32_t i) {
                    const float acc = lambar_of_water(P, vw, xyz(vb.p4[i]), false, X.sph.contrib, aw.u, W);
                    if (lane == 0u) lambar_store(P, fb, vb.gi[i], acc * P.inv_rho0);
                });
        }
    }
}

// ------------------------------------------ position adjoint of one iteration (gather)
// xb (water, snow) += every position derivative at the iteration's input positions: PBF
// direct terms (lambda held), lambda through S and rho, contact terms, and the density
// terms of rho-bar (which also carries the XSPH and heat contributions at these
// positions when they were accumulated before).  pbf != 0 adds the constraint terms;
// pbf == 0 runs the density part alone (heat, substep start).
template <bool WARP>
__global__ void __launch_bounds__(ADJ_TPB) ka_pos_rev(DevParams P, uint32_t nw, uint32_t ns, uint32_t nb, SetView vw,
                                                  SetView vs, SetView vb, Sets X, AdjField fw, AdjField fs,
                                                  AdjField fb, AdjSet aw, AdjSet as, float* __restrict__ kst, int pbf, int contact)
{
    wait_prior();
    __shared__ AdjBuf bufs[WARP ? ADJ_TPB / 32 : 1];
    AdjBuf& W = bufs[WARP ? threadIdx.x >> 5 : 0];
    vw.n = nw; vs.n = ns; vb.n = nb;
    ADJ_LOOP(WARP, t, nw + ns) {
        const int set = t < nw ? 0 : 1;
        const uint32_t i = set == 0 ? t : t - nw;
        const SetView& own = set == 0 ? vw : vs;
        const uint32_t o = own.gi[i];
        const float3 p = xyz(own.p4[i]);
        const AdjCell<WARP> c(P, p);
        const AdjField& Fi = set == 0 ? fw : fs;
        const AdjSet& Ai = set == 0 ? aw : as;
        const snowb_particle_data& Di = set == 0 ? X.sph : X.dem;
        const float mi = Di.mass[o], wi_inv = Di.massInv[o], ci = Di.contrib[o];
        const float rhob_i = Fi.rhob[o], Sb_i = Fi.Sb[o];
        const float lam_i = pbf ? Fi.lam[o] : 0.f;
        const float3 ui = pbf ? ldv3(Ai.u, o) : f3(0.f, 0.f, 0.f);
        // sums 0..2: position adjoint (up to four addends a neighbour); 3..5: k_stretch direction
        AdjSums<WARP, 6> acc;
        for (int k = 0; k < 3; ++k) {
            const SetView& v = k == 0 ? vw : (k == 1 ? vs : vb);
            const AdjField& Fj = k == 0 ? fw : (k == 1 ? fs : fb);
            const bool self = k == set;
            adj_neighbors<4>(P, v, p, c, self ? i : SNOWB_UMAX, P.h2_lt, W, acc, [&](uint32_t j, float* out) {
#pragma unroll
                for (int q = 0; q < 24; ++q) out[q] = 0.f;
                const float4 q = __ldg(v.p4 + j);
                const float3 r = sub3(p, xyz(q));
                const float d2 = dot3(r, r);
                const float d = sqrtf(d2);
                const uint32_t oj = v.gi[j];
                const float wj = k == 2 ? P.rho0 * q.w : q.w;
                // density: d rho_i/dx_i = w_j Gp(r); d rho_j/dx_i = w_i Gp(r)
                put3<4>(out, 0, 0, sc3(wj * rhob_i + mi * Fj.rhob[oj], G_poly6(P, r, d)));
                if (!pbf) return;
                // S through lambda: s_ij^2 Sbar_i + s_ji^2 Sbar_j
                {
                    float sij = P.inv_rho0, sji = P.inv_rho0;
                    if (k == 2) sij = P.inv_rho0 * ((P.rho0 * q.w) / mi);
                    const float a = (sij * sij) * Sb_i + (sji * sji) * Fj.Sb[oj];
                    put3<4>(out, 0, 1, sc3(a, grad_gsq(P, r, d)));
                }
                if (set == 0) {
                    // water: PBF own / coupling / boundary terms
                    if (k == 0) {
                        const float cj = X.sph.contrib[oj];
                        const float3 uj = ldv3(aw.u, oj);
                        const float a = (ci * cj) * P.inv_rho0 * (lam_i + Fj.lam[oj]);
                        put3<4>(out, 0, 2, sc3(a, jv_spiky(P, r, d, sub3(ui, uj))));
                    } else if (k == 1) {
                        if (d2 < P.r2_le) {
                            const float a = ci * P.inv_rho0 * (lam_i + Fj.lam[oj]);
                            put3<4>(out, 0, 2, sc3(a, jv_gpoly6(P, r, d, ui)));
                        }
                        if (contact && d2 < P.r2_lt) {
                            // snow particle j pushed by this water particle: -k_st c_j kappa_ji Jc u_j
                            const float wj_inv = X.dem.massInv[oj];
                            const float kap = (-wj_inv) * (1.f / (wj_inv + wi_inv));
                            const float a = -(P.k_stretch * X.dem.contrib[oj]) * kap;
                            put3<4>(out, 0, 3, sc3(a, jv_contact(P, r, d, ldv3(as.u, oj), P.two_r)));
                        }
                    } else {
                        const float a = ci * P.inv_rho0 * (lam_i + Fj.lam[oj]);
                        put3<4>(out, 0, 2, sc3(a, jv_spiky(P, r, d, ui)));
                    }
                } else {
                    // snow: coupling term of water neighbours, contact terms
                    if (k == 0) {
                        if (d2 < P.r2_le) {
                            const float ck = X.sph.contrib[oj];
                            const float a = -(ck * P.inv_rho0) * (Fj.lam[oj] + lam_i);
                            put3<4>(out, 0, 2, sc3(a, jv_gpoly6(P, r, d, ldv3(aw.u, oj))));
                        }
                        if (contact && d2 < P.r2_lt) {
                            const float wj_inv = X.sph.massInv[oj];
                            const float kap = (-wi_inv) * (1.f / (wi_inv + wj_inv));
                            const float a = (P.k_stretch * ci) * kap;
                            put3<4>(out, 0, 3, sc3(a, jv_contact(P, r, d, ui, P.two_r)));
                            put3<4>(out, 3, 0, sc3(ci * kap, phi_contact(P, r, d)));
                        }
                    } else if (k == 1) {
                        if (d2 < P.r2_lt) {
                            const float wj_inv = X.dem.massInv[oj];
                            const float kij = ci * ((-wi_inv) * (1.f / (wi_inv + wj_inv)));
                            const float kji = X.dem.contrib[oj] * ((-wj_inv) * (1.f / (wj_inv + wi_inv)));
                            const float3 y = sub3(sc3(kij, ui), sc3(kji, ldv3(as.u, oj)));
                            put3<4>(out, 0, 2, jv_contact(P, r, d, y, P.two_r));
                        }
                    } else {
                        if (d2 < P.r2_lt) {
                            const float wj_inv = X.bnd.massInv[oj];
                            const float kij = ci * ((-wi_inv) * (1.f / (wi_inv + wj_inv)));
                            put3<4>(out, 0, 2, jv_contact(P, r, d, sc3(kij, ui), P.two_r));
                        }
                    }
                }
            });
        }
        const float3 xb = acc.of3(0), kst_dir = acc.of3(3);
        if (ADJ_LEAD(WARP)) {
            st3(Ai.xb, o, add3(ldv3(Ai.xb, o), xb));
            if (pbf) kst[t] = set == 1 ? dot3(ui, kst_dir) : 0.f;
        }
    }
}
// Scalar parameter gradients from per-particle values a (and b, when not null): warp sums in
// float, one double atomic per warp.
__global__ void ka_param_sum(uint32_t n, const float* __restrict__ a, const float* __restrict__ b, double* ga, double* gb)
{
    wait_prior();
    float x = 0.f, y = 0.f;
    GRID_LOOP(t, n) {
        x += a[t];
        if (b) y += b[t];
    }
    for (int s = 16; s > 0; s >>= 1) {
        x += __shfl_down_sync(0xffffffffu, x, s);
        y += __shfl_down_sync(0xffffffffu, y, s);
    }
    if ((threadIdx.x & 31) == 0) {
        if (x != 0.f) atomicAdd(ga, (double)x);
        if (b && y != 0.f) atomicAdd(gb, (double)y);
    }
}

// --------------------------------------------------------------- interlink adjoint
// records snapshotted at the iteration's start; masks of the forward (d <= brk L, d <= h,
// |res| <= 1 per end) recomputed from the same positions.
__device__ __forceinline__ bool link_live(const DevParams& P, float3 r, float d, float L, float wi, float wj,
                                          float3& res)
{
    if (L == 0.f) return false;
    if (d > P.brk * L) return false;
    if (d > P.h) return false;
    const float ws = wi + wj, C = d - L;
    const float3 n3 = div3(r, d + P.pbd_eps);
    res = sc3(((P.k_ref * -wi) * (1.f / ws)) * C, n3);
    if (len3(res) > 1.f || nan3(res) || inf3(res)) return false;
    return true;
}
// Lbar (per slot) accumulates the adjoint of the link's rest length from both ends' terms,
// for the links formed in this substep (their length is the distance at formation).
__global__ void ka_interlink_rev(DevParams P, uint32_t ns, const snowb_float3* __restrict__ x,
                                 const uint32_t* __restrict__ rec, const float* __restrict__ len,
                                 const float* __restrict__ invm, AdjSet as, AdjParams G, float* Lbar)
{
    wait_prior();
    const uint32_t M = P.maxc;
    float kref_acc = 0.f;
    GRID_LOOP(i, ns) {
        const float3 xi = ldv3(x, i);
        const float3 ui = ldv3(as.u, i);
        const float wi = invm[i];
        float3 xb = f3(0.f, 0.f, 0.f);
        for (uint32_t s = M * i; s < M * (i + 1); ++s) {
            const uint32_t j = rec[s];
            if (j == SNOWB_UMAX || j == i || j >= ns) continue;
            const float L = len[s];
            const float3 r = sub3(xi, ldv3(x, j));
            const float d = len3(r);
            const float wj = invm[j];
            float3 res;
            float lb = 0.f;
            if (link_live(P, r, d, L, wi, wj, res)) {
                const float K = (P.k_ref * -wi) * (1.f / (wi + wj));
                xb = add3(xb, sc3(K, jv_contact(P, r, d, ui, L)));
                if (P.k_ref != 0.f) kref_acc += dot3(ui, res) / P.k_ref;
                lb -= K * dot3(ui, r) / (d + P.pbd_eps);          // d res / dL = -K r / (d + eps)
            }
            // the partner's term on this particle (its own record of the link, same length)
            const float3 rj = sc3(-1.f, r);
            const float3 uj = ldv3(as.u, j);
            float3 resj;
            if (link_live(P, rj, d, L, wj, wi, resj)) {
                const float Kj = (P.k_ref * -wj) * (1.f / (wj + wi));
                xb = sub3(xb, sc3(Kj, jv_contact(P, rj, d, uj, L)));
                lb -= Kj * dot3(uj, rj) / (d + P.pbd_eps);
            }
            Lbar[s] += lb;
        }
        st3(as.xb, i, add3(ldv3(as.xb, i), xb));
    }
    for (int s = 16; s > 0; s >>= 1) kref_acc += __shfl_down_sync(0xffffffffu, kref_acc, s);
    if ((threadIdx.x & 31) == 0 && kref_acc != 0.f) atomicAdd(G.g + 0, (double)kref_acc);
}

// links formed in this substep (slot empty at the substep's start, filled at the first
// iteration): their rest length is |x0_i - x0_j| at the formation positions x0.  Lbar
// carries each slot's rest-length adjoint from later substeps; it is consumed (zeroed)
// here, where the length came into being.
__global__ void ka_linkform_rev(DevParams P, uint32_t ns, const snowb_float3* __restrict__ x0,
                                const uint32_t* __restrict__ rec_pre, const uint32_t* __restrict__ rec0,
                                float* Lbar, snowb_float3* xb)
{
    wait_prior();
    const uint32_t M = P.maxc;
    GRID_LOOP(i, ns) {
        const float3 xi = ldv3(x0, i);
        float3 acc = f3(0.f, 0.f, 0.f);
        for (uint32_t s = M * i; s < M * (i + 1); ++s) {
            const uint32_t j = rec0[s];
            if (j == SNOWB_UMAX || rec_pre[s] != SNOWB_UMAX || j >= ns) continue;
            const float lb = Lbar[s];
            Lbar[s] = 0.f;
            const float3 r = sub3(xi, ldv3(x0, j));
            const float d = len3(r);
            if (d > 0.f && lb != 0.f) acc = add3(acc, sc3(lb / d, r));
        }
        st3(xb, i, add3(ldv3(xb, i), acc));
    }
}

// ---------------------------------------------------------------- friction adjoint
// vector-Jacobian product of friction_term: ub = adjoint of the result; returns the
// adjoints of dx and of r (the pair vector p_i - p_j).
__device__ __forceinline__ void friction_vjp(const DevParams& P, float3 dx, float w0, float w1, float d, float3 r,
                                             float3 ub, float3& dxb, float3& rb)
{
    const float ws = w0 + w1;
    const float de = d + P.pbd_eps;
    const float3 n = div3(r, de);
    const float pen = P.two_r - d;
    const float dn = dot3(dx, n);
    const float3 dxt = sub3(dx, sc3(dn, n));
    const float len = len3(dxt);
    float3 ab = sc3(-(w0 / ws), ub);   // adjoint of the (scaled) tangential displacement
    float3 tb = ab;                    // adjoint of dxt
    float pen_b = 0.f;
    if (len > P.mu_s * pen) {
        const float den = len + 0.000001f;
        const float c = (P.mu_k * pen) / den;
        if (c < 1.f) {
            const float adt = dot3(ab, dxt);
            tb = sc3(c, ab);
            if (len > 0.f) tb = add3(tb, sc3(-adt * (P.mu_k * pen) / (den * den) / len, dxt));
            pen_b = adt * P.mu_k / den;
        }
    }
    // dxt = dx - (dx.n) n
    const float tn = dot3(tb, n);
    dxb = sub3(tb, sc3(tn, n));
    const float3 nb = sub3(sc3(-tn, dx), sc3(dn, tb));
    // n = r / (d + eps): J_n = I/de - r r^T / (d de^2)
    const float rn = dot3(r, nb);
    rb = sub3(sc3(1.f / de, nb), sc3(d > 0.f ? rn / (d * de * de) : 0.f, r));
    // pen = 2r - d
    if (d > 0.f) rb = sub3(rb, sc3(pen_b / d, r));
}
// snow particles at the friction pass's positions (sorted view vs) and the start
// positions after integration x0p; u = sor * adjoint of the positions after friction.
template <bool WARP>
__global__ void __launch_bounds__(ADJ_TPB) ka_friction_rev(DevParams P, uint32_t ns, uint32_t nb, SetView vs, SetView vb,
                                                           Sets X, AdjSet as)
{
    wait_prior();
    __shared__ AdjBuf bufs[WARP ? ADJ_TPB / 32 : 1];
    AdjBuf& W = bufs[WARP ? threadIdx.x >> 5 : 0];
    vs.n = ns; vb.n = nb;
    ADJ_LOOP(WARP, i, ns) {
        const uint32_t o = vs.gi[i];
        const float3 p = xyz(vs.p4[i]);
        const AdjCell<WARP> c(P, p);
        const float3 op0 = ldv3(as.x0p, o);
        const float w0 = X.dem.massInv[o];
        const float3 ui = ldv3(as.u, o);
        AdjSums<WARP, 6> acc;   // sums 0..2: positions, 3..5: start positions; two addends a neighbour
        adj_neighbors<2>(P, vs, p, c, i, P.r2_le, W, acc, [&](uint32_t j, float* out) {
            const float3 pp1 = xyz(__ldg(vs.p4 + j));
            const float3 r = sub3(p, pp1);
            const float d = sqrtf(dot3(r, r));
            const uint32_t oj = vs.gi[j];
            const float3 op1 = ldv3(as.x0p, oj);
            const float w1 = X.dem.massInv[oj];
            const float3 dx = add3(sub3(p, op0), sub3(pp1, op1));
            float3 dxb, rb;
            friction_vjp(P, dx, w0, w1, d, r, ui, dxb, rb);        // term of i
            put3<2>(out, 0, 0, add3(dxb, rb));
            put3<2>(out, 3, 0, sc3(-1.f, dxb));
            friction_vjp(P, dx, w1, w0, d, sc3(-1.f, r), ldv3(as.u, oj), dxb, rb);   // term of j
            put3<2>(out, 0, 1, sub3(dxb, rb));
            put3<2>(out, 3, 1, sc3(-1.f, dxb));
        });
        adj_neighbors<1>(P, vb, p, c, SNOWB_UMAX, P.r2_le, W, acc, [&](uint32_t j, float* out) {
            const float3 r = sub3(p, xyz(__ldg(vb.p4 + j)));
            float3 dxb, rb;
            friction_vjp(P, sub3(p, op0), w0, X.bnd.massInv[vb.gi[j]], sqrtf(dot3(r, r)), r, ui, dxb, rb);
            put3<1>(out, 0, 0, add3(dxb, rb));
            put3<1>(out, 3, 0, sc3(-1.f, dxb));
        });
        const float3 pb = acc.of3(0), x0b = acc.of3(3);
        if (ADJ_LEAD(WARP)) {
            st3(as.xb, o, add3(ldv3(as.xb, o), pb));
            st3(as.x0b, o, add3(ldv3(as.x0b, o), x0b));
        }
    }
}

// -------------------------------------------------------------------- XSPH adjoint
// XSPH of set A (own) over A and B with velocities vA, vB, viscosity c; gb = adjoint of
// A's new velocities.  One launch handles both roles: warps [0, nA) take particles of A
// (own sum: velocity, position and density adjoints), warps [nA, nA + nB) particles of
// B (as neighbours of A).  Outputs are added to vbA/vbB (velocity adjoints), xbA/xbB and
// rhobA/rhobB.  A's own velocity adjoint keeps its identity term.
template <bool WARP>
__global__ void __launch_bounds__(ADJ_TPB) ka_xsph_rev(DevParams P, uint32_t nA, uint32_t nB, SetView vA, SetView vB,
                                                   const snowb_float3* __restrict__ velA,
                                                   const snowb_float3* __restrict__ velB,
                                                   const float* __restrict__ massA, const float* __restrict__ massB,
                                                   const float* __restrict__ rhoA, const float* __restrict__ rhoB,
                                                   float c, const snowb_float3* __restrict__ gb,
                                                   snowb_float3* vbA, snowb_float3* vbB, snowb_float3* xbA,
                                                   snowb_float3* xbB, float* rhobA, float* rhobB)
{
    wait_prior();
    __shared__ AdjBuf bufs[WARP ? ADJ_TPB / 32 : 1];
    AdjBuf& W = bufs[WARP ? threadIdx.x >> 5 : 0];
    vA.n = nA; vB.n = nB;
    ADJ_LOOP(WARP, t, nA + nB) {
        const bool inA = t < nA;
        const uint32_t i = inA ? t : t - nA;
        const SetView& own = inA ? vA : vB;
        const uint32_t o = own.gi[i];
        const float3 p = xyz(own.p4[i]);
        const AdjCell<WARP> cell(P, p);
        const float3 vi = ldv3(inA ? velA : velB, o);
        const float mi = (inA ? massA : massB)[o], rhoi = (inA ? rhoA : rhoB)[o];
        const float ai = mi / rhoi;
        // sums 0..2: positions (two addends a neighbour), 3..5: velocities, 6: density, 7: weights
        AdjSums<WARP, 8> acc;
        // i as a neighbour of A-particle j: c a_i (v_i - v_j) W, adjoint g_j
        auto as_neighbor = [&](float* out, int q, uint32_t oj, float3 vj, float3 r, float d, float Wd) {
            const float3 gj = ldv3(gb, oj);
            put3<2>(out, 3, 0, sc3(c * ai * Wd, gj));
            put3<2>(out, 0, q, sc3(c * ai * dot3(sub3(vi, vj), gj), G_poly6(P, r, d)));
            out[12] = -c * (mi / (rhoi * rhoi)) * Wd * dot3(sub3(vi, vj), gj);
        };
        float3 vb;
        if (inA) {
            const float3 gi = ldv3(gb, o);
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const SetView& v = k == 0 ? vA : vB;
                adj_neighbors<2>(P, v, p, cell, k == 0 ? i : SNOWB_UMAX, P.h2_lt, W, acc, [&](uint32_t j, float* out) {
                    for (int q = 0; q < 16; ++q) out[q] = 0.f;
                    const float3 r = sub3(p, xyz(__ldg(v.p4 + j)));
                    const float d = sqrtf(dot3(r, r));
                    const uint32_t oj = v.gi[j];
                    const float3 vj = ldv3(k == 0 ? velA : velB, oj);
                    const float aj = (k == 0 ? massA : massB)[oj] / (k == 0 ? rhoA : rhoB)[oj];
                    const float Wd = W_poly6(P, d);
                    out[14] = aj * Wd;
                    // own term: c a_j (v_j - v_i) W(r)
                    put3<2>(out, 0, 0, sc3(c * aj * dot3(sub3(vj, vi), gi), G_poly6(P, r, d)));
                    if (k == 0) as_neighbor(out, 1, oj, vj, r, d, Wd);
                });
            }
            vb = add3(acc.of3(3), sc3(1.f - c * acc.of(7), gi));
        } else {
            adj_neighbors<2>(P, vA, p, cell, SNOWB_UMAX, P.h2_lt, W, acc, [&](uint32_t j, float* out) {
                for (int q = 0; q < 16; ++q) out[q] = 0.f;
                const float3 r = sub3(p, xyz(__ldg(vA.p4 + j)));
                const float d = sqrtf(dot3(r, r));
                const uint32_t oj = vA.gi[j];
                as_neighbor(out, 0, oj, ldv3(velA, oj), r, d, W_poly6(P, d));
            });
            vb = acc.of3(3);
        }
        const float3 xb = acc.of3(0);
        const float rb = acc.of(6);
        if (ADJ_LEAD(WARP)) {
            snowb_float3 *const vo = inA ? vbA : vbB, *const xo = inA ? xbA : xbB;
            st3(vo, o, add3(ldv3(vo, o), vb));
            st3(xo, o, add3(ldv3(xo, o), xb));
            (inA ? rhobA : rhobB)[o] += rb;
        }
    }
}

// -------------------------------------------------------------------- heat adjoint
// T1_i = T_i + dt/(C_i rho_i) sum_j (m_j/rho_j) kh_ij (T_j - T_i) L(d_ij), neighbours in
// both sets (fixed quirks).  Tb = adjoint of T1 in, T0b = adjoint of T out; rho-bar and
// position adjoints added; conductivity gradients accumulated.
__device__ __forceinline__ float kh(float ki, float kj) { return ((4.f * ki) * kj) / (ki + kj); }
template <bool WARP>
__global__ void __launch_bounds__(ADJ_TPB) ka_heat_rev(DevParams P, uint32_t nw, uint32_t ns, SetView vw, SetView vs,
                                                   Sets X, const float* __restrict__ Tw, const float* __restrict__ Ts,
                                                   const float* __restrict__ Tbw, const float* __restrict__ Tbs,
                                                   float* T0bw, float* T0bs, AdjField fw, AdjField fs, AdjSet aw,
                                                   AdjSet as, float* __restrict__ gkw_t, float* __restrict__ gks_t,
                                                       float dt)
{
    wait_prior();
    __shared__ AdjBuf bufs[WARP ? ADJ_TPB / 32 : 1];
    AdjBuf& W = bufs[WARP ? threadIdx.x >> 5 : 0];
    vw.n = nw; vs.n = ns;
    ADJ_LOOP(WARP, t, nw + ns) {
        const int set = t < nw ? 0 : 1;
        const uint32_t i = set == 0 ? t : t - nw;
        const SetView& own = set == 0 ? vw : vs;
        const uint32_t o = own.gi[i];
        const float3 p = xyz(own.p4[i]);
        const AdjCell<WARP> c(P, p);
        const float Ti = (set == 0 ? Tw : Ts)[o];
        const float Tbi = (set == 0 ? Tbw : Tbs)[o];
        const float ki = set == 0 ? P.k_water : P.k_snow;
        const float Ci = set == 0 ? P.C_water : P.C_snow;
        const float mi = (set == 0 ? X.sph.mass : X.dem.mass)[o];
        const float rhoi = (set == 0 ? fw.rho : fs.rho)[o];
        const float bi = dt / (Ci * rhoi);
        // sums 0: T, 1: weights, 2: dT, 3: density, 4, 5: conductivities, 6..8: positions
        AdjSums<WARP, 9> acc;
        for (int k = 0; k < 2; ++k) {
            const SetView& v = k == 0 ? vw : vs;
            const float kj = k == 0 ? P.k_water : P.k_snow;
            const float Cj = k == 0 ? P.C_water : P.C_snow;
            const float kk = kh(ki, kj);
            // d kh / d k_water and d kh / d k_snow of this pair
            float dkw, dks;
            if (set == k) { dkw = set == 0 ? 2.f : 0.f; dks = set == 1 ? 2.f : 0.f; }
            else {
                const float s2 = (P.k_water + P.k_snow) * (P.k_water + P.k_snow);
                dkw = 4.f * P.k_snow * P.k_snow / s2;
                dks = 4.f * P.k_water * P.k_water / s2;
            }
            adj_neighbors<1>(P, v, p, c, k == set ? i : SNOWB_UMAX, P.h2_lt, W, acc, [&](uint32_t j, float* out) {
                const float3 r = sub3(p, xyz(__ldg(v.p4 + j)));
                const float d = sqrtf(dot3(r, r));
                const uint32_t oj = v.gi[j];
                const float Tj = (k == 0 ? Tw : Ts)[oj];
                const float Tbj = (k == 0 ? Tbw : Tbs)[oj];
                const float mj = (k == 0 ? X.sph.mass : X.dem.mass)[oj];
                const float rhoj = (k == 0 ? fw.rho : fs.rho)[oj];
                const float bj = dt / (Cj * rhoj);
                const float L = L_visc(P, d);
                const float aij = (mj / rhoj) * kk, aji = (mi / rhoi) * kk;
                // temperatures
                out[1] = aij * L;
                out[0] = Tbj * bj * aji * L;
                out[2] = aij * (Tj - Ti) * L;
                // this particle's density in the neighbour's term
                out[3] = Tbj * bj * (-(mi / (rhoi * rhoi)) * kk) * (Ti - Tj) * L;
                // positions through L(d): dL/dx_i = -visc_lap r/d
                const float a = Tbi * bi * aij * (Tj - Ti) + Tbj * bj * aji * (Ti - Tj);
                put3<1>(out, 6, 0, d > 0.f ? sc3(a * (-P.visc_lap) / d, r) : f3(0.f, 0.f, 0.f));
                // conductivities (own term only: every pair is counted once per end)
                const float q = Tbi * bi * (mj / rhoj) * (Tj - Ti) * L;
                out[4] = q * dkw;
                out[5] = q * dks;
            });
        }
        const float T0b = acc.of(0) + Tbi * (1.f - bi * acc.of(1));
        const float rb = acc.of(3) + -Tbi * (bi / rhoi) * acc.of(2);
        const float gkw = acc.of(4), gks = acc.of(5);
        const float3 xb = acc.of3(6);
        if (ADJ_LEAD(WARP)) {
            (set == 0 ? T0bw : T0bs)[o] = T0b;
            (set == 0 ? fw.rhob : fs.rhob)[o] += rb;
            const AdjSet& A = set == 0 ? aw : as;
            st3(A.xb, o, add3(ldv3(A.xb, o), xb));
            gkw_t[t] = gkw;
            gks_t[t] = gks;
        }
    }
}

// --------------------------------------------------- integrate / finalize adjoints
// finalize: v = (x_new - x0p)/dt, x = x_new.  xb (in: adjoint of the final positions,
// out: adjoint of x_new), vb in: adjoint of v; x0b -= vb/dt.
__global__ void ka_finalize_rev(uint32_t n, float dt, const snowb_float3* __restrict__ vb, snowb_float3* xb,
                                snowb_float3* x0b)
{
    wait_prior();
    GRID_LOOP(i, n) {
        const float3 v = div3(ldv3(vb, i), dt);
        st3(xb, i, add3(ldv3(xb, i), v));
        st3(x0b, i, sub3(ldv3(x0b, i), v));
    }
}
// integrate_one with cd_on, branches recomputed from (x0, v0).  In: xpb (adjoint of the
// predicted positions), x0b (adjoint of the positions array after integration).  Out:
// xout (adjoint of x0, added), vout (adjoint of v0, written).
__global__ void ka_integrate_rev(DevParams P, uint32_t n, float dt, int cd_on, const snowb_float3* __restrict__ x0,
                                 const snowb_float3* __restrict__ v0, const snowb_float3* __restrict__ xpb,
                                 const snowb_float3* __restrict__ x0b, snowb_float3* xout, snowb_float3* vout)
{
    wait_prior();
    GRID_LOOP(i, n) {
        const float3 xp_b = ldv3(xpb, i);
        float3 posb = add3(ldv3(x0b, i), xp_b);
        float3 tb = sc3(dt, xp_b);
        float3 tv = add3(ldv3(v0, i), f3(dt * P.gx, dt * P.gy, dt * P.gz));
        tv = f3(tv.x * P.damping, tv.y * P.damping, tv.z * P.damping);
        const float3 pos = ldv3(x0, i);
        bool floor_fix = false;
        if (cd_on) {
            // forward, remembering each reflection: component, sign source, applied
            float3 st[5];
            int hit[5] = {0, 0, 0, 0, 0};
            const float3 tp = add3(pos, sc3(dt, tv));
            st[0] = tv;
            if (tp.x + P.r >= P.wx1) { hit[0] = 1; tv.x = -fabsf(tv.x); tv = sc3(P.b_damping, tv); }
            st[1] = tv;
            if (tp.x - P.r <= P.wx0) { hit[1] = 1; tv.x = fabsf(tv.x); tv = sc3(P.b_damping, tv); }
            st[2] = tv;
            if (tp.z + P.r >= P.wz1) { hit[2] = 1; tv.z = -fabsf(tv.z); tv = sc3(P.b_damping, tv); }
            st[3] = tv;
            if (tp.z - P.r <= P.wz0) { hit[3] = 1; tv.z = fabsf(tv.z); tv = sc3(P.b_damping, tv); }
            st[4] = tv;
            if (pos.y - P.r <= P.floor_y) { hit[4] = 1; floor_fix = true; tv.y = fabsf(tv.y); tv = sc3(P.b_damping, tv); }
            const float sp = len3(tv);
            if (sp > P.max_speed) {
                const float3 th = div3(tv, sp);
                tb = sc3(P.max_speed / sp, sub3(tb, sc3(dot3(th, tb), th)));
            }
            // reverse through the reflections: tv' = bd * (component sign-flipped)
            if (hit[4]) { tb = sc3(P.b_damping, tb); tb.y *= (st[4].y > 0.f ? 1.f : (st[4].y < 0.f ? -1.f : 0.f)); }
            if (hit[3]) { tb = sc3(P.b_damping, tb); tb.z *= (st[3].z > 0.f ? 1.f : (st[3].z < 0.f ? -1.f : 0.f)); }
            if (hit[2]) { tb = sc3(P.b_damping, tb); tb.z *= (st[2].z > 0.f ? -1.f : (st[2].z < 0.f ? 1.f : 0.f)); }
            if (hit[1]) { tb = sc3(P.b_damping, tb); tb.x *= (st[1].x > 0.f ? 1.f : (st[1].x < 0.f ? -1.f : 0.f)); }
            if (hit[0]) { tb = sc3(P.b_damping, tb); tb.x *= (st[0].x > 0.f ? -1.f : (st[0].x < 0.f ? 1.f : 0.f)); }
        }
        if (floor_fix) posb.y = 0.f;
        st3(vout, i, sc3(P.damping, tb));
        st3(xout, i, add3(ldv3(xout, i), posb));
    }
}
// recording checks: the adjoint assumes contrib == 1 and no phase change
__global__ void ka_check_contrib(uint32_t nw, uint32_t ns, const float* __restrict__ cw, const float* __restrict__ cs,
                                 uint32_t* viol)
{
    wait_prior();
    GRID_LOOP(t, nw + ns) {
        const float c = t < nw ? cw[t] : cs[t - nw];
        if (c != 1.f) atomicOr(viol, 2u);
    }
}
__global__ void ka_check_phase(const DevState* __restrict__ S, uint32_t* viol)
{
    wait_prior();
    if (blockIdx.x == 0 && threadIdx.x == 0 && S->changed) atomicOr(viol, 1u);
}
// out = s * a
__global__ void ka_scale3(uint32_t n, snowb_float3* out, float s, const snowb_float3* __restrict__ a)
{
    wait_prior();
    GRID_LOOP(i, n) st3(out, i, sc3(s, ldv3(a, i)));
}
// out = a + s * b  (float3 arrays, first n entries)
__global__ void ka_axpy3(uint32_t n, snowb_float3* out, const snowb_float3* __restrict__ a, float s,
                         const snowb_float3* __restrict__ b)
{
    wait_prior();
    GRID_LOOP(i, n) st3(out, i, add3(ldv3(a, i), sc3(s, ldv3(b, i))));
}

}  // namespace snowb
