// ssfr.cuh -- screen-space fluid rendering as CUDA kernels into device images.  This is the
// reference's default view (Renderer::Render with m_b_render_fluid, Renderer.cpp:92-109):
// snow drawn as point sprites into a scene image, the water's sphere depth, smoothed by a
// separable bilateral filter, its additive thickness, and a full-screen composite that
// refracts the scene through the water surface.  Same arithmetic as the shaders, no graphics
// API; every image is width x height, row 0 at the bottom as in a GL framebuffer.
//
//  - sphere depth (point_depth_vs.glsl / point_depth_fs.glsl, Renderer::RenderSceneDepth
//    :404-483 for the snow, RenderFluidDepth :485-540 for the water): clip = PV (x, 1),
//    sprite side point_size / clip.w, eye = V (x, 1); per covered pixel n.xy = 2 pc - 1,
//    discarded when |n.xy|^2 > 1, n.z = sqrt(1 - |n.xy|^2); depth = (P (eye + r n, 1)).z / .w
//    written as the fragment depth (clamped to 0..1 by the depth buffer), depth test LESS
//    against the cleared 1: the buffer keeps the minimum.
//  - thickness (ssfr_thickness_*.glsl, RenderThickness :602-646): same sprites, additive
//    blending of n.z * 0.005 into a buffer cleared to the clear colour, no depth test (the
//    target has no depth attachment).  The sum is accumulated in 32.32 fixed point (each
//    term rounded to 2^-32), so it does not depend on the order of the atomics.
//  - bilateral smoothing (bilateral_fs.glsl, SmoothDepth :542-600): first along y, then
//    along x (blur_dir = (1, 1/H), then (1/W, 1)): taps x = -R, -R+1, .. <= R, nearest
//    texel with GL_REPEAT wrap (RenderTargetTexture.h:19-22), taps at depth >= 1 skipped,
//    weight exp(-(x s)^2) exp(-((d_tap - d) f)^2); depth <= 0 gives 0, depth >= 1 gives 1.
//  - composite (ssfr_fluid_fs.glsl, RenderFluid :648-690): eye position from depth through
//    the inverse projection, normal from the smaller of the one-sided differences, Phong
//    specular (exponent 1000), refraction of the scene with thickness-based transmission,
//    the shader's fresnel, diffuse and sky/ground reflection terms.
#pragma once
#include "render.cuh"

namespace snowb {

struct SsfrCam {
    float PV[16];           // projection * view (glm's product, column-major)
    float V[16], P[16];     // model_view (the model matrix is the identity) and projection
    float Pinv[16], Vinv[16];
    float point_size, radius;
    uint32_t W, H;
};
struct SsfrShade {
    float filter_radius, blur_scale, falloff;
    float light[4];         // light_color (rgb, w = surface weight)
    float clear[4];         // clear colour (thickness and scene background)
};

__device__ __forceinline__ float3 f3sub(float3 a, float3 b) { return f3(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ float3 f3norm(float3 v)
{
    const float l = sqrtf(dot3(v, v));
    return f3(v.x / l, v.y / l, v.z / l);
}
__device__ __forceinline__ float smoothstep_f(float e0, float e1, float x)
{
    float t = (x - e0) / (e1 - e0);
    t = fminf(fmaxf(t, 0.f), 1.f);
    return t * t * (3.f - 2.f * t);
}
__device__ __forceinline__ float mix_f(float a, float b, float t) { return a * (1.f - t) + b * t; }
__device__ __forceinline__ uint32_t wrap_texel(int i, uint32_t n)
{
    if ((uint32_t)i < n) return (uint32_t)i;
    const int m = i % (int)n;
    return (uint32_t)(m < 0 ? m + (int)n : m);
}

struct DepthVtx {
    bool live;
    float xw, yw, side;
    float3 eye;
};
__device__ __forceinline__ DepthVtx depth_vertex(const SsfrCam& c, float3 p)
{
    DepthVtx v;
    const float4 cl = mat_vec(c.PV, p.x, p.y, p.z, 1.f);
    const float4 e = mat_vec(c.V, p.x, p.y, p.z, 1.f);
    v.live = cl.w > 0.f && cl.x >= -cl.w && cl.x <= cl.w && cl.y >= -cl.w && cl.y <= cl.w && cl.z >= -cl.w &&
             cl.z <= cl.w;
    v.xw = (cl.x / cl.w + 1.f) * 0.5f * (float)c.W;
    v.yw = (cl.y / cl.w + 1.f) * 0.5f * (float)c.H;
    v.side = c.point_size / cl.w;
    v.eye = f3(e.x, e.y, e.z);
    return v;
}
// n.xy of a covered pixel and r2 = |n.xy|^2; false when the fragment is discarded
__device__ __forceinline__ bool sphere_coord(const DepthVtx& v, int px, int py, float& nx, float& ny, float& nz)
{
    point_coord(v.xw, v.yw, v.side, px, py, nx, ny);
    const float r2 = nx * nx + ny * ny;
    if (r2 > 1.f) return false;
    nz = sqrtf(1.f - r2);
    return true;
}

// One set's spheres, LANES lanes a particle (see splat_pixels).  DEPTH: into depth (float bits,
// cleared to 1.0), the minimum over fragments.  THICK: thickness, 32.32 fixed point per pixel.
// MASK: only where mask (another set's depth) lies inside 0..1.
template <uint32_t LANES, bool DEPTH, bool THICK, bool MASK>
__device__ __forceinline__ void splat_spheres(const SsfrCam& c, const snowb_float3* __restrict__ pos, uint32_t n,
                                              uint32_t* depth, unsigned long long* thick,
                                              const float* __restrict__ mask, uint32_t block, uint32_t blocks)
{
    SPLAT_LOOP(i, n, block, blocks) {
        const DepthVtx v = depth_vertex(c, ldv3(pos, i));
        if (!v.live) continue;
        int x0, x1, y0, y1;
        sprite_span(v.xw, v.side, c.W, x0, x1);
        sprite_span(v.yw, v.side, c.H, y0, y1);
        splat_pixels<LANES>(x0, x1, y0, y1, [&](int px, int py) {
            const size_t k = (size_t)py * c.W + px;
            if (MASK) {
                const float m = mask[k];
                if (m <= 0.f || m >= 1.f) return;
            }
            float nx, ny, nz;
            if (!sphere_coord(v, px, py, nx, ny, nz)) return;
            if (THICK) {
                const float t = nz * 0.005f;
                atomicAdd(thick + k, __float2ull_rn(t * 4294967296.f));
            }
            if (DEPTH) {
                const float ex = v.eye.x + nx * c.radius, ey = v.eye.y + ny * c.radius, ez = v.eye.z + nz * c.radius;
                const float4 cl = mat_vec(c.P, ex, ey, ez, 1.f);
                float d = cl.z / cl.w;
                if (!(d < 1.f)) return;               // LESS against the cleared 1 (NaN fails too)
                d = d > 0.f ? d : 0.f;                // clamp to 0..1 (and -0 to +0)
                const uint32_t db = __float_as_uint(d);
                if (db < depth[k]) atomicMin(depth + k, db);
            }
        });
    }
}
template <uint32_t LANES>
__global__ void __launch_bounds__(128) ks_sphere_depth(SsfrCam c, const snowb_float3* __restrict__ pos, uint32_t n,
                                                       uint32_t* depth)
{
    wait_prior();
    splat_spheres<LANES, true, false, false>(c, pos, n, depth, nullptr, nullptr, blockIdx.x, gridDim.x);
}
template <uint32_t LANES>
__global__ void __launch_bounds__(128) ks_thickness(SsfrCam c, const snowb_float3* __restrict__ pos, uint32_t n,
                                                    unsigned long long* thick)
{
    wait_prior();
    splat_spheres<LANES, false, true, false>(c, pos, n, nullptr, thick, nullptr, blockIdx.x, gridDim.x);
}
__device__ __forceinline__ float thickness_value(unsigned long long q, float clear_r)
{
    return clear_r + __ull2float_rn(q) * 2.3283064365386963e-10f;   // 2^-32
}

// One bilateral pass: horizontal = 0 filters along y, 1 along x; block of blocks, every thread
// of each.  The spatial weights are the same for every pixel: a block that has a pixel to
// filter forms them once (half of the pass's exponentials), the others only copy.
constexpr uint32_t BILATERAL_TAPS = 513;   // filter_radius <= 256
struct BilateralTaps {
    float x[BILATERAL_TAPS], w[BILATERAL_TAPS];
};
__device__ __forceinline__ void bilateral(const SsfrCam& c, const SsfrShade& s, const float* __restrict__ in,
                                          float* __restrict__ out, int horizontal, BilateralTaps& B, uint32_t block,
                                          uint32_t blocks)
{
    const uint32_t np = c.W * c.H;
    uint32_t taps = 0u;   // 0: not formed yet
    for (uint32_t base = block * blockDim.x; base < np; base += blocks * blockDim.x) {
        const uint32_t k = base + threadIdx.x;
        const float depth = k < np ? in[k] : 1.f;
        const bool filter = !(depth <= 0.f) && !(depth >= 1.f);
        if (__syncthreads_or(filter) && taps == 0u) {
            uint32_t n = 0u;
            for (float x = -s.filter_radius; x <= s.filter_radius; x += 1.f, ++n)
                if (n % blockDim.x == threadIdx.x) {
                    const float r = x * s.blur_scale;
                    B.x[n] = x;
                    B.w[n] = expf(-r * r);
                }
            taps = n;
            __syncthreads();
        }
        if (k >= np) continue;
        if (!filter) { out[k] = depth <= 0.f ? 0.f : 1.f; continue; }
        const int px = (int)(k % c.W), py = (int)(k / c.W);
        float sum = 0.f, wsum = 0.f;
        for (uint32_t n = 0; n < taps; ++n) {
            size_t t;
            if (horizontal) t = (size_t)py * c.W + wrap_texel((int)floorf(((float)px + 0.5f) + B.x[n]), c.W);
            else t = (size_t)wrap_texel((int)floorf(((float)py + 0.5f) + B.x[n]), c.H) * c.W + px;
            const float sd = in[t];
            if (sd >= 1.f) continue;
            const float w = B.w[n];
            const float r2 = (sd - depth) * s.falloff;
            const float g = expf(-r2 * r2);
            sum += sd * w * g;
            wsum += w * g;
        }
        if (wsum > 0.f) sum /= wsum;
        out[k] = sum < 1.f ? fmaxf(sum, 0.f) : 1.f;
    }
}
__global__ void __launch_bounds__(256) ks_bilateral(SsfrCam c, SsfrShade s, const float* __restrict__ in,
                                                    float* __restrict__ out, int horizontal)
{
    wait_prior();
    __shared__ BilateralTaps B;
    bilateral(c, s, in, out, horizontal, B, blockIdx.x, gridDim.x);
}

__device__ __forceinline__ float3 uv_to_eye(const SsfrCam& c, float u, float v, float z)
{
    const float4 e = mat_vec(c.Pinv, u * 2.f - 1.f, v * 2.f - 1.f, z, 1.f);
    return f3(e.x / e.w, e.y / e.w, e.z / e.w);
}

// Full-screen composite into rgba.
__global__ void ks_compose(SsfrCam c, SsfrShade s, const float* __restrict__ D, const unsigned long long* __restrict__ TH,
                           const float* __restrict__ scene, const float* __restrict__ SD, float* __restrict__ out,
                           int scene4, int out4)
{
    wait_prior();
    auto scene_at = [&](size_t t) {
        if (scene4) return __ldg(reinterpret_cast<const float4*>(scene) + t);
        return make_float4(scene[4 * t], scene[4 * t + 1], scene[4 * t + 2], scene[4 * t + 3]);
    };
    const float iw = 1.f / (float)c.W, ih = 1.f / (float)c.H;
    GRID_LOOP(k, c.W * c.H) {
        const float depth = D[k];
        float4 o;
        if (depth == 0.f) {
            o = make_float4(0.f, 0.f, 0.f, 0.f);
        } else if (depth == 1.f || depth >= SD[k]) {
            o = scene_at(k);
        } else {
            const int px = (int)(k % c.W), py = (int)(k / c.W);
            const float thick = fmaxf(thickness_value(TH[k], s.clear[0]), 0.3f);
            const float u = ((float)px + 0.5f) / (float)c.W, v = ((float)py + 0.5f) / (float)c.H;
            const float3 eye = uv_to_eye(c, u, v, depth);
            const size_t row = (size_t)py * c.W;
            const float3 zl = f3sub(eye, uv_to_eye(c, u - iw, v, D[row + wrap_texel(px - 1, c.W)]));
            const float3 zr = f3sub(uv_to_eye(c, u + iw, v, D[row + wrap_texel(px + 1, c.W)]), eye);
            const float3 zt = f3sub(uv_to_eye(c, u, v + ih, D[(size_t)wrap_texel(py + 1, c.H) * c.W + px]), eye);
            const float3 zb = f3sub(eye, uv_to_eye(c, u, v - ih, D[(size_t)wrap_texel(py - 1, c.H) * c.W + px]));
            const float3 dx = fabsf(zr.z) < fabsf(zl.z) ? zr : zl;
            const float3 dy = fabsf(zb.z) < fabsf(zt.z) ? zb : zt;
            const float3 nrm = f3norm(f3(dx.y * dy.z - dy.y * dx.z, dx.z * dy.x - dy.z * dx.x, dx.x * dy.y - dy.x * dx.y));
            const float4 wp = mat_vec(c.Vinv, eye.x, eye.y, eye.z, 1.f);
            const float4 l4 = mat_vec(c.V, 0.f, 1.f, 0.f, 0.f);
            const float3 l = f3(l4.x, l4.y, l4.z);
            const float3 ne = f3norm(eye);
            const float3 vd = f3(-ne.x, -ne.y, -ne.z);
            const float3 hv = f3norm(f3(vd.x + l.x, vd.y + l.y, vd.z + l.z));
            const float spec = powf(fmaxf(0.f, dot3(nrm, hv)), 1000.f);
            const float rs = (1.33f * 0.025f) * smoothstep_f(0.1f, 0.4f, wp.y);
            const float ru = u + nrm.x * rs * 0.75f, rv = v + nrm.y * rs * 1.f;
            const size_t rt = (size_t)wrap_texel((int)floorf(rv * (float)c.H), c.H) * c.W +
                              wrap_texel((int)floorf(ru * (float)c.W), c.W);
            const float tr0 = expf(-(0.9804f - s.light[0]) * thick);
            const float tr1 = expf(-(1.0f - s.light[1]) * thick);
            const float tr2 = expf(-(0.7255f - s.light[2]) * thick);
            const float4 sc = scene_at(rt);
            const float3 refr = f3(sc.x * tr0, sc.y * tr1, sc.z * tr2);
            const float3 lv = f3norm(f3(wp.x - 0.f, wp.y - 1000.f, wp.z - 0.f));
            const float ddl = (lv.x * -0.f + lv.y * -1.f) + lv.z * -0.f;
            const float att = fmaxf(smoothstep_f(0.95f, 1.0f, fabsf(ddl)), 0.05f);
            const float ln = dot3(l, nrm) * att;
            const float fres = 0.1f + 0.9f * powf(fminf(0.f, 1.f - dot3(nrm, vd)), 5.f);
            const float mx = mix_f(1.f, 1.f, ln * 0.5f + 0.5f);
            const float3 dif = f3(s.light[0] * mx * (1.f - s.light[3]), s.light[1] * mx * (1.f - s.light[3]),
                                  s.light[2] * mx * (1.f - s.light[3]));
            const float sky0 = 0.8078f * 1.2f, sky1 = 0.4784f * 1.2f, sky2 = 0.2078f * 1.2f;
            const float nv = dot3(nrm, vd);
            const float3 re = f3(vd.x - 2.f * nv * nrm.x, vd.y - 2.f * nv * nrm.y, vd.z - 2.f * nv * nrm.z);
            const float4 rw = mat_vec(c.Vinv, re.x, re.y, re.z, 0.f);
            const float ss = smoothstep_f(0.15f, 0.25f, rw.y);
            const float3 refl = f3(1.f + mix_f(1.f, sky0, ss), 1.f + mix_f(1.f, sky1, ss), 1.f + mix_f(1.f, sky2, ss));
            o.x = dif.x + (mix_f(refr.x, refl.x, fres) + spec) * s.light[3];
            o.y = dif.y + (mix_f(refr.y, refl.y, fres) + spec) * s.light[3];
            o.z = dif.z + (mix_f(refr.z, refl.z, fres) + spec) * s.light[3];
            o.w = 1.f;
        }
        put_pixel(out, k, o, out4);
    }
}
__global__ void ks_fill(uint32_t npix, uint32_t* __restrict__ depth_bits, uint32_t value,
                        unsigned long long* __restrict__ thick)
{
    wait_prior();
    GRID_LOOP(k, npix) {
        if (depth_bits) depth_bits[k] = value;
        if (thick) thick[k] = 0ull;
    }
}

// ------------------------------------------------------------------ the whole view
// What snowb_render_fluid runs between the clear and the second filter pass and the composite
// (the stages above, for callers of the single stages, give the same image in 11 launches).
// Each launch takes the work that does not wait on one another, blocks [0, split) one part:
//  1. clear of the sprite keys, both depths and the thickness;
//  2. the snow's sprites | the water's spheres, depth and thickness from one fragment;
//  3. shading of every pixel of the scene (no separate clear of the image) and the first
//     filter pass | the snow's sphere depth, only where the water has a depth inside 0..1:
//     the composite compares it nowhere else (a filtered depth is 0 or 1 wherever the
//     unfiltered one is).
// The README-scale view at 1600 x 900 (148k snow, 6k water): 172 -> 88 us for the call, 75 since
// launches overlap the end of the one before (launch_prior).
__global__ void ks_view_clear(uint32_t npix, unsigned long long* __restrict__ zbuf,
                              unsigned long long* __restrict__ thick, uint32_t* __restrict__ scene_depth,
                              uint32_t* __restrict__ fluid_depth)
{
    wait_prior();
    GRID_LOOP(k, npix) {
        zbuf[k] = ~0ull;
        thick[k] = 0ull;
        scene_depth[k] = fluid_depth[k] = 0x3f800000u;
    }
}
template <uint32_t LANES>
__global__ void __launch_bounds__(128) ks_view_splat(RenderCam rc, RenderColour col, SsfrCam c,
                                                     const snowb_float3* __restrict__ snow, uint32_t n_snow,
                                                     const snowb_float3* __restrict__ water, uint32_t n_water,
                                                     unsigned long long* zbuf, uint32_t* fluid_depth,
                                                     unsigned long long* thick, uint32_t split)
{
    wait_prior();
    if (blockIdx.x < split) splat_points<LANES, true>(rc, col, snow, n_snow, 0u, zbuf, blockIdx.x, split);
    else
        splat_spheres<LANES, true, true, false>(c, water, n_water, fluid_depth, thick, nullptr, blockIdx.x - split,
                                         gridDim.x - split);
}
template <uint32_t LANES>
__global__ void __launch_bounds__(256) ks_view_filter(RenderCam rc, RenderColour col, SsfrCam c, SsfrShade s,
                                                      const snowb_float3* __restrict__ snow,
                                                      const float* __restrict__ T, uint32_t n_snow,
                                                      const unsigned long long* __restrict__ zbuf,
                                                      float* __restrict__ scene, const float* __restrict__ fluid_depth,
                                                      float* __restrict__ tmp, uint32_t* scene_depth, uint32_t split)
{
    wait_prior();
    __shared__ BilateralTaps B;
    if (blockIdx.x >= split) {
        splat_spheres<LANES, true, false, true>(c, snow, n_snow, scene_depth, nullptr, fluid_depth, blockIdx.x - split,
                                         gridDim.x - split);
        return;
    }
    const uint32_t np = c.W * c.H;
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < np; k += split * blockDim.x) {
        float4 o;
        if (!shade_pixel(rc, col, snow, T, 0u, zbuf[k], k, o))
            o = make_float4(s.clear[0], s.clear[1], s.clear[2], s.clear[3]);
        put_pixel(scene, k, o, 1);   // the workspace is 16-byte aligned
    }
    bilateral(c, s, fluid_depth, tmp, 0, B, blockIdx.x, split);
}

}  // namespace snowb
