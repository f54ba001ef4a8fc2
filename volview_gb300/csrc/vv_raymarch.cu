// vv_raymarch.cu — the real-time ray marcher `record` runs when path tracing is
// off (renderer.rs:1707-1790): the ambient-occlusion volume (shaders/ao.comp),
// the shadow volume swept slice by slice away from the key light
// (shaders/shadow.comp, renderer.rs:1907-1950), and emission-absorption ray
// marching with single scattering (shaders/dvr.comp) into the HDR image.
//
// The lighting volumes are pixel-linear (x fastest) half-precision images at
// half (shadow, RGBA16F) and a quarter (occlusion, R16F) of the CT's resolution,
// sampled with linear filtering and a white border like the reference's border
// sampler. The scene's volumes, labels, tables and the sample model are the
// path tracer's (vv_pt_device.cuh).
#include <cuda_runtime.h>

#include <cstdlib>

#include "vv_pt_device.cuh"

namespace vv {
namespace VV_FMT_NS {  // this density format's kernels and launchers
namespace {

__device__ __forceinline__ float h2f(uint16_t h) { return __half2float(__ushort_as_half(h)); }
__device__ __forceinline__ uint16_t f2h(float f) { return __half_as_ushort(__float2half_rn(f)); }
__device__ __forceinline__ float comp3(f3 v, int i) { return i == 0 ? v.x : (i == 1 ? v.y : v.z); }
__device__ __forceinline__ void set3(f3& v, int i, float s) {
    if (i == 0) v.x = s;
    else if (i == 1) v.y = s;
    else v.z = s;
}

// common.glsl:68-74
__device__ __forceinline__ f3 index_to_tex(const PtArgs& A, f3 idx) { return (idx + 0.5f) / U3(A.u.dims); }
__device__ __forceinline__ f3 tex_to_index(const PtArgs& A, f3 tex) { return tex * U3(A.u.dims) - 0.5f; }

// common.glsl:385-391: a shadow-ray sample (ghosts and clipped parts cast no
// shadow; a clipped point's other fields are not read).
// In the modes that draw labels alone, a brick of majorant 0 holds no label mask,
// and neither do two voxels around it: the extinction is 0 without a look at the
// volume. Where the transfer function draws, a majorant of 0 does not say so: a
// density's bucket maximum starts one LUT entry above the lower of the two entries
// that the density is interpolated between.
__device__ Sample sample_point(const PtArgs& A, f3 idx) {
    int plane;
    const bool skips = A.u.path[3] != 0u && A.u.labels[0] >= 2.0f;
    if ((skips && __ldg(A.majorant + brick_index(A, idx)) <= 0.0f) || clip_depth(A, idx, plane) > 0.0f) {
        Sample s;
        s.albedo = mk(0.0f);
        s.extinction = 0.0f;
        return s;
    }
    return sample_point_unclipped(A, idx);
}

// common.glsl:160-162
__device__ __forceinline__ float density_view(const PtArgs& A, f3 idx) {
    return A.u.env[1] > 0.5f ? density_cubic(A, idx) : density_tri(A, idx);
}

// common.glsl:195-199: the cumulative integrals, interpolated by hand.
__device__ __forceinline__ float4 preint_at(const PtArgs& A, float density) {
    float x = gclamp(density, 0.0f, 1.0f) * 4095.0f;
    int i = min((int)x, 4094);
    float4 a = __ldg(A.preint + i), b = __ldg(A.preint + i + 1);
    float f = x - (float)i;
    return make_float4(mixf(a.x, b.x, f), mixf(a.y, b.y, f), mixf(a.z, b.z, f), mixf(a.w, b.w, f));
}

// common.glsl:206-214: the pre-integrated sample of a segment from `front` to `back`.
__device__ __noinline__ Sample tf_segment(const PtArgs& A, float front, float back) {
    if (fabsf(back - front) < 1e-4f) return tf_point(A, 0.5f * (front + back));
    float4 pb = preint_at(A, back), pf = preint_at(A, front);
    float d = back - front;
    float4 mean = make_float4((pb.x - pf.x) / d, (pb.y - pf.y) / d, (pb.z - pf.z) / d, (pb.w - pf.w) / d);
    f3 albedo;
    if (mean.w > 1e-6f) {
        albedo = mk(mean.x / mean.w, mean.y / mean.w, mean.z / mean.w);
    } else {
        float4 t = transfer(A, back);
        albedo = mk(t.x, t.y, t.z);
    }
    Sample s = tf_point(A, back);
    s.albedo = albedo;
    s.extinction = gmax(mean.w, 0.0f);
    return s;
}

// common.glsl:218-230
__device__ __noinline__ float preint_half_depth(const PtArgs& A, float front, float back) {
    float target = 0.5f * (preint_at(A, front).w + preint_at(A, back).w);
    float lo = 0.0f, hi = 1.0f;
    for (int i = 0; i < 6; i++) {
        float mid = 0.5f * (lo + hi);
        bool before = (preint_at(A, mixf(front, back, mid)).w < target) == (back > front);
        lo = before ? mid : lo;
        hi = before ? hi : mid;
    }
    return 0.5f * (lo + hi);
}

// dvr.comp:14-21: measured tissue as dense as the path tracer draws it.
__device__ __forceinline__ void as_dense_as_traced(const PtArgs& A, Sample& s) {
    if (measured(A, s)) s.extinction = dot(tissue_sigma(A, s), mk(1.0f / 3.0f));
}
__device__ __noinline__ Sample labelled(const PtArgs& A, Sample s, f3 idx) {
    s = apply_labels(A, s, idx);
    as_dense_as_traced(A, s);
    return s;
}
// The labelled sample at `idx` in the modes that draw labels alone: the masks
// decide before the density and the transfer function are looked at, as in
// sample_labels. With GRAD and smooth sampling, the density's gradient comes
// with a density that a ramp needs: a sample shaded where it was taken needs no
// second read.
template <bool GRAD>
__device__ __noinline__ Sample labelled_at(const PtArgs& A, f3 idx, uint32_t mode, f3& grad, bool& has_grad) {
    Sample s;
    has_grad = false;
    uint32_t label;
    bool ghost;
    if (!drawn_label(A, idx, mode, label, ghost)) {
        s.extinction = 0.0f;
        return s;
    }
    float d = 0.0f;
    if (label_ramps(A, label, mode, ghost)) {
        if (A.u.env[1] > 0.5f) {
            if (GRAD) {
                d = density_cubic_with_gradient(A, idx, grad);
                has_grad = true;
            } else {
                d = density_cubic(A, idx);
            }
        } else {
            d = density_tri(A, idx);
        }
    }
    s = labelled_sample(A, label, mode, ghost, d);
    as_dense_as_traced(A, s);
    return s;
}

// shading.glsl:61-63: interleaved gradient noise.
__device__ __forceinline__ float ign(float px, float py) {
    float a = px * 0.06711056f + py * 0.00583715f;
    float b = 52.9829189f * (a - floorf(a));
    return b - floorf(b);
}

// The shadow volume while slice `slice` of `axis` is written, sampled as the border
// sampler does: linear between texel centres, texels outside the volume white
// (1, 1, 1, 1). A lookup at the slice before lands within rounding of that slice's
// texels, so it may also weigh the slice being written, by up to 1e-5: those texels
// count as 0, as they are before the launch, and not as whatever other threads
// have written by then.
// CHAINED: the launch that writes the texels read here may not have ended when the
// reading one started, so the read-only path, which is for data that does not
// change while a kernel lives, is not for them; the loads are ordinary ones, after
// the wait for that launch.
struct LightVol {
    const ushort4* data;  // RGBA16F, x fastest
    int w, h, d, axis, slice;
};
template <bool CHAINED> __device__ __forceinline__ float4 lv_texel(const LightVol& v, int x, int y, int z) {
    const bool out = x < 0 || y < 0 || z < 0 || x >= v.w || y >= v.h || z >= v.d;
    const bool own = (v.axis == 0 ? x : v.axis == 1 ? y : z) == v.slice;
    const uint16_t none = out ? 0x3c00 : 0;  // 1 or 0
    ushort4 t = make_ushort4(none, none, none, none);
    if (!out && !own) {
        const ushort4* at = v.data + ((long)z * v.h + y) * v.w + x;
        t = CHAINED ? *at : __ldg(at);
    }
    return make_float4(h2f(t.x), h2f(t.y), h2f(t.z), h2f(t.w));
}
template <bool CHAINED> __device__ __forceinline__ float4 lv_linear(const LightVol& v, f3 tc) {
    float x = tc.x * (float)v.w - 0.5f, y = tc.y * (float)v.h - 0.5f, z = tc.z * (float)v.d - 0.5f;
    int i0 = (int)floorf(x), j0 = (int)floorf(y), k0 = (int)floorf(z);
    float a = x - (float)i0, b = y - (float)j0, c = z - (float)k0;
    float4 t[8];  // all loads before the sums: a slice is one chain of latencies
#pragma unroll
    for (int k = 0; k < 8; k++) t[k] = lv_texel<CHAINED>(v, i0 + (k & 1), j0 + ((k >> 1) & 1), k0 + (k >> 2));
    float4 r = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
    for (int k = 0; k < 8; k++) {
        float w = (k & 1 ? a : 1.0f - a) * (k & 2 ? b : 1.0f - b) * (k & 4 ? c : 1.0f - c);
        r.x += t[k].x * w;
        r.y += t[k].y * w;
        r.z += t[k].z * w;
        r.w += t[k].w * w;
    }
    return r;
}
__device__ __forceinline__ float4 f4add(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }
__device__ __forceinline__ float4 f4mul(float s, float4 a) { return make_float4(s * a.x, s * a.y, s * a.z, s * a.w); }

// A linear fetch of a lighting texture at texel-space position p (texel i's
// centre at i; the border texel sits at -1 and w).
__device__ __forceinline__ float4 lt_fetch(const LightTex& v, float x, float y, float z) {
    if (v.rgba) return tex3D<float4>(v.tex, x + 1.5f, y + 1.5f, z + 1.5f);
    return make_float4(tex3D<float>(v.tex, x + 1.5f, y + 1.5f, z + 1.5f), 0.0f, 0.0f, 1.0f);
}
__device__ __forceinline__ float4 lt_linear(const LightTex& v, f3 tc) {
    return lt_fetch(v, tc.x * (float)v.w - 0.5f, tc.y * (float)v.h - 0.5f, tc.z * (float)v.d - 0.5f);
}
// common.glsl:141-152: B-spline filtering from 8 linear fetches (folded taps of
// common.glsl:89-108).
__device__ __noinline__ float4 lt_cubic(const LightTex& v, f3 tc) {
    f3 size = mk((float)v.w, (float)v.h, (float)v.d);
    f3 idx = tc * size - 0.5f;
    f3 i = mk(floorf(idx.x), floorf(idx.y), floorf(idx.z));
    f3 f = idx - i, f2 = f * f, f3v = f2 * f;
    f3 w0 = (1.0f - 3.0f * f + 3.0f * f2 - f3v) / 6.0f;
    f3 w1 = (4.0f - 6.0f * f2 + 3.0f * f3v) / 6.0f;
    f3 w2 = (1.0f + 3.0f * f + 3.0f * f2 - 3.0f * f3v) / 6.0f;
    f3 w3 = f3v / 6.0f;
    f3 g0 = w0 + w1, g1 = w2 + w3;
    f3 a = i - 1.0f + w1 / g0, b = i + 1.0f + w3 / g1;  // the folded taps, in texels
    float4 z0 = f4add(f4mul(g0.y, f4add(f4mul(g0.x, lt_fetch(v, a.x, a.y, a.z)), f4mul(g1.x, lt_fetch(v, b.x, a.y, a.z)))),
                      f4mul(g1.y, f4add(f4mul(g0.x, lt_fetch(v, a.x, b.y, a.z)), f4mul(g1.x, lt_fetch(v, b.x, b.y, a.z)))));
    float4 z1 = f4add(f4mul(g0.y, f4add(f4mul(g0.x, lt_fetch(v, a.x, a.y, b.z)), f4mul(g1.x, lt_fetch(v, b.x, a.y, b.z)))),
                      f4mul(g1.y, f4add(f4mul(g0.x, lt_fetch(v, a.x, b.y, b.z)), f4mul(g1.x, lt_fetch(v, b.x, b.y, b.z)))));
    return f4add(f4mul(g0.z, z0), f4mul(g1.z, z1));
}
// common.glsl:154-157
__device__ __forceinline__ float4 lighting_lookup(const PtArgs& A, const LightTex& v, f3 tc) {
    return A.u.env[1] > 0.5f ? lt_cubic(v, tc) : lt_linear(v, tc);
}

// common.glsl:483-486: cosine-weighted mean light map radiance around `n`
// (32 x 16 RGBA16F, linear, clamped to the edge).
__device__ __noinline__ f3 env_map_diffuse(const PtArgs& A, f3 n) {
    float2 uv = env_uv(A, n);
    const int W = 32, H = 16;
    float x = uv.x * (float)W - 0.5f, y = uv.y * (float)H - 0.5f;
    int i0 = (int)floorf(x), j0 = (int)floorf(y);
    float a = x - (float)i0, b = y - (float)j0;
    f3 c = mk(0.0f);
    for (int dj = 0; dj < 2; dj++)
        for (int di = 0; di < 2; di++) {
            int i = clampi(i0 + di, 0, W - 1), j = clampi(j0 + dj, 0, H - 1);
            ushort4 t = __ldg(A.env_diffuse + j * W + i);
            float w = (di ? a : 1.0f - a) * (dj ? b : 1.0f - b);
            c += mk(h2f(t.x), h2f(t.y), h2f(t.z)) * w;
        }
    return U3(A.u.ambient) * c;
}

// dvr.comp:76-96: the first surface a ray meets, bisected between the previous
// sample and this one for where the opacity reaches half of this sample's.
__device__ __noinline__ f3 refine_surface(const PtArgs& A, f3 idx, f3 d_idx, float step_mm, float target) {
    float inside = 0.0f, outside = -step_mm;
    for (int i = 0; i < 5; i++) {
        float mid = 0.5f * (inside + outside);
        f3 at = idx + d_idx * mid;
        const uint32_t mode = (uint32_t)A.u.labels[0];
        f3 unused;
        bool no_grad;
        bool opaque = (mode >= 2u ? labelled_at<false>(A, at, mode, unused, no_grad)
                                  : labelled(A, tf_point(A, density_view(A, at)), at)).extinction >= target;
        inside = opaque ? mid : inside;
        outside = opaque ? outside : mid;
    }
    return idx + d_idx * inside;
}

// dvr.comp:98-141: light reflected and scattered towards the viewer at a
// sample (lighting volumes, BRDF, subsurface, ambient); ghosted structures'
// opacity `alpha` is rescaled to their shell.
__device__ __noinline__ f3 shade_sample(const PtArgs& A, const LightTex& SV, const LightTex& AV, f3 idx, Sample s,
                                        f3 v, int cap_plane, float cut, float step_mm, bool has_grad, f3 grad,
                                        float& alpha) {
    m3 to_index = w2i3(A);
    f3 l = U3(A.u.light_dir);
    float light = A.u.light_dir[3];
    f3 n;
    float surfaceness;
    float extinction_scale = has_grad ? surface_frame<true>(A, idx, s, v, cap_plane, cut, 1.5f * step_mm, n,
                                                            surfaceness, grad)
                                      : surface_frame(A, idx, s, v, cap_plane, cut, 1.5f * step_mm, n, surfaceness);
    SurfaceNoise noise;
    apply_surface_texture(A, idx, s, noise);
    if (s.ghost) alpha = 1.0f - expf(-s.extinction * extinction_scale * step_mm);
    f3 shadow_at = index_to_tex(A, idx + mul(to_index, n * (1.5f * A.u.light_cells[0] * surfaceness)));
    f3 ao_at = index_to_tex(A, idx + mul(to_index, n * (A.u.light_cells[1] * surfaceness)));
    float shadow_t = A.u.lighting[0] != 0u ? lighting_lookup(A, SV, shadow_at).w : 1.0f;
    f3 sss_at = index_to_tex(A, idx - mul(to_index, n * (A.u.subsurface[3] * surfaceness)));
    f3 diffused = mk(1.0f);
    if (A.u.lighting[0] != 0u) {
        float4 dl = lighting_lookup(A, SV, sss_at);
        diffused = mk(dl.x, dl.y, dl.z);
    }
    float occlusion = A.u.lighting[1] != 0u ? lighting_lookup(A, AV, ao_at).x : 1.0f;
    n = bump_normal(A, s, n, noise);
    n = dot(n, v) < 0.0f ? -n : n;
    float nl = gmax(dot(n, l), 0.0f);
    f3 diffuse;
    f3 specular = brdf_coated(n, v, l, s, diffuse);
    f3 surface = (specular + diffuse) * (1.0f - s.subsurface) * nl * shadow_t + diffuse * s.subsurface * diffused;
    f3 volume = s.albedo / (4.0f * PI) * mix3(mk(shadow_t), diffused, s.subsurface);
    f3 direct = mix3(volume, surface, surfaceness) * light;
    f3 ambient_light = A.u.lighting[3] == 2u
                           ? mix3(U3(A.u.ambient), env_map_diffuse(A, n), surfaceness * (1.0f - s.subsurface))
                           : U3(A.u.ambient);
    f3 ambient = s.albedo * ambient_light * occlusion;
    return direct + ambient;
}

}  // namespace

// ao.comp: mean transmittance over 16 directions within 15 mm, remapped so a
// flat surface is unoccluded; one thread per occlusion voxel.
__global__ void __launch_bounds__(64) k_ao(const __grid_constant__ PtArgs A, uint16_t* __restrict__ out, int ax, int ay,
                                           int az) {
    int x = blockIdx.x * 4 + (threadIdx.x & 3), y = blockIdx.y * 4 + ((threadIdx.x >> 2) & 3),
        z = blockIdx.z * 4 + (threadIdx.x >> 4);
    if (x >= ax || y >= ay || z >= az) return;
    f3 center = tex_to_index(A, mk(((float)x + 0.5f) / (float)ax, ((float)y + 0.5f) / (float)ay,
                                   ((float)z + 0.5f) / (float)az));
    m3 to_index = w2i3(A);
    const float dt = 15.0f / 8.0f;
    float visible = 0.0f;
    for (int i = 0; i < 16; i++) {
        float zz = 1.0f - ((float)i + 0.5f) * (2.0f / 16.0f);
        float r = sqrtf(1.0f - zz * zz);
        float phi = (float)i * 2.39996323f;
        f3 d = mul(to_index, mk(r * cosf(phi), r * sinf(phi), zz));
        float depth = 0.0f;
        for (int j = 0; j < 8; j++) depth += sample_point(A, center + d * (((float)j + 0.5f) * dt)).extinction * dt;
        visible += expf(-depth);
    }
    out[((long)z * ay + y) * ax + x] = f2h(gmin(2.0f * visible / 16.0f, 1.0f));
}

// shadow.comp, in two parts. What a voxel of the shadow volume lets through on
// the way from the slice before it, directly and diffused, is a matter of its
// own sample: k_shadow_factors takes it for the whole volume at once (x, y, z:
// the diffused light's factors, w: the direct light's).
struct ShadowSweep {
    f3 dims, l_idx;  // the volume's texels; one step towards the light is l_idx * s
    float s;
};
__device__ __forceinline__ ShadowSweep shadow_sweep_of(const PtArgs& A, int sx, int sy, int sz, int axis) {
    ShadowSweep w;
    w.dims = mk((float)sx, (float)sy, (float)sz);
    w.l_idx = mul(w2i3(A), U3(A.u.light_dir)) * (w.dims / U3(A.u.dims));
    w.s = 1.0f / gmax(fabsf(comp3(w.l_idx, axis)), 1e-6f);
    return w;
}
__device__ __forceinline__ float4 shadow_factors(const PtArgs& A, const ShadowSweep& w, f3 here) {
    f3 prev = here + w.l_idx * w.s;
    f3 mid_tex = ((here + prev) * 0.5f + 0.5f) / w.dims;
    Sample m = sample_point(A, tex_to_index(A, mid_tex));
    f3 chroma = m.albedo / gmax(gmax(m.albedo.x, gmax(m.albedo.y, m.albedo.z)), 1e-4f);
    f3 ie = m.extinction * A.u.subsurface[1] * (1.2f - chroma);
    return make_float4(expf(-ie.x * w.s), expf(-ie.y * w.s), expf(-ie.z * w.s), expf(-m.extinction * w.s));
}
__global__ void __launch_bounds__(128) k_shadow_factors(const __grid_constant__ PtArgs A, float4* __restrict__ out,
                                                        int sx, int sy, int sz, int axis) {
    const int x = blockIdx.x * 8 + (threadIdx.x & 7), y = blockIdx.y * 4 + ((threadIdx.x >> 3) & 3),
              z = blockIdx.z * 4 + (threadIdx.x >> 5);
    if (x >= sx || y >= sy || z >= sz) return;
    out[((long)z * sy + y) * sx + x] =
        shadow_factors(A, shadow_sweep_of(A, sx, sy, sz, axis), mk((float)x, (float)y, (float)z));
}
// One slice of the sweep from the previous one: the light that reaches the
// slice before it, in five linear lookups, times the factors (from `factors`,
// or taken here where the caller has no room for them). The slices are a chain
// of dependent launches, so what is not part of the chain is kept out of it.
// Measured on 301 x 255 x 203 voxels: factors in the slices 17.5 us for each of 151;
// ahead of them 43 us in all. The loads of a lookup are unconditional but for their
// predicates, so that they overlap (with a branch per texel the sweep below took
// 1.12, 1.14, 0.78, 0.76 ms).
template <bool GIVEN>
__global__ void __launch_bounds__(64) k_shadow_slice(const __grid_constant__ PtArgs A, ushort4* __restrict__ vol,
                                                     const float4* __restrict__ factors, int sx, int sy, int sz,
                                                     int axis, int slice) {
    int u_axis = (axis + 1) % 3, v_axis = (axis + 2) % 3;
    int pu = blockIdx.x * 8 + (threadIdx.x & 7), pv = blockIdx.y * 8 + (threadIdx.x >> 3);
    int sdim[3] = {sx, sy, sz};
    int p[3];
    p[axis] = slice;
    p[u_axis] = pu;
    p[v_axis] = pv;
    if (p[0] >= sx || p[1] >= sy || p[2] >= sz || pu >= sdim[u_axis] || pv >= sdim[v_axis]) return;
    const ShadowSweep w = shadow_sweep_of(A, sx, sy, sz, axis);
    const long at = ((long)p[2] * sy + p[1]) * sx + p[0];
    f3 here = mk((float)p[0], (float)p[1], (float)p[2]);
    // A chained launch's set-up overlaps the slice before it, whose end (and so that
    // of all before) it waits for here. Its blocks come once that slice's have ended:
    // let in earlier (launch_dependents), they would have to read past L1, which may
    // hold sectors from before, and cost more than they gain (below).
    const float4 f = GIVEN ? __ldg(factors + at) : shadow_factors(A, w, here);
    if (GIVEN) asm volatile("griddepcontrol.wait;" ::: "memory");
    f3 prev = here + w.l_idx * w.s;
    LightVol V{vol, sx, sy, sz, axis, slice};
    float4 back = lv_linear<GIVEN>(V, (prev + 0.5f) / w.dims);
    float direct = back.w * f.w;
    f3 axis_u = mk(0.0f), axis_v = mk(0.0f);
    set3(axis_u, u_axis, A.u.subsurface[2]);
    set3(axis_v, v_axis, A.u.subsurface[2]);
    // The products' sum rounded one way whether the loop is unrolled or not.
    f3 gathered = mk(__fmul_rn(0.4f, back.x), __fmul_rn(0.4f, back.y), __fmul_rn(0.4f, back.z));
#pragma unroll
    for (int i = 0; i < 4; i++) {
        f3 offset = (i & 1) == 0 ? axis_u : axis_v;
        offset *= i < 2 ? 1.0f : -1.0f;
        float4 t = lv_linear<GIVEN>(V, (prev + offset + 0.5f) / w.dims);
        gathered = mk(fmaf(0.15f, t.x, gathered.x), fmaf(0.15f, t.y, gathered.y), fmaf(0.15f, t.z, gathered.z));
    }
    f3 indirect = gathered * mk(f.x, f.y, f.z);
    vol[at] = make_ushort4(f2h(indirect.x), f2h(indirect.y), f2h(indirect.z), f2h(direct));
}

// dvr.comp: one ray per pixel, emission-absorption with single scattering. Bound
// by instruction issue: a lit sample costs thousands of instructions (the
// surface's relief and texture noises, six mask fetches, three lighting
// lookups), the steps between them a few hundred. A warp (8 x 4 pixels) marches
// until `gather` of its rays stand at a sample to light, or none marches, and
// lights those together. Measured on 512 x 512 x 400 at 1024^2: 28.6 ms per
// frame with the lighting inside each step and 16 noises per relief, 17.4 with
// the phases and masks read first, 14.4 with the shared noises (relief_heights).
// Gathering 1, 8, 16, 24, 28, 32 rays: 19.0, 18.6, 18.2, 17.3, 17.0, 17.8 ms
// there and 21.0, 20.9, 20.6, 21.9, 22.9, 22.4 for a 511 x 387 clip drag.
// Without labels a lit sample has no relief and no texture and costs little more
// than a step, so rays that wait for company only lose time: dvr_gather.
#ifndef VV_DVR_MIN_BLOCKS
#define VV_DVR_MIN_BLOCKS 4
#endif
#ifndef VV_DVR_GATHER
#define VV_DVR_GATHER 24
#endif
// MASKS_FIRST: for the modes that draw labels alone, without pre-integration. A
// drawn label replaces what the transfer function gives there, so a sample outside
// the masks needs no density (labelled_at); pre-integrated segments take every
// step's. Launched as the one-lane form of k_dvr_masks only (VV_DVR_LANES=1).
template <bool MASKS_FIRST>
__global__ void __launch_bounds__(64, VV_DVR_MIN_BLOCKS) k_dvr(const __grid_constant__ PtArgs A, const LightTex SV,
                                                               const LightTex AV, int gather) {
    int px = blockIdx.x * 8 + (threadIdx.x & 7), py = blockIdx.y * 8 + (threadIdx.x >> 3);
    const bool inside = px < (int)A.u.flags[2] && py < (int)A.u.flags[3];
    float nx = ((float)px + 0.5f) / (float)A.u.flags[2] * 2.0f - 1.0f;
    float ny = ((float)py + 0.5f) / (float)A.u.flags[3] * 2.0f - 1.0f;
    f3 dir = normalize(U3(A.u.forward) + nx * U3(A.u.right) - ny * U3(A.u.up));
    const float* m4 = A.u.w2i;
    f3 e = U3(A.u.eye);
    f3 o_idx = mk(m4[0] * e.x + m4[4] * e.y + m4[8] * e.z + m4[12], m4[1] * e.x + m4[5] * e.y + m4[9] * e.z + m4[13],
                  m4[2] * e.x + m4[6] * e.y + m4[10] * e.z + m4[14]);
    m3 to_index = w2i3(A);
    f3 d_idx = mul(to_index, dir);
    f3 inv_d = brick_inv_dir(d_idx);
    float2 t = intersect_volume(A, o_idx, d_idx);
    float step_mm = A.u.dims[3];
    bool preintegrate = A.u.lighting[2] != 0u;
    const uint32_t mode = (uint32_t)A.u.labels[0];
    f3 v = -dir;
    f3 radiance = mk(0.0f);
    float transmittance = 1.0f;
    bool refined = false;
    enum { OUT, MARCH, SHADE };
    int state = inside && t.x < t.y ? MARCH : OUT;
    float tt = 0.0f, prev_density = -1.0f, front_density = -1.0f;
    f3 idx, grad = mk(0.0f);
    Sample s;
    int cap_plane = -1;
    float cut = 0.0f;
    bool has_grad = false, segment = false;
    if (state == MARCH) {
        tt = t.x + ign((float)px, (float)py) * step_mm;
        if (!MASKS_FIRST) prev_density = density_view(A, o_idx + d_idx * (tt - step_mm));
    }
    for (;;) {
        unsigned shading;
        for (;;) {
            const unsigned marching = __ballot_sync(0xffffffffu, state == MARCH);
            shading = __ballot_sync(0xffffffffu, state == SHADE);
            if (!marching || __popc(shading) >= gather) break;
            if (state != MARCH) continue;
            if (!(tt < t.y && transmittance > 0.01f)) {
                state = OUT;
                continue;
            }
            idx = o_idx + d_idx * tt;
            float maj = A.u.path[3] == 0u ? 1e30f : __ldg(A.majorant + brick_index(A, idx));
            if (maj <= 0.0f) {
                tt += brick_exit(idx, inv_d, far_planes(inv_d));
                prev_density = -1.0f;
                tt += step_mm;
                continue;
            }
            cut = clip_depth(A, idx, cap_plane);
            if (cut > 0.0f) {
                prev_density = -1.0f;
                tt += step_mm;
                continue;
            }
            if (MASKS_FIRST) {
                s = labelled_at<true>(A, idx, mode, grad, has_grad);
            } else {
                // With smooth sampling the gradient comes with the density: a
                // sample shaded where it was taken needs no second read.
                has_grad = A.u.env[1] > 0.5f;
                float density = has_grad ? density_cubic_with_gradient(A, idx, grad) : density_tri(A, idx);
                front_density = prev_density;
                segment = preintegrate && front_density >= 0.0f;
                s = segment ? tf_segment(A, front_density, density) : tf_point(A, density);
                prev_density = density;
                s = labelled(A, s, idx);
            }
            if (s.extinction <= 0.0f) tt += step_mm;
            else state = SHADE;
        }
        if (!shading) break;
        if (state == SHADE) {
            float alpha = 1.0f - expf(-s.extinction * step_mm);
            if (segment && alpha > 0.2f && transmittance > 0.5f && s.label == 0u &&
                fabsf(prev_density - front_density) > 1e-4f) {
                idx = idx - d_idx * (step_mm * (1.0f - preint_half_depth(A, front_density, prev_density)));
                has_grad = false;
            } else if (!refined && alpha > 0.2f && transmittance > 0.9f) {
                refined = true;
                idx = refine_surface(A, idx, d_idx, step_mm, 0.5f * s.extinction);
                has_grad = false;
            }
            f3 lit = shade_sample(A, SV, AV, idx, s, v, cap_plane, cut, step_mm, has_grad, grad, alpha);
            radiance += transmittance * alpha * lit;
            transmittance *= 1.0f - alpha;
            tt += step_mm;
            state = MARCH;
        }
    }
    if (inside)
        A.hdr[(long)py * A.width + px] = make_ushort4(f2h(radiance.x), f2h(radiance.y), f2h(radiance.z),
                                                      f2h(transmittance));
}

// k_dvr for the modes that draw labels alone, without pre-integration: two or
// four lanes per ray. Where a ray samples depends on the volume only, not on
// what it has gathered, so the lanes of a ray take its next samples in kept,
// non-empty bricks side by side and light those that need it together; what
// they found is then composited in the ray's order, with the same sums. One
// lane per ray left the image waiting for its slowest warps (rays along a
// translucent skull light hundreds of samples in turn, 3.4 warps active per SM).
// The one decision that depends on the samples before is the refinement of the
// first opaque surface: a sample that might be it behind a ghost, whose opacity
// its lighting decides, waits with those after it for the next turn. Measured
// against one lane per ray: 13.6 -> 9.2 ms for the 1024^2 frame, 20.6 -> 10.2 for
// the 511 x 387 clip drag.
constexpr int rays_x(int lanes) { return lanes == 4 ? 4 : 2; }  // a warp's rays: 4 x 2, or 2 x 8 pixels
template <int RAY_LANES>
__global__ void __launch_bounds__(64, VV_DVR_MIN_BLOCKS)
    k_dvr_masks(const __grid_constant__ PtArgs A, const LightTex SV, const LightTex AV) {
    constexpr unsigned ALL = 0xffffffffu;
    constexpr int RAYS_X = rays_x(RAY_LANES), RAYS_Y = 32 / RAY_LANES / RAYS_X;
    const int lane = (int)(threadIdx.x & 31u), sub = lane & (RAY_LANES - 1), first = lane - sub;
    const int ray = lane / RAY_LANES, px = blockIdx.x * RAYS_X + ray % RAYS_X,
              py = (blockIdx.y * 2 + (int)(threadIdx.x >> 5)) * RAYS_Y + ray / RAYS_X;
    constexpr unsigned GROUP = (1u << RAY_LANES) - 1u;
    const bool inside = px < (int)A.u.flags[2] && py < (int)A.u.flags[3];
    float nx = ((float)px + 0.5f) / (float)A.u.flags[2] * 2.0f - 1.0f;
    float ny = ((float)py + 0.5f) / (float)A.u.flags[3] * 2.0f - 1.0f;
    f3 dir = normalize(U3(A.u.forward) + nx * U3(A.u.right) - ny * U3(A.u.up));
    const float* m4 = A.u.w2i;
    f3 e = U3(A.u.eye);
    f3 o_idx = mk(m4[0] * e.x + m4[4] * e.y + m4[8] * e.z + m4[12], m4[1] * e.x + m4[5] * e.y + m4[9] * e.z + m4[13],
                  m4[2] * e.x + m4[6] * e.y + m4[10] * e.z + m4[14]);
    m3 to_index = w2i3(A);
    f3 d_idx = mul(to_index, dir);
    f3 inv_d = brick_inv_dir(d_idx);
    float2 t = intersect_volume(A, o_idx, d_idx);
    const float step_mm = A.u.dims[3];
    const uint32_t mode = (uint32_t)A.u.labels[0];
    f3 v = -dir;
    // The ray's: the same in its lanes.
    f3 radiance = mk(0.0f);
    float transmittance = 1.0f, pos = INFINITY;  // past its end: a ray that misses the volume never marches
    bool refined = false, marching = inside && t.x < t.y;
    // The lane's sample.
    bool lit = false, has_grad = false;
    f3 idx = mk(0.0f), grad = mk(0.0f);
    Sample s;
    s.extinction = 0.0f;
    s.ghost = false;
    int cap_plane = -1;
    float cut = 0.0f;
    if (marching) pos = t.x + ign((float)px, (float)py) * step_mm;
    for (;;) {
        unsigned waiting;
        for (;;) {
            waiting = __ballot_sync(ALL, lit);
            if ((waiting >> first) & GROUP) marching = false;  // a ray lights before it marches on
            const unsigned march = __ballot_sync(ALL, marching);
            if (!march || __popc(waiting) >= VV_DVR_GATHER) break;
            if (!marching) continue;
            // The ray's next samples; this lane's is number `sub`.
            bool mine = false;
            int found = 0;
            while (found < RAY_LANES && pos < t.y) {
                const f3 at = o_idx + d_idx * pos;
                const float maj = A.u.path[3] == 0u ? 1e30f : __ldg(A.majorant + brick_index(A, at));
                if (maj <= 0.0f) {
                    pos += brick_exit(at, inv_d, far_planes(inv_d));
                } else {
                    int plane;
                    const float c = clip_depth(A, at, plane);
                    if (c <= 0.0f) {
                        if (found == sub) {
                            mine = true;
                            idx = at;
                            cut = c;
                            cap_plane = plane;
                        }
                        found++;
                    }
                }
                pos += step_mm;
            }
            if (mine) {
                s = labelled_at<true>(A, idx, mode, grad, has_grad);
                lit = !(s.extinction <= 0.0f);
            }
            if (found == 0) marching = false;
        }
        if (!waiting) break;
        // Light the samples whose place in the ray's order decides nothing more
        // about them: all, but for a possible first surface behind a ghost.
        const float alpha_in = 1.0f - expf(-s.extinction * step_mm);
        float before = transmittance;  // bounds what reaches a sample, exact until a ghost is passed
        bool seen = refined, exact = true, refine = false;
        int stop = RAY_LANES;
#pragma unroll
        for (int i = 0; i < RAY_LANES; i++) {
            const bool li = __shfl_sync(ALL, (int)lit, first + i) != 0;
            const bool gi = __shfl_sync(ALL, (int)s.ghost, first + i) != 0;
            const float ai = __shfl_sync(ALL, alpha_in, first + i);
            if (!li || stop < RAY_LANES) continue;
            if (!seen && ai > 0.2f && before > 0.9f) {
                if (!exact) {
                    stop = i;
                    continue;
                }
                seen = true;
                if (i == sub) refine = true;
            }
            if (gi) exact = false;
            else before *= 1.0f - ai;
        }
        const bool now = lit && sub < stop;
        float alpha = alpha_in;
        f3 colour = mk(0.0f);
        if (now) {
            if (refine) {
                idx = refine_surface(A, idx, d_idx, step_mm, 0.5f * s.extinction);
                has_grad = false;
            }
            colour = shade_sample(A, SV, AV, idx, s, v, cap_plane, cut, step_mm, has_grad, grad, alpha);
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < RAY_LANES; i++) {
            const bool ni = __shfl_sync(ALL, (int)now, first + i) != 0;
            const bool ri = __shfl_sync(ALL, (int)refine, first + i) != 0;
            const float ai = __shfl_sync(ALL, alpha, first + i);
            const f3 ci = mk(__shfl_sync(ALL, colour.x, first + i), __shfl_sync(ALL, colour.y, first + i),
                             __shfl_sync(ALL, colour.z, first + i));
            if (!ni || !(transmittance > 0.01f)) continue;
            if (ri) refined = true;
            radiance += transmittance * ai * ci;
            transmittance *= 1.0f - ai;
        }
        if (now || !(transmittance > 0.01f)) lit = false;
        const unsigned left = __ballot_sync(ALL, lit);
        if (!((left >> first) & GROUP)) marching = inside && transmittance > 0.01f && pos < t.y;
    }
    if (inside && sub == 0)
        A.hdr[(long)py * A.width + px] = make_ushort4(f2h(radiance.x), f2h(radiance.y), f2h(radiance.z),
                                                      f2h(transmittance));
}

cudaError_t launch_ao(const PtArgs& a, uint16_t* out, int ax, int ay, int az, cudaStream_t s) {
    dim3 g((ax + 3) / 4, (ay + 3) / 4, (az + 3) / 4);
    k_ao<<<g, 64, 0, s>>>(a, out, ax, ay, az);
    return cudaGetLastError();
}

cudaError_t launch_shadow_sweep(const PtArgs& a, ushort4* vol, int sx, int sy, int sz, int axis, int sign,
                                float4* factors, cudaStream_t s, int* launches) {
    int sd[3] = {sx, sy, sz};
    int u_axis = (axis + 1) % 3, v_axis = (axis + 2) % 3;
    dim3 g((sd[u_axis] + 7) / 8, (sd[v_axis] + 7) / 8);
    cudaError_t e = cudaMemsetAsync(vol, 0, (size_t)sx * sy * sz * sizeof(ushort4), s);
    if (e != cudaSuccess) return e;
    if (factors) {
        k_shadow_factors<<<dim3((sx + 7) / 8, (sy + 3) / 4, (sz + 3) / 4), 128, 0, s>>>(a, factors, sx, sy, sz, axis);
        *launches += 1;
    }
    int n = sd[axis];
    for (int i = 0; i < n; i++) {
        int slice = sign > 0 ? n - 1 - i : i;
        if (factors) {
            // Programmatic dependent launch. A sweep of 126 x 122 x 94 texels towards the
            // default light, along x, y, z, factors and copy included: 0.86, 0.81, 0.63,
            // 0.54 ms (plain launches that take the factors themselves 2.31, 2.13, 1.99,
            // 1.88). With launch_dependents and loads past L1 the branching form took
            // 1.37, 1.82, 1.04, 1.14 instead of its 1.12, 1.14, 0.78, 0.76.
            cudaLaunchConfig_t config = {};
            config.gridDim = g;
            config.blockDim = dim3(64);
            config.stream = s;
            cudaLaunchAttribute early[1];
            early[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            early[0].val.programmaticStreamSerializationAllowed = i > 0;  // the first follows the factors in full
            config.attrs = early;
            config.numAttrs = 1;
            e = cudaLaunchKernelEx(&config, k_shadow_slice<true>, a, vol, (const float4*)factors, sx, sy, sz, axis, slice);
            if (e != cudaSuccess) return e;
        } else {
            k_shadow_slice<false><<<g, 64, 0, s>>>(a, vol, nullptr, sx, sy, sz, axis, slice);
        }
    }
    *launches += n;
    return cudaGetLastError();
}

// The texture array of a lighting volume: texel (x, y, z) of the volume at
// (x + 1, y + 1, z + 1), white (1, 1, 1, 1) around it.
__global__ void k_pad_lighting(const uint16_t* __restrict__ vol, int channels, int w, int h, int d,
                               cudaSurfaceObject_t surf) {
    int x = blockIdx.x * 8 + (threadIdx.x & 7), y = blockIdx.y * 8 + (threadIdx.x >> 3), z = blockIdx.z;
    if (x >= w + 2 || y >= h + 2 || z >= d + 2) return;
    const uint16_t one = 0x3c00u;  // 1.0 in binary16
    bool inside = x >= 1 && y >= 1 && z >= 1 && x <= w && y <= h && z <= d;
    long i = inside ? ((long)(z - 1) * h + (y - 1)) * w + (x - 1) : 0;
    if (channels == 4) {
        ushort4 t = inside ? __ldg((const ushort4*)vol + i) : make_ushort4(one, one, one, one);
        surf3Dwrite(t, surf, x * (int)sizeof(ushort4), y, z);
    } else {
        uint16_t t = inside ? __ldg(vol + i) : one;
        surf3Dwrite(t, surf, x * (int)sizeof(uint16_t), y, z);
    }
}

cudaError_t launch_pad_lighting(const uint16_t* vol, int channels, int w, int h, int d, cudaSurfaceObject_t surf,
                                cudaStream_t s) {
    dim3 g((w + 2 + 7) / 8, (h + 2 + 7) / 8, d + 2);
    k_pad_lighting<<<g, 64, 0, s>>>(vol, channels, w, h, d, surf);
    return cudaGetLastError();
}

// Rays that k_dvr gathers before it lights them. 512^2, a head of 256 x 256 x 200, the
// transfer function alone: 1, 4, 8, 16, 24 rays 2.6, 2.2, 2.7, 3.0, 3.7 ms, pre-integrated
// 2.8, 2.8, 3.1, 4.2, 5.0; lighting inside each step 2.7 and 2.9. With labels (Tint)
// 7.4, 7.6, 6.3, 6.5, 6.8 ms, and pre-integrated Hybrid 8.0 to 8.2 for all.
static int dvr_gather(const PtArgs& a) { return a.u.labels[0] >= 1.0f ? VV_DVR_GATHER : 4; }

cudaError_t launch_dvr(const PtArgs& a, const LightTex& shadow, const LightTex& ao, cudaStream_t s) {
    // Lanes per ray: four below 3 * 2^17 pixels, where the slowest rays set the
    // time, two above, where lanes past a ray's end cost more than they save, and
    // one where a sample needs the one before it (pre-integration, transfer
    // function modes). Two against four lanes, ms per frame, head/neck 512 x 512
    // x 400: 3.88 / 1.95 at 256^2, 4.54 / 3.52 at 512^2, 5.58 / 4.73 at 640^2, 6.53 /
    // 6.30 at 768^2, 9.20 / 10.27 at 1024^2; 256 x 256 x 200: 3.06 / 2.90 at 512^2,
    // 3.71 / 4.27 at 640^2. The two are equal near 800^2 on the larger volume and
    // near 550^2 on the smaller: the line lies between. VV_DVR_LANES overrides (1, 2 or 4; other
    // values are ignored).
    const bool masks = a.u.labels[0] >= 2.0f && a.u.lighting[2] == 0u;
    int lanes = 1;
    if (masks) {
        lanes = (uint64_t)a.width * a.height < 3u << 17 ? 4 : 2;
        const char* e = std::getenv("VV_DVR_LANES");
        const int asked = e ? std::atoi(e) : 0;
        if (asked == 1 || asked == 2 || asked == 4) lanes = asked;
    }
    if (lanes == 4)
        k_dvr_masks<4><<<dim3((a.width + 3) / 4, (a.height + 3) / 4), 64, 0, s>>>(a, shadow, ao);
    else if (lanes == 2)
        k_dvr_masks<2><<<dim3((a.width + 1) / 2, (a.height + 15) / 16), 64, 0, s>>>(a, shadow, ao);
    else if (masks)
        k_dvr<true><<<dim3((a.width + 7) / 8, (a.height + 7) / 8), 64, 0, s>>>(a, shadow, ao, dvr_gather(a));
    else
        k_dvr<false><<<dim3((a.width + 7) / 8, (a.height + 7) / 8), 64, 0, s>>>(a, shadow, ao, dvr_gather(a));
    return cudaGetLastError();
}

}  // namespace VV_FMT_NS
}  // namespace vv
