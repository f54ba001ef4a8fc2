// vv_volume.cu — the per-volume passes: density upload, normals, label masks,
// brick majorants, and the unbricking copy used by readback.
//
// These passes are HBM-bound integer/FP stencils. Their arithmetic uses
// round-to-nearest intrinsics (__fmul_rn, __fadd_rn, ...) in the order the
// reference shaders evaluate it, so that their outputs match the reference bit
// for bit (the normals and masks are quantised, and a fused multiply-add could
// move a value across a rounding boundary).
#include <cuda_runtime.h>

#include <cuda_bf16.h>

#include "vv_device.cuh"
#include "vv_kernels.h"

namespace vv {

static const float HU_MIN = -1024.0f, HU_MAX = 3071.0f;

// hu_to_unorm16 (crates/render/src/transfer.rs:121-124) into the bricked
// layout; one thread per bricked element, reading the x-fastest source. The
// precision variants store the same normalised density t as FP16 or BF16
// (rounded to nearest even) or FP32 instead of round(t * 65535).
__global__ void k_density(const int16_t* __restrict__ hu, void* __restrict__ out, Vol v) {
    long e = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= vol_elems(v)) return;
    int x, y, z;
    vcoord(v, e, x, y, z);
    float t = 0.0f;
    if (x < v.nx && y < v.ny && z < v.nz) {
        float h = (float)hu[((long)z * v.ny + y) * v.nx + x];
        t = __fdiv_rn(__fsub_rn(h, HU_MIN), __fsub_rn(HU_MAX, HU_MIN));
        t = fminf(fmaxf(t, 0.0f), 1.0f);
    }
    switch (v.dfmt) {
        case DF_FP16: ((uint16_t*)out)[e] = __half_as_ushort(__float2half_rn(t)); break;
        case DF_BF16: ((uint16_t*)out)[e] = __bfloat16_as_ushort(__float2bfloat16_rn(t)); break;
        case DF_FP32: ((float*)out)[e] = t; break;
        default: ((uint16_t*)out)[e] = (uint16_t)roundf(__fmul_rn(t, 65535.0f));
    }
}

__device__ __forceinline__ float dens(const void* d, const Vol& v, int x, int y, int z) {
    x = clampi(x, 0, v.nx - 1);
    y = clampi(y, 0, v.ny - 1);
    z = clampi(z, 0, v.nz - 1);
    return density_texel(d, v.dfmt, voff(v, x, y, z));
}

__device__ __forceinline__ int8_t to_snorm8(float f) {
    return (int8_t)rintf(__fmul_rn(fminf(fmaxf(f, -1.0f), 1.0f), 127.0f));
}

// normals.comp:14-37: 3x3x3 Sobel, /32, world transform, -g/|g| and clamp(|g|*400).
__global__ void k_normals(const void* __restrict__ d, uint32_t* __restrict__ out, Vol v, m3 w) {
    long e = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= vol_elems(v)) return;
    int x, y, z;
    vcoord(v, e, x, y, z);
    if (x >= v.nx || y >= v.ny || z >= v.nz) { out[e] = 0; return; }
    float gx = 0.0f, gy = 0.0f, gz = 0.0f;
    for (int a = -1; a <= 1; a++)
        for (int b = -1; b <= 1; b++) {
            float wt = (float)((2 - abs(a)) * (2 - abs(b)));
            gx = __fadd_rn(gx, __fmul_rn(wt, __fsub_rn(dens(d, v, x + 1, y + a, z + b), dens(d, v, x - 1, y + a, z + b))));
            gy = __fadd_rn(gy, __fmul_rn(wt, __fsub_rn(dens(d, v, x + a, y + 1, z + b), dens(d, v, x + a, y - 1, z + b))));
            gz = __fadd_rn(gz, __fmul_rn(wt, __fsub_rn(dens(d, v, x + a, y + b, z + 1), dens(d, v, x + a, y + b, z - 1))));
        }
    gx = __fdiv_rn(gx, 32.0f);
    gy = __fdiv_rn(gy, 32.0f);
    gz = __fdiv_rn(gz, 32.0f);
    // transpose(mat3(world_to_index)) * g
    auto dotrn = [](f3 c, float p, float q, float r) {
        return __fadd_rn(__fadd_rn(__fmul_rn(c.x, p), __fmul_rn(c.y, q)), __fmul_rn(c.z, r));
    };
    float wx = dotrn(w.c0, gx, gy, gz), wy = dotrn(w.c1, gx, gy, gz), wz = dotrn(w.c2, gx, gy, gz);
    float l = __fsqrt_rn(dotrn(mk(wx, wy, wz), wx, wy, wz));
    float nx = 0.0f, ny = 0.0f, nz = 0.0f;
    if (l > 1e-7f) {
        nx = __fdiv_rn(-wx, l);
        ny = __fdiv_rn(-wy, l);
        nz = __fdiv_rn(-wz, l);
    }
    float s = fminf(fmaxf(__fmul_rn(l, 400.0f), 0.0f), 1.0f);
    uint32_t q = (uint32_t)(uint8_t)to_snorm8(nx) | ((uint32_t)(uint8_t)to_snorm8(ny) << 8) |
                 ((uint32_t)(uint8_t)to_snorm8(nz) << 16) | ((uint32_t)(uint8_t)to_snorm8(s) << 24);
    out[e] = q;
}

// --------------------------------------------------------------------- masks
struct MaskArgs {
    Vol v;
    const void* density;
    const uint8_t* labels;
    const uint8_t* soft;  // RGBA8 nodes, x-fastest
    int sdims[3];
    int soft_push[4];     // axes, flip bits | 8 = present
    int margin;
    int mode;
    const float4* colors; // label_colors table
    float dims[3];
    uint8_t* cls;         // soft grid prepared for this visibility (k_soft_nodes, k_soft_flags)
    uint8_t* flags;
    float2* nodes;
};

__device__ __forceinline__ bool label_shown(const float4* c, uint32_t l) { return __ldg(&c[l].w) > 0.5f; }
__device__ __forceinline__ bool label_ghosted(const float4* c, uint32_t l) { return l != 0u && __ldg(&c[l].w) > 1.5f; }
__device__ __forceinline__ bool label_solid(const float4* c, uint32_t l, uint32_t mode) {
    if (label_ghosted(c, l)) return false;
    return mode == 1u ? (l == 0u || label_shown(c, l)) : (l != 0u && label_shown(c, l));
}

__device__ __forceinline__ uint8_t label_at(const MaskArgs& A, int x, int y, int z) {
    return __ldg(A.labels + voff(A.v, x, y, z));
}

// Trilinear density at continuous index v (common.glsl:68-78): texel space via
// the normalised coordinate, as the texture unit computes it.
__device__ float density_linear_rn(const MaskArgs& A, float ix, float iy, float iz) {
    float p[3] = {ix, iy, iz};
    int i0[3];
    float fr[3];
    for (int k = 0; k < 3; k++) {
        float tc = __fdiv_rn(__fadd_rn(p[k], 0.5f), A.dims[k]);
        float uu = __fsub_rn(__fmul_rn(tc, A.dims[k]), 0.5f);
        float fl = floorf(uu);
        i0[k] = (int)fl;
        fr[k] = __fsub_rn(uu, fl);
    }
    float r = 0.0f;
    for (int dk = 0; dk < 2; dk++)
        for (int dj = 0; dj < 2; dj++)
            for (int di = 0; di < 2; di++) {
                float wgt = __fmul_rn(__fmul_rn(di ? fr[0] : __fsub_rn(1.0f, fr[0]), dj ? fr[1] : __fsub_rn(1.0f, fr[1])),
                                      dk ? fr[2] : __fsub_rn(1.0f, fr[2]));
                r = __fadd_rn(r, __fmul_rn(dens(A.density, A.v, i0[0] + di, i0[1] + dj, i0[2] + dk), wgt));
            }
    return r;
}

__device__ __forceinline__ float soft_score(bool best, bool second, float m) {
    const float CERTAIN = 4.0f;
    if (best == second) return best ? CERTAIN : -CERTAIN;
    return best ? fminf(m, CERTAIN) : -fminf(m, CERTAIN);
}

// A soft-grid node as the mask pass reads it: the CT density at the node
// (there), then the node's margin byte with which of its two labels are drawn
// solid (bits 8, 9: best, runner-up) and ghosted (bits 10, 11).
enum { NODE_SOLID = 8, NODE_GHOST = 10 };
__device__ __forceinline__ uint32_t node_word(const MaskArgs& A, const uint8_t* t) {
    uint32_t best = t[0], second = t[1], mode = (uint32_t)A.mode;
    return (uint32_t)t[2] | ((uint32_t)label_solid(A.colors, best, mode) << NODE_SOLID) |
           ((uint32_t)label_solid(A.colors, second, mode) << (NODE_SOLID + 1)) |
           ((uint32_t)label_ghosted(A.colors, best) << NODE_GHOST) |
           ((uint32_t)label_ghosted(A.colors, second) << (NODE_GHOST + 1));
}
__device__ __forceinline__ float node_score(uint32_t word, int which) {
    return soft_score((word >> which) & 1u, (word >> (which + 1)) & 1u, (float)(word & 0xffu) * 0.0625f);
}
// The spacing of the voxels in grid units, per grid axis (mask.comp:62-100).
__device__ __forceinline__ void grid_scale(const MaskArgs& A, float can[3], float to_grid[3]) {
    int D[3] = {A.v.nx, A.v.ny, A.v.nz};
    for (int k = 0; k < 3; k++) {
        can[k] = (float)D[A.soft_push[k]];
        to_grid[k] = __fdiv_rn(__fsub_rn((float)A.sdims[k], 1.0f), fmaxf(__fsub_rn(can[k], 1.0f), 1.0f));
    }
}
// The CT density at soft-grid node (n0, n1, n2).
__device__ __forceinline__ float node_density(const MaskArgs& A, const int node[3], const float can[3],
                                              const float to_grid[3]) {
    float vv[3];
    for (int a = 0; a < 3; a++) {
        float c = __fdiv_rn((float)node[a], to_grid[a]);
        vv[A.soft_push[a]] = ((A.soft_push[3] >> a) & 1) != 0 ? __fsub_rn(__fsub_rn(can[a], 1.0f), c) : c;
    }
    return density_linear_rn(A, vv[0], vv[1], vv[2]);
}

// The soft grid prepared for one visibility, in the scratch the host points
// `cls`, `flags` and `nodes` into: per node its class (2 bits per mask: 1 the
// score is +CERTAIN, 2 it is -CERTAIN, 0 between) and, with TABLE, its record.
// A voxel's 27 nodes are shared with its neighbours: evaluated per voxel, the
// densities at them (8 taps and 6 divisions each) were the mask pass.
template <bool TABLE> __global__ void __launch_bounds__(256) k_soft_nodes(const MaskArgs A) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= A.sdims[0] * A.sdims[1] * A.sdims[2]) return;
    const uint32_t word = node_word(A, A.soft + 4 * (long)i);
    uint32_t c = 0;
    for (int k = 0; k < 2; k++) {
        float s = node_score(word, k ? NODE_GHOST : NODE_SOLID);
        c |= (s >= 4.0f ? 1u : s <= -4.0f ? 2u : 0u) << (2 * k);
    }
    A.cls[i] = (uint8_t)c;
    if (TABLE) {
        int node[3] = {i % A.sdims[0], (i / A.sdims[0]) % A.sdims[1], i / (A.sdims[0] * A.sdims[1])};
        float can[3], to_grid[3];
        grid_scale(A, can, to_grid);
        A.nodes[i] = make_float2(node_density(A, node, can, to_grid), __uint_as_float(word));
    }
}
// Per node: whether finer labels replaced it (FLAG_OVER), else whether the 27
// nodes around it all have the same class in both masks, none of them between
// (FLAG_SAME, with the class in bits 0-3). There the weighted mean of the
// scores is exactly +-CERTAIN, whatever the weights (a power of two times
// their sum, divided by their sum), and the masks exactly 0 or 1.
enum { FLAG_SAME = 16, FLAG_OVER = 32 };
__global__ void __launch_bounds__(256) k_soft_flags(const MaskArgs A) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int X = A.sdims[0], Y = A.sdims[1], Z = A.sdims[2];
    if (i >= X * Y * Z) return;
    int x = i % X, y = (i / X) % Y, z = i / (X * Y);
    const uint32_t own = A.cls[i];
    uint32_t differ = 0;
    for (int dz = -1; dz <= 1; dz++)
        for (int dy = -1; dy <= 1; dy++) {
            const uint8_t* row = A.cls + ((long)clampi(z + dz, 0, Z - 1) * Y + clampi(y + dy, 0, Y - 1)) * X;
            for (int dx = -1; dx <= 1; dx++) differ |= row[clampi(x + dx, 0, X - 1)] ^ own;
        }
    const bool same = differ == 0 && (own & 3u) != 0 && (own >> 2) != 0 && X > 1 && Y > 1 && Z > 1;
    A.flags[i] = (uint8_t)(A.soft[4 * (long)i + 3] != 0 ? FLAG_OVER : same ? FLAG_SAME | own : 0);
}

// mask.comp:62-100: joint bilateral upsampling of the soft grid's margins.
// TABLE: the nodes' densities and scores come from k_soft_nodes's records,
// else they are evaluated here (grids whose records do not fit the scratch);
// the arithmetic and its order are the same.
template <bool TABLE>
__device__ void soft_masks(const MaskArgs& A, int px, int py, int pz, const float xg[3], float& mr, float& mg) {
    const float SIGMA_CT = 40.0f / 4095.0f, CERTAIN = 4.0f;
    float can[3], to_grid[3];
    if (!TABLE) grid_scale(A, can, to_grid);
    float here = dens(A.density, A.v, px, py, pz);
    int center[3] = {(int)roundf(xg[0]), (int)roundf(xg[1]), (int)roundf(xg[2])};
    float sx = 0.0f, sy = 0.0f, wsum = 0.0f;
    for (int dz = -1; dz <= 1; dz++)
        for (int dy = -1; dy <= 1; dy++)
#pragma unroll(TABLE ? 3 : 1)
            for (int dx = -1; dx <= 1; dx++) {
                int node[3] = {clampi(center[0] + dx, 0, A.sdims[0] - 1), clampi(center[1] + dy, 0, A.sdims[1] - 1),
                               clampi(center[2] + dz, 0, A.sdims[2] - 1)};
                float d0 = __fsub_rn((float)node[0], xg[0]), d1 = __fsub_rn((float)node[1], xg[1]),
                      d2 = __fsub_rn((float)node[2], xg[2]);
                float dd = __fadd_rn(__fadd_rn(__fmul_rn(d0, d0), __fmul_rn(d1, d1)), __fmul_rn(d2, d2));
                float w_space = expf(__fdiv_rn(-dd, 2.0f * 0.6f * 0.6f));
                const long at = ((long)node[2] * A.sdims[1] + node[1]) * A.sdims[0] + node[0];
                float there;
                uint32_t word;
                if (TABLE) {
                    float2 rec = A.nodes[at];
                    there = rec.x;
                    word = __float_as_uint(rec.y);
                } else {
                    there = node_density(A, node, can, to_grid);
                    word = node_word(A, A.soft + 4 * at);
                }
                float df = __fsub_rn(here, there);
                float w_ct = expf(__fdiv_rn(-__fmul_rn(df, df), __fmul_rn(__fmul_rn(2.0f, SIGMA_CT), SIGMA_CT)));
                float s0 = node_score(word, NODE_SOLID), s1 = node_score(word, NODE_GHOST);
                float w = __fadd_rn(__fmul_rn(w_space, w_ct), __fmul_rn(1e-6f, w_space));
                sx = __fadd_rn(sx, __fmul_rn(w, s0));
                sy = __fadd_rn(sy, __fmul_rn(w, s1));
                wsum = __fadd_rn(wsum, w);
            }
    float a = __fdiv_rn(sx, wsum), b = __fdiv_rn(sy, wsum);
    mr = fminf(fmaxf(__fadd_rn(0.5f, __fdiv_rn(a, 2.0f * CERTAIN)), 0.0f), 1.0f);
    mg = fminf(fmaxf(__fadd_rn(0.5f, __fdiv_rn(b, 2.0f * CERTAIN)), 0.0f), 1.0f);
}

// The first of the four x-consecutive voxels of 4-voxel group `g` of the
// bricked layout (element 4 g): a 4-wide row of a 4^3 sub-brick.
__device__ __forceinline__ void group_coord(const Vol& v, uint32_t g, int& x, int& y, int& z) {
    uint32_t b = g >> 7, w = g & 127u, sub = w >> 4, in = w & 15u;
    uint32_t by = b / (uint32_t)v.bx;
    x = (int)((b - by * v.bx) << 3 | (sub & 1u) << 2);
    uint32_t bz = by / (uint32_t)v.by;
    y = (int)((by - bz * v.by) << 3 | ((sub >> 1) & 1u) << 2 | (in & 3u));
    z = (int)(bz << 3 | (sub >> 2) << 2 | in >> 2);
}

// How the mask pass knows the soft grid: no scratch for it (LEVEL 0: as mask.comp
// has it), the nodes' flags (1), the flags and the nodes' records (2).
//
// mask.comp:107-138 (pass 0): binary or soft masks, and the tint-mode cut margin.
// A thread takes a row of four voxels (one 16-byte store). The soft masks are
// bound by arithmetic (54 expf and 54 divisions per voxel); k_soft_flags
// settles the voxels away from where the drawn labels end, k_soft_nodes the
// node densities of the rest. Measured on the 512 x 512 x 400 head/neck volume
// with its 171 x 171 x 134 grid: 53.2 -> 1.72 ms (and 0.14 for both small kernels).
template <int LEVEL>
__global__ void __launch_bounds__(256) k_mask_binary(const MaskArgs A, uint4* __restrict__ out, uint32_t groups) {
    uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= groups) return;
    int x0, y, z;
    group_coord(A.v, g, x0, y, z);
    uint32_t o[4] = {0u, 0u, 0u, 0u};
    if (x0 < A.v.nx && y < A.v.ny && z < A.v.nz) {
        const uint32_t mode = (uint32_t)A.mode;
        const uint32_t four = __ldg((const uint32_t*)A.labels + g);
        const int D[3] = {A.v.nx, A.v.ny, A.v.nz};
        float xg[3] = {0.0f, 0.0f, 0.0f};
        for (int k = 0; k < 4; k++) {
            const int x = x0 + k;
            if (x >= A.v.nx) break;
            const uint32_t label = (four >> (8 * k)) & 0xffu;
            float mr = label_solid(A.colors, label, mode) ? 1.0f : 0.0f;
            float mg = label_ghosted(A.colors, label) ? 1.0f : 0.0f;
            if ((A.soft_push[3] & 8) != 0) {
                // soft_coord (mask.comp:40-50); along a row only the grid axes that run in x change.
                const int P[3] = {x, y, z};
                for (int a = 0; a < 3; a++) {
                    if (k > 0 && A.soft_push[a] != 0) continue;
                    float can = (float)D[A.soft_push[a]];
                    float val = (float)P[A.soft_push[a]];
                    float s = ((A.soft_push[3] >> a) & 1) != 0 ? __fsub_rn(__fsub_rn(can, 1.0f), val) : val;
                    xg[a] = __fdiv_rn(__fmul_rn(s, __fsub_rn((float)A.sdims[a], 1.0f)), fmaxf(__fsub_rn(can, 1.0f), 1.0f));
                }
                if (label < 250u) {
                    // texelFetch inside the grid by construction
                    const int n0 = clampi((int)roundf(xg[0]), 0, A.sdims[0] - 1);
                    const int n1 = clampi((int)roundf(xg[1]), 0, A.sdims[1] - 1);
                    const int n2 = clampi((int)roundf(xg[2]), 0, A.sdims[2] - 1);
                    const long at = ((long)n2 * A.sdims[1] + n1) * A.sdims[0] + n0;
                    const uint32_t f = LEVEL > 0 ? (uint32_t)A.flags[at] : A.soft[4 * at + 3] != 0 ? FLAG_OVER : 0;
                    if (f & FLAG_SAME) {
                        mr = (f & 3u) == 1u ? 1.0f : 0.0f;
                        mg = (f & 12u) == 4u ? 1.0f : 0.0f;
                    } else if (!(f & FLAG_OVER)) {
                        soft_masks<LEVEL == 2>(A, x, y, z, xg, mr, mg);
                    }
                }
            }
            int m = A.margin;
            if (mode == 1u && m > 0 && label == 0u) {
                for (int a = -m; a <= m && mr > 0.0f; a++)
                    for (int b = -m; b <= m && mr > 0.0f; b++)
                        for (int c = -m; c <= m; c++) {
                            uint32_t l = label_at(A, clampi(x + a, 0, A.v.nx - 1), clampi(y + b, 0, A.v.ny - 1),
                                                  clampi(z + c, 0, A.v.nz - 1));
                            if (l != 0u && (!label_shown(A.colors, l) || label_ghosted(A.colors, l))) {
                                mr = 0.0f;
                                break;
                            }
                        }
            }
            const uint32_t code = mask_encode(mr, A.v.mfmt) | (mask_encode(mg, A.v.mfmt) << 16);
            o[0] = k == 0 ? code : o[0];
            o[1] = k == 1 ? code : o[1];
            o[2] = k == 2 ? code : o[2];
            o[3] = k == 3 ? code : o[3];
        }
    }
    out[g] = make_uint4(o[0], o[1], o[2], o[3]);
}

// The code of 1.0 in a mask format, and whether both channels of a texel are
// exactly 0 or 1.
__device__ __forceinline__ uint32_t mask_one(int mfmt) {
    return mfmt == MF_FP16 ? 0x3c00u : mfmt == MF_BF16 ? 0x3f80u : 0xffffu;
}
__device__ __forceinline__ bool mask_settled(uint32_t m, uint32_t one) {
    const uint32_t r = m & 0xffffu, g = m >> 16;
    return (r == 0u || r == one) && (g == 0u || g == one);
}

// mask.comp:260-278 (passes 1-3): binomial blur of radius R along one axis, a
// row of four voxels per thread. HBM-bound (a read and a write of 4 bytes per
// voxel), once the arithmetic is out of the way: the binomials C(2R, j) and
// their sum 2^(2R) are exact in FP32, so taps that are all 0 or all 1 blur to
// themselves exactly (all but the boundaries), the sum's division is an exact
// scaling, and the index arithmetic is 32-bit. Measured on 512 x 512 x 400 at
// radius 1: 2.1 -> 0.21-0.25 ms per pass (3.4-4.0 TB/s).
template <int R, int AXIS>
__global__ void __launch_bounds__(256) k_mask_blur(const uint4* __restrict__ src, uint4* __restrict__ dst, const Vol v,
                                                   uint32_t groups) {
    const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= groups) return;
    int x0, y, z;
    group_coord(v, g, x0, y, z);
    if (x0 >= v.nx || y >= v.ny || z >= v.nz) {
        dst[g] = make_uint4(0u, 0u, 0u, 0u);
        return;
    }
    // Tap j of voxel k: in y and z the same group of another row; in x voxel
    // x0 + k + j - R of this row, from the groups around it.
    constexpr int N = 2 * R + 1;
    constexpr int TAPS = AXIS == 0 ? 4 + 2 * R : N;
    constexpr int SIDE = (R + 3) / 4;  // groups to each side
    uint32_t t[AXIS == 0 ? 1 : N][4];
    uint32_t row[AXIS == 0 ? 4 * (2 * SIDE + 1) : 1];  // voxels x0 - 4 SIDE ..
    const uint32_t* s32 = (const uint32_t*)src;
    uint32_t first, differ = 0u;
    if (AXIS == 0) {
        const int oyz = offy(v, y) + offz(v, z);
#pragma unroll
        for (int q = -SIDE; q <= SIDE; q++) {
            const int xq = x0 + 4 * q;
            uint4 w;
            if (xq >= 0 && xq + 3 < v.nx) {
                w = __ldg((const uint4*)(s32 + oyz + offx(xq)));
            } else {  // clamped to the edge voxel by voxel
                w.x = __ldg(s32 + oyz + offx(clampi(xq, 0, v.nx - 1)));
                w.y = __ldg(s32 + oyz + offx(clampi(xq + 1, 0, v.nx - 1)));
                w.z = __ldg(s32 + oyz + offx(clampi(xq + 2, 0, v.nx - 1)));
                w.w = __ldg(s32 + oyz + offx(clampi(xq + 3, 0, v.nx - 1)));
            }
            uint32_t* o = row + 4 * (q + SIDE);
            o[0] = w.x; o[1] = w.y; o[2] = w.z; o[3] = w.w;
        }
        first = row[4 * SIDE];
#pragma unroll
        for (int k = 0; k < TAPS; k++) differ |= row[4 * SIDE - R + k] ^ first;
    } else {
#pragma unroll
        for (int j = 0; j < N; j++) {
            const int yj = AXIS == 1 ? clampi(y + j - R, 0, v.ny - 1) : y;
            const int zj = AXIS == 2 ? clampi(z + j - R, 0, v.nz - 1) : z;
            const uint4 w = __ldg((const uint4*)(s32 + offx(x0) + offy(v, yj) + offz(v, zj)));
            t[j][0] = w.x; t[j][1] = w.y; t[j][2] = w.z; t[j][3] = w.w;
        }
        first = t[R][0];
#pragma unroll
        for (int j = 0; j < N; j++)
#pragma unroll
            for (int k = 0; k < 4; k++) differ |= t[j][k] ^ first;
    }
    uint32_t o[4];
    if (differ == 0u && mask_settled(first, mask_one(v.mfmt))) {
        o[0] = o[1] = o[2] = o[3] = first;
    } else {
#pragma unroll
        for (int k = 0; k < 4; k++) {
            float sx = 0.0f, sy = 0.0f, c = 1.0f;
#pragma unroll
            for (int j = 0; j < N; j++) {
                const uint32_t m = AXIS == 0 ? row[4 * SIDE - R + k + j] : t[AXIS == 0 ? 0 : j][k];
                sx = __fadd_rn(sx, __fmul_rn(c, mask_decode(m & 0xffffu, v.mfmt)));
                sy = __fadd_rn(sy, __fmul_rn(c, mask_decode(m >> 16, v.mfmt)));
                c = c * (float)(2 * R - j) / (float)(j + 1);  // exact: folds to C(2R, j + 1)
            }
            constexpr float scale = 1.0f / (float)(1 << (2 * R));
            o[k] = mask_encode(__fmul_rn(sx, scale), v.mfmt) | (mask_encode(__fmul_rn(sy, scale), v.mfmt) << 16);
        }
    }
#pragma unroll
    for (int k = 1; k < 4; k++)
        if (x0 + k >= v.nx) o[k] = 0u;  // the padding of the last brick
    dst[g] = make_uint4(o[0], o[1], o[2], o[3]);
}

// majorant.comp:26-71: the extinction bound of each brick over the brick and
// two voxels of border. A warp takes a brick: its 12 x 12 rows of up to four
// 4-voxel groups, one group per lane and step (8 or 16 bytes of density, 16 of
// mask, neighbouring bricks' overlap from L1). The extremes are taken on the
// stored codes, which are in the order of the values (densities and masks are
// in [0, 1]), and decoded once. One thread per brick read 1 728 voxels in
// turn: 2.48 -> 0.52 ms on 512 x 512 x 400.
template <bool WIDE>
__global__ void __launch_bounds__(256) k_majorant(const void* __restrict__ d, const uint32_t* __restrict__ mask, Vol v,
                                                  int mode, float label_ext, const float* __restrict__ bucket,
                                                  float* __restrict__ out) {
    const int b = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = (int)(threadIdx.x & 31u);
    if (b >= v.bx * v.by * v.bz) return;
    const int bxi = b % v.bx, byi = (b / v.bx) % v.by, bzi = b / (v.bx * v.by);
    const int lo[3] = {max(bxi * 8 - 2, 0), max(byi * 8 - 2, 0), max(bzi * 8 - 2, 0)};
    const int hi[3] = {min(bxi * 8 + 9, v.nx - 1), min(byi * 8 + 9, v.ny - 1), min(bzi * 8 + 9, v.nz - 1)};
    const int g0 = lo[0] >> 2, gn = (hi[0] >> 2) - g0 + 1, rows = hi[1] - lo[1] + 1;
    const int n = gn * rows * (hi[2] - lo[2] + 1);
    uint32_t dmin = 0xffffffffu, dmax = 0u, mmax = 0u;
    for (int i = lane; i < n; i += 32) {
        const int q = i / gn, x = (g0 + i - q * gn) << 2, y = lo[1] + q % rows, z = lo[2] + q / rows;
        const int o = voff(v, x, y, z);  // the group's first element; its four lie in one brick
        uint32_t c[4];
        if (WIDE) {
            const uint4 w = __ldg((const uint4*)((const uint32_t*)d + o));
            c[0] = w.x; c[1] = w.y; c[2] = w.z; c[3] = w.w;
        } else {
            const uint2 w = __ldg((const uint2*)((const uint16_t*)d + o));
            c[0] = w.x & 0xffffu; c[1] = w.x >> 16; c[2] = w.y & 0xffffu; c[3] = w.y >> 16;
        }
        uint32_t m[4] = {0u, 0u, 0u, 0u};
        if (mode != 0) {
            const uint4 w = __ldg((const uint4*)(mask + o));
            m[0] = w.x; m[1] = w.y; m[2] = w.z; m[3] = w.w;
        }
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (x + k >= lo[0] && x + k <= hi[0]) {
                dmin = min(dmin, c[k]);
                dmax = max(dmax, c[k]);
                mmax = max(mmax, max(m[k] & 0xffffu, m[k] >> 16));
            }
    }
    dmin = __reduce_min_sync(0xffffffffu, dmin);
    dmax = __reduce_max_sync(0xffffffffu, dmax);
    mmax = __reduce_max_sync(0xffffffffu, mmax);
    if (lane != 0) return;
    auto value = [&](uint32_t c) {
        return WIDE ? __uint_as_float(c)
                    : v.dfmt == DF_FP16 ? density_decode<DF_FP16>((uint16_t)c)
                                        : v.dfmt == DF_BF16 ? density_decode<DF_BF16>((uint16_t)c) : unorm16(c);
    };
    auto tf_max = [&](float lo_, float hi_) {
        int first = clampi((int)(lo_ * 64.0f), 0, 63), last = clampi((int)(hi_ * 64.0f), 0, 63);
        float m = 0.0f;
        for (int k = first; k <= last; k++) m = gmax(m, bucket[k]);
        return m;
    };
    float bound;
    if (mode == 0) bound = tf_max(value(dmin), value(dmax));
    else if (mmax == 0u) bound = 0.0f;
    else if (mode == 1) bound = tf_max(value(dmin), value(dmax));
    else bound = label_ext;
    out[b] = bound;
}

// flight_majorant (pt.comp:157-163) of every brick, for the tracer's uniforms:
// the brick's bound, or none without empty-space skipping; at least the tissue's
// where labels are drawn alone; at most the largest of the three caps.
__global__ void __launch_bounds__(256) k_flight_majorant(const float* __restrict__ bound, int n, int skip, int labelled,
                                                         float tissue, float label_ext, float* __restrict__ out) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= n) return;
    float m = skip ? bound[b] : 1e30f;
    if (m > 0.0f && labelled) m = gmax(m, tissue);
    out[b] = gmin(m, gmax(MAX_EXTINCTION, gmax(label_ext, tissue)));
}

// Bricked -> x-fastest copy of `elem`-byte elements.
__global__ void k_unbrick(const uint8_t* __restrict__ src, uint8_t* __restrict__ dst, Vol v, int elem) {
    long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    long n = (long)v.nx * v.ny * v.nz;
    if (i >= n) return;
    int x = (int)(i % v.nx), y = (int)((i / v.nx) % v.ny), z = (int)(i / ((long)v.nx * v.ny));
    long o = voff(v, x, y, z);
    for (int k = 0; k < elem; k++) dst[i * elem + k] = src[o * elem + k];
}

// x-fastest -> bricked copy of bytes (labels).
__global__ void k_brick_u8(const uint8_t* __restrict__ src, uint8_t* __restrict__ dst, Vol v) {
    long e = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= vol_elems(v)) return;
    int x, y, z;
    vcoord(v, e, x, y, z);
    dst[e] = (x < v.nx && y < v.ny && z < v.nz) ? src[((long)z * v.ny + y) * v.nx + x] : 0;
}

static unsigned blocks_for(long n, int t) { return (unsigned)((n + t - 1) / t); }

// One word per device, in the library's own image: shared by all renderers and
// engines of the process, and none of them has to outlive another's passes.
__device__ uint32_t g_passes;
cudaError_t passes_on_device(uint32_t** count) { return cudaGetSymbolAddress((void**)count, g_passes); }

cudaError_t launch_density(const int16_t* hu, void* out, const Vol& v, cudaStream_t s) {
    k_density<<<blocks_for(vol_elems(v), 256), 256, 0, s>>>(hu, out, v);
    return cudaGetLastError();
}
cudaError_t launch_normals(const void* d, uint32_t* out, const Vol& v, const m3& w2i, cudaStream_t s) {
    k_normals<<<blocks_for(vol_elems(v), 256), 256, 0, s>>>(d, out, v, w2i);
    return cudaGetLastError();
}
// The three blur passes (x: scratch to out, y: back, z: to out).
template <int R> static void blur_axes(uint4* scratch, uint4* out, const Vol& v, uint32_t groups, cudaStream_t s) {
    const unsigned nb = blocks_for(groups, 256);
    k_mask_blur<R, 0><<<nb, 256, 0, s>>>(scratch, out, v, groups);
    k_mask_blur<R, 1><<<nb, 256, 0, s>>>(out, scratch, v, groups);
    k_mask_blur<R, 2><<<nb, 256, 0, s>>>(scratch, out, v, groups);
}
cudaError_t launch_masks(const MaskLaunch& L, cudaStream_t s, int* launches) {
    MaskArgs A;
    A.v = L.v;
    A.density = L.density;
    A.labels = L.labels;
    A.soft = L.soft;
    for (int k = 0; k < 3; k++) A.sdims[k] = L.soft_dims[k];
    for (int k = 0; k < 4; k++) A.soft_push[k] = L.soft_push[k];
    A.margin = L.margin;
    A.mode = L.mode;
    A.colors = L.colors;
    A.dims[0] = (float)L.v.nx;
    A.dims[1] = (float)L.v.ny;
    A.dims[2] = (float)L.v.nz;
    const uint32_t groups = (uint32_t)(vol_elems(L.v) / 4);
    const unsigned nb = blocks_for(groups, 256);
    uint4* scratch = (uint4*)L.scratch;
    uint4* out = (uint4*)L.out;
    // The prepared soft grid goes into the output volume (written by the first
    // blur, after the binary pass has read it): two bytes per node, and eight
    // more for the records. The grids of a third or half of the voxels' pitch
    // fit whole; one node per voxel leaves the records out.
    const size_t room = (size_t)vol_elems(L.v) * sizeof(uint32_t);
    const size_t nodes = L.soft ? (size_t)L.soft_dims[0] * L.soft_dims[1] * L.soft_dims[2] : 0;
    const size_t bytes = (2 * nodes + 15) / 16 * 16;
    int level = 0;
    if (nodes > 0 && nodes < (1u << 30) && bytes <= room) {
        A.cls = (uint8_t*)L.out;
        A.flags = A.cls + nodes;
        A.nodes = (float2*)(A.cls + bytes);
        level = bytes + 8 * nodes <= room ? 2 : 1;
        if (level == 2) k_soft_nodes<true><<<blocks_for((long)nodes, 256), 256, 0, s>>>(A);
        else k_soft_nodes<false><<<blocks_for((long)nodes, 256), 256, 0, s>>>(A);
        k_soft_flags<<<blocks_for((long)nodes, 256), 256, 0, s>>>(A);
        *launches += 2;
    }
    if (level == 2) k_mask_binary<2><<<nb, 256, 0, s>>>(A, scratch, groups);
    else if (level == 1) k_mask_binary<1><<<nb, 256, 0, s>>>(A, scratch, groups);
    else k_mask_binary<0><<<nb, 256, 0, s>>>(A, scratch, groups);
    switch (L.radius) {
        case 0: blur_axes<0>(scratch, out, L.v, groups, s); break;
        case 1: blur_axes<1>(scratch, out, L.v, groups, s); break;
        case 2: blur_axes<2>(scratch, out, L.v, groups, s); break;
        case 3: blur_axes<3>(scratch, out, L.v, groups, s); break;
        case 4: blur_axes<4>(scratch, out, L.v, groups, s); break;
        case 5: blur_axes<5>(scratch, out, L.v, groups, s); break;
        case 6: blur_axes<6>(scratch, out, L.v, groups, s); break;
        case 7: blur_axes<7>(scratch, out, L.v, groups, s); break;
        case 8: blur_axes<8>(scratch, out, L.v, groups, s); break;
        default: return cudaErrorInvalidValue;  // the host clamps the radius to 0..8
    }
    *launches += 4;
    return cudaGetLastError();
}
cudaError_t launch_majorant(const void* d, const uint32_t* mask, const Vol& v, int mode, float label_ext,
                            const float* bucket, float* out, cudaStream_t s) {
    const unsigned nb = blocks_for((long)v.bx * v.by * v.bz, 8);  // a warp per brick
    if (v.dfmt == DF_FP32) k_majorant<true><<<nb, 256, 0, s>>>(d, mask, v, mode, label_ext, bucket, out);
    else k_majorant<false><<<nb, 256, 0, s>>>(d, mask, v, mode, label_ext, bucket, out);
    return cudaGetLastError();
}
cudaError_t launch_flight_majorant(const float* bound, int n, bool skip, bool labelled, float tissue, float label_ext,
                                   float* out, cudaStream_t s) {
    k_flight_majorant<<<blocks_for(n, 256), 256, 0, s>>>(bound, n, skip, labelled, tissue, label_ext, out);
    return cudaGetLastError();
}
cudaError_t launch_unbrick(const void* src, void* dst, const Vol& v, int elem, cudaStream_t s) {
    long n = (long)v.nx * v.ny * v.nz;
    k_unbrick<<<blocks_for(n, 256), 256, 0, s>>>((const uint8_t*)src, (uint8_t*)dst, v, elem);
    return cudaGetLastError();
}
cudaError_t launch_brick_u8(const uint8_t* src, uint8_t* dst, const Vol& v, cudaStream_t s) {
    k_brick_u8<<<blocks_for(vol_elems(v), 256), 256, 0, s>>>(src, dst, v);
    return cudaGetLastError();
}

}  // namespace vv
