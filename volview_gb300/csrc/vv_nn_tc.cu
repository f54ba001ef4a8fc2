// vv_nn_tc.cu — the learned denoiser's 3x3 convolution on the fifth-generation
// tensor cores: tcgen05.mma (kind::f16, FP16 operands from shared memory, FP32
// accumulators in tensor memory) fed by TMA (cp.async.bulk.tensor).
//
// Implicit GEMM over 128-pixel segments of image rows (widths that are
// multiples of 128): M = the segment's 128 output pixels, N = the output
// channels padded to a multiple of 16, K = 9 taps x the input channels.
// Operands are K-major in the canonical no-swizzle layout: 8-row x 16-byte
// core matrices, the 8-row groups of one 16-byte K slice 128 bytes apart (the
// stride byte offset), consecutive K slices LBO bytes apart.
//
// A CTA keeps all nine taps' weights of its output channels in shared memory
// and walks down a run of rows of one column of segments (the same 128 pixels
// of consecutive rows). Its input rows, each with its one-pixel halo (130
// pixels), sit in a ring of row slots: a segment uses three (rows y-1, y, y+1)
// and the others take the rows ahead, so every input row is copied once per
// run. TMA copies a row as one box of its 16-byte channel slices x 130 pixels,
// zero-filled outside the image (same padding); each slice is one K slice of
// the layout above. Tap (dy, dx)'s A operand is row y+dy-1's slices starting
// dx pixels in: the descriptor's start address moves by 16 bytes per pixel.
// Roles:
//   warp 4 (its elected lane): waits for a segment's last row, issues its
//     9 x cin / 16 MMAs into one of two TMEM accumulators, commits them to an
//     mbarrier, and copies a row ahead into the slot the previous segment has
//     finished with;
//   warps 0-3: read the finished accumulator (warp w owns TMEM lanes
//     32w..32w+31, one output pixel per lane), release it, add the bias,
//     apply the ReLU and store FP16.
// So a segment's copies, the next segment's MMAs and the previous segment's
// epilogue overlap. Every wait on an mbarrier is bounded: past the limit the
// thread records the failure in a device status word (vv_nn_tc_status) and
// goes on, and the CTA still frees its tensor memory.
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>
#include <stdint.h>

#include <algorithm>

#include "../../include/volpt_nn.h"

namespace vv {
namespace nn {

__device__ int g_tc_status;  // 0, or 1 after a bounded wait gave up

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Shared-memory matrix descriptor (tcgen05): start address, leading (K) and
// stride (M/N) byte offsets, each >> 4; bits 46-48 = 0b001; base offset 0,
// relative leading offset, no swizzle. The low word holds the address and the
// leading offset, the high word the stride (128 bytes here) and the constant.
__device__ __forceinline__ uint32_t desc_lo(uint32_t addr, uint32_t lbo) {
    return ((addr & 0x3FFFFu) >> 4) | ((lbo >> 4) << 16);
}
constexpr uint32_t DESC_HI = (128u >> 4) | (1u << 14);
// D (+)= A B on one 128 x N x 16 step, issued by the warp's elected lane; the
// first step of a segment overwrites.
__device__ __forceinline__ void mma(uint32_t acc, uint32_t da, uint32_t db, uint32_t idesc, int accumulate,
                                    uint32_t elected) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t.reg .b64 a, b;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %6, 0;\n\t"
        "mov.b64 a, {%1, %5};\n\tmov.b64 b, {%2, %5};\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, p;\n\t}\n" ::"r"(acc),
        "r"(da), "r"(db), "r"(idesc), "r"(accumulate), "r"(DESC_HI), "r"(elected));
}
__device__ __forceinline__ uint32_t elect_one() {
    uint32_t one;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}\n" : "=r"(one));
    return one;
}
// Instruction descriptor, kind::f16: FP32 accumulator (bits 4-5 = 1), FP16 A
// and B (bits 7-9, 10-12 = 0), both K-major (bits 15, 16 = 0), N >> 3 at bits
// 17-22, M >> 4 at bits 24-28.
__host__ __device__ constexpr uint32_t instr_desc(int m, int n) {
    return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0));
}

// Waits until the mbarrier's phase of parity `parity` has completed; false
// when the bounded wait gave up (the status word is set).
__device__ __forceinline__ bool bar_wait(uint32_t bar, uint32_t parity) {
    for (int it = 0; it < (1 << 22); it++) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return true;
    }
    atomicExch(&g_tc_status, 1);
    return false;
}

constexpr int TC_M = 128;                     // output pixels per segment (TMEM lanes)
constexpr int HALO = TC_M + 2;                // input pixels per row slice
constexpr int SLICE = HALO * 16;              // bytes of one 8-channel slice of a row: the A operand's LBO
constexpr int EPI_THREADS = 128;              // warps 0-3
constexpr int TC_THREADS = EPI_THREADS + 32;  // + warp 4, the issuing warp
constexpr int RING_MAX = 8;                   // row slots: a segment reads three, the others load ahead

__host__ __device__ constexpr uint32_t tmem_cols(int np) {
    return 2 * np <= 32 ? 32 : 2 * np <= 64 ? 64 : 2 * np <= 128 ? 128 : 2 * np <= 256 ? 256 : 512;
}
// A row slot's bytes, a multiple of the 128 a TMA destination needs.
__host__ __device__ constexpr uint32_t slot_bytes(int cin) { return ((uint32_t)(cin / 8) * SLICE + 127u) & ~127u; }
// Weights, a segment's output, the ring of row slots, and slack to align to 1024 bytes.
static size_t tc_smem(int np, int cin, int ring) {
    return 9 * (size_t)np * 2 * cin + (size_t)TC_M * 2 * np + (size_t)ring * slot_bytes(cin) + 1024;
}

// What bounded it and no longer does (1024^2, 32 -> 32 channels, 65 -> 46 us;
// 16 -> 32 56 -> 39; 512^2 112 -> 48 76 -> 52; the same values to the bit):
// - one row ahead only, so a CTA's period per segment was a row copy's latency
//   (2 us): the ring holds as many rows as fit (loads_ahead);
// - one divergent lane's issue, 107 cycles per MMA: the whole warp walks the
//   segments, so that addresses live in uniform registers (1024^2 80 -> 32
//   with one CTA per SM 137 -> 86-92 us);
// - 4-7 us of staging weights by divisions and half sectors before the first
//   row was asked for: the rows are asked for first, the weights come in whole
//   sectors;
// - stores of 16-byte pieces, channels apart: a warp's pixels leave as one
//   bulk copy.
// What bounds it now: the MMAs' A operand, 4 KB of shared memory per 128 x N x
// 16 MMA (32 cycles whatever N is), and at 1024^2 with few channels the
// epilogue's chain per segment.
template <int NP>
__global__ void __launch_bounds__(TC_THREADS, 1) k_conv3x3_tc(const __grid_constant__ CUtensorMap rows, int n, int h,
                                                           int w, int cin, const __half* __restrict__ wt,
                                                           const float* __restrict__ bias, int cout, int relu,
                                                           __half* __restrict__ y, int run_rows, int ring) {
    constexpr uint32_t COLS = tmem_cols(NP);
    constexpr uint32_t IDESC = instr_desc(TC_M, NP);
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ __align__(8) uint64_t bars[RING_MAX + 4];  // full[ring] (TMA), then mma[2] (tcgen05.commit), free[2]
    __shared__ __align__(16) float bias_s[NP];
    __shared__ uint32_t tmem_slot;
    // The warp's number by a shuffle: the compiler then knows it uniform, and
    // keeps the issuing warp's addresses in uniform registers.
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int chunks = cin >> 3;
    const int per_row = w / TC_M;
    // This CTA's run: column (image, segment) blockIdx.x % columns, rows
    // [y0, y1) of it.
    const int columns = n * per_row;
    const int column = (int)(blockIdx.x % columns), run = (int)(blockIdx.x / columns);
    const int img = column / per_row, x0 = (column - img * per_row) * TC_M;
    const int y0 = run * run_rows, y1 = min(h, y0 + run_rows);
    const int ntiles = y1 > y0 ? y1 - y0 : 0;
    // Its output channels: all of them, or the group blockIdx.y's.
    const int co0 = blockIdx.y * NP, cog = min(NP, cout - co0);
    wt += (long)co0 * 9 * cin;
    const uint32_t w_tap = NP * 2 * cin;  // one tap's weights
    const uint32_t seg = slot_bytes(cin);
    const uint32_t hbase = (smem_u32(smem) + 1023u) & ~1023u;  // the ring of row slots
    const uint32_t wbase = hbase + ring * seg;
    const uint32_t obase = wbase + 9 * w_tap;  // a segment's output, 32 pixels per warp
    const uint32_t full0 = smem_u32(&bars[0]), mma0 = smem_u32(&bars[RING_MAX]), free0 = smem_u32(&bars[RING_MAX + 2]);

    // Relative row q of the run is image row y0 - 1 + q, in slot q % ring; its
    // copy is that slot's (q / ring)-th: one box of the row's 16-byte channel
    // slices, each of 130 pixels.
    const uint32_t bytes = chunks * SLICE;
    auto load_row = [&](int q, int slot) {
        const uint32_t bar = full0 + 8 * slot;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
        asm volatile(
            "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
            " [%0], [%1, {%2, %3, %4, %5, %6}], [%7];" ::"r"(hbase + slot * seg),
            "l"((uint64_t)&rows), "r"(0), "r"(x0 - 1), "r"(0), "r"(y0 - 1 + q), "r"(img), "r"(bar)
            : "memory");
    };
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                     "r"(COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == EPI_THREADS) {
        for (int k = 0; k < ring; k++) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(full0 + 8 * k));
        for (int k = 0; k < 2; k++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mma0 + 8 * k));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(free0 + 8 * k), "r"(EPI_THREADS));
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        if (ntiles > 0)
            for (int q = 0; q < min(ring, ntiles + 2); q++) load_row(q, q);
    }
    __syncwarp();
    // Every tap's weights, rows padded to NP with zeros. Sixteen lanes copy
    // two 16-byte slices of eight rows: whole 32-byte sectors of global memory,
    // 128 consecutive bytes of shared memory per slice.
    {
        const int half = tid >> 4, r8 = tid & 7, c1 = (tid >> 3) & 1;
        for (int u = half; u < 9 * (NP / 8); u += TC_THREADS / 16) {
            const int tap = u % 9, r = (u / 9) * 8 + r8;
            const bool ok = r < cog;
            const __half* src = ok ? wt + ((long)r * 9 + tap) * cin + c1 * 8 : wt;
            uint32_t dst = wbase + tap * w_tap + c1 * (NP * 16) + r * 16;
            for (int c = 0; c < chunks; c += 2) {
                cp_async16(dst, src, ok);
                dst += 2 * NP * 16;
                if (ok) src += 16;
            }
        }
        for (int c = tid; c < NP; c += TC_THREADS) bias_s[c] = bias && c < cog ? bias[co0 + c] : 0.0f;
        asm volatile("cp.async.commit_group;");
        asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = tmem_slot;

    if (warp == 4) {
        // The whole warp walks the segments (its addresses stay uniform), the
        // elected lane issues.
        const uint32_t elected = elect_one();
        if (ntiles > 0) {
            bar_wait(full0, 0);  // rows y-1 and y of the first segment
            bar_wait(full0 + 8, 0);
            int first = 0, third = 2, phase = 0;  // slots of rows i and i + 2, the latter's copy
            for (int i = 0; i < ntiles; i++) {
                const int b = i & 1;
                bar_wait(full0 + 8 * third, phase);
                if (i >= 2) bar_wait(free0 + 8 * b, ((i >> 1) - 1) & 1);  // accumulator b read out
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t acc = tmem + b * NP;
                // The descriptors' low words: the operands' addresses move by
                // constants, so one thread keeps the tensor pipe fed.
                const uint32_t tap_step = (cin / 16) * 2 * SLICE / 16;
                uint32_t db = desc_lo(wbase, NP * 16);
                int slot = first;
                for (int dy = 0; dy < 3; dy++) {
                    uint32_t da = desc_lo(hbase + slot * seg, SLICE);
                    for (int dx = 0; dx < 3; dx++) {
#pragma unroll 1
                        for (int k = 0; k < cin / 16; k++) {
                            mma(acc, da, db, IDESC, dy + dx + k, elected);
                            da += 2 * SLICE / 16;
                            db += 2 * NP;
                        }
                        da += 1 - tap_step;  // one pixel on
                    }
                    slot = slot + 1 == ring ? 0 : slot + 1;
                }
                if (elected) asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                                 mma0 + 8 * b)
                             : "memory");
                // Row i - 1 was last read by the previous segment's MMAs: its
                // slot takes row i - 1 + ring. Three slots are all this
                // segment's, whose own MMAs free the first.
                const int last = i - (ring > 3);
                if (last >= 0 && last + ring < ntiles + 2) {
                    bar_wait(mma0 + 8 * (last & 1), (last >> 1) & 1);
                    if (elected) load_row(last + ring, last == i ? first : first == 0 ? ring - 1 : first - 1);
                }
                first = first + 1 == ring ? 0 : first + 1;
                if (++third == ring) {
                    third = 0;
                    phase ^= 1;
                }
            }
        }
        __syncwarp();
    } else {
        // Epilogue: warps 0-3, one output pixel per thread; a warp's 32 pixels
        // are consecutive in memory and leave as one bulk copy. With groups of
        // channels they are not: each pixel's go out by themselves, in whole
        // sectors.
        const uint32_t out = obase + warp * 64 * cout;
        const bool whole = cog == cout;
        for (int i = 0; i < ntiles; i++) {
            const int b = i & 1;
            const bool ok = bar_wait(mma0 + 8 * b, (i >> 1) & 1);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            uint32_t r[NP];
            const uint32_t row_addr = tmem + b * NP + ((uint32_t)(warp * 32) << 16);
#pragma unroll
            for (int c0 = 0; c0 < NP; c0 += 16) {
                uint32_t* q = r + c0;
                asm volatile(
                    "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, "
                    "[%16];"
                    : "=r"(q[0]), "=r"(q[1]), "=r"(q[2]), "=r"(q[3]), "=r"(q[4]), "=r"(q[5]), "=r"(q[6]), "=r"(q[7]),
                      "=r"(q[8]), "=r"(q[9]), "=r"(q[10]), "=r"(q[11]), "=r"(q[12]), "=r"(q[13]), "=r"(q[14]),
                      "=r"(q[15])
                    : "r"(row_addr + c0));
            }
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            // The values are used only after the wait.
#pragma unroll
            for (int c = 0; c < NP; c++) asm volatile("" : "+r"(r[c]));
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(free0 + 8 * b) : "memory");
            // The warp's previous copy has read its pixels.
            if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
            __syncwarp();
#pragma unroll
            for (int c0 = 0; c0 < NP; c0 += 8) {
                if (c0 >= cog) continue;
                uint32_t packed[4];
#pragma unroll
                for (int j = 0; j < 8; j += 4) {
                    const float4 add = *(const float4*)(bias_s + c0 + j);
                    float v[4] = {__uint_as_float(r[c0 + j]), __uint_as_float(r[c0 + j + 1]),
                                  __uint_as_float(r[c0 + j + 2]), __uint_as_float(r[c0 + j + 3])};
                    if (bias) {
                        v[0] += add.x;
                        v[1] += add.y;
                        v[2] += add.z;
                        v[3] += add.w;
                    }
                    if (relu)
                        for (int k = 0; k < 4; k++) v[k] = fmaxf(v[k], 0.0f);
                    for (int k = 0; k < 2; k++)
                        packed[j / 2 + k] = (uint32_t)__half_as_ushort(__float2half_rn(v[2 * k])) |
                                            ((uint32_t)__half_as_ushort(__float2half_rn(v[2 * k + 1])) << 16);
                }
                if (!whole) {
                    if (ok)
                        *(uint4*)(y + (((long)img * h + y0 + i) * w + x0 + tid) * cout + co0 + c0) =
                            make_uint4(packed[0], packed[1], packed[2], packed[3]);
                    continue;
                }
                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(out + (lane * cout + c0) * 2),
                             "r"(packed[0]), "r"(packed[1]), "r"(packed[2]), "r"(packed[3])
                             : "memory");
            }
            if (!whole) continue;
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0 && ok) {
                const long p = ((long)img * h + y0 + i) * w + x0 + warp * 32;
                asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(
                                 (uint64_t)__cvta_generic_to_global(y + p * cout)),
                             "r"(out), "r"(64 * cout)
                             : "memory");
                asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            }
        }
        if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
        __syncwarp();
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(COLS));
}

// The input tensor (n, h, w, cin) FP16 as a 5-D TMA map, innermost first: the
// channels of a slice, pixels, slices, rows, images; a box is one row's slices
// of 130 pixels.
static bool encode_rows_map(CUtensorMap* map, const void* x, int n, int h, int w, int cin) {
    static PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
    if (!encode) {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess || !fn)
            return false;
        encode = (PFN_cuTensorMapEncodeTiled_v12000)fn;
    }
    const cuuint64_t dims[5] = {8, (cuuint64_t)w, (cuuint64_t)(cin / 8), (cuuint64_t)h, (cuuint64_t)n};
    const cuuint64_t strides[4] = {(cuuint64_t)cin * 2, 16, (cuuint64_t)w * cin * 2, (cuuint64_t)h * w * cin * 2};
    const cuuint32_t box[5] = {8, HALO, (cuuint32_t)(cin / 8), 1, 1};
    const cuuint32_t elem[5] = {1, 1, 1, 1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 5, const_cast<void*>(x), dims, strides, box, elem,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The shared memory a block may ask for, beside its static variables.
constexpr int TC_SMEM_MAX = 226 * 1024;

// Resident CTAs per SM for `smem` bytes of dynamic shared memory: by shared
// memory (with 1 KB per CTA the system reserves and the static barriers), by
// threads, and by TMEM (at most 512 columns per SM between them, so that no
// allocation waits).
static int resident_ctas(size_t smem, int np, int sm_smem) {
    int per_sm = sm_smem / (int)(smem + 2048);
    per_sm = per_sm < 2048 / TC_THREADS ? per_sm : 2048 / TC_THREADS;
    per_sm = per_sm < (int)(512 / tmem_cols(np)) ? per_sm : (int)(512 / tmem_cols(np));
    return per_sm < 1 ? 1 : per_sm;
}

// CTAs per SM, at most four, then the row slots that leave room for them.
// 1024^2, 16 -> 32 / 32 -> 32 / 32 -> 8 channels: one CTA per SM 61.7 / 65.8 /
// 59.7 us, four 39.2 / 47.5 / 35.0. An earlier form of the kernel: six CTAs
// against four 43.5 and 39.5 us (16 -> 32), four, six and eight slots 59.7,
// 51.4 and 51.4 us (32 -> 32).
static void loads_ahead(int np, int cin, int sm_smem, int fewest, int* ring, int* per_sm) {
    *per_sm = std::min(4, resident_ctas(tc_smem(np, cin, fewest), np, sm_smem));
    *ring = fewest;
    while (*ring < RING_MAX && tc_smem(np, cin, *ring + 1) <= TC_SMEM_MAX &&
           resident_ctas(tc_smem(np, cin, *ring + 1), np, sm_smem) >= *per_sm)
        ++*ring;
}

template <int NP>
static cudaError_t launch_tc(const CUtensorMap& map, int n, int h, int w, int cin, const __half* wt, const float* bias,
                             int cout, int relu, __half* y, cudaStream_t s, int groups, int fewest) {
    int dev = 0, sms = 0, sm_smem = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sm_smem, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
    if (e != cudaSuccess) return e;
    static bool configured = false;
    if (!configured) {
        e = cudaFuncSetAttribute(k_conv3x3_tc<NP>, cudaFuncAttributeMaxDynamicSharedMemorySize, TC_SMEM_MAX);
        if (e != cudaSuccess) return e;
        configured = true;
    }
    int ring = 0, per_sm = 0;
    loads_ahead(NP, cin, sm_smem, fewest, &ring, &per_sm);
    const size_t smem = tc_smem(NP, cin, ring);
    // Runs of rows: every resident CTA takes one, the runs of a column of
    // segments as long as the CTAs per column allow.
    const long columns = (long)n * (w / TC_M);
    const long slots = (long)sms * per_sm;
    const long per_column = std::max(1L, slots / (columns * groups));
    const int run_rows = (int)((h + per_column - 1) / per_column);
    const long grid = columns * ((h + run_rows - 1) / run_rows);
    k_conv3x3_tc<NP><<<dim3((unsigned)grid, groups), TC_THREADS, smem, s>>>(map, n, h, w, cin, wt, bias, cout, relu, y, run_rows,
                                                              ring);
    return cudaGetLastError();
}

// The tensor-core convolution when the shape suits it (widths that are
// multiples of 128, and the weights, a segment's output and the rows within
// 226 KB of shared memory); returns false to leave the shape to the mma.sync
// convolution. Up to 96 output channels whose weights fit beside four rows run
// as one group. With `grouped`, the others are split into the fewest groups
// that fit beside four rows, or three (each group reads the input again):
// against mma.sync 256^2 144 -> 64 channels 83 -> 39 us (two groups), 128^2
// 176 -> 80 41 -> 31 (five), four images of 256^2 64 -> 144 230 -> 78 (two),
// of 128^2 80 -> 176 94 -> 35 (two), one of 8 x 128 144 -> 64 18.7 -> 13.0.
// Six image sizes from 8 x 128 to 256^2, 16 to 368 -> 8 to 176 channels, up to
// eleven groups: no shape was slower than on mma.sync.
// *err receives the launch's error.
bool conv3x3_tc(const __half* x, int n, int h, int w, int cin, const __half* wt, const float* bias, int cout,
                int relu, __half* y, cudaStream_t s, bool grouped, cudaError_t* err) {
    if (w % TC_M) return false;
    if (((uintptr_t)x | (uintptr_t)wt | (uintptr_t)y) % 16) return false;
    int np = (cout + 15) / 16 * 16, groups = 1, fewest = 4;
    if (np > 96 || tc_smem(np, cin, 4) > TC_SMEM_MAX) {
        if (!grouped) return false;
        const int wide = np;
        for (groups = 2;; groups++) {
            np = ((wide + groups - 1) / groups + 15) / 16 * 16;
            fewest = tc_smem(np, cin, 4) <= TC_SMEM_MAX ? 4 : 3;
            if (np <= 96 && tc_smem(np, cin, fewest) <= TC_SMEM_MAX) break;
            if (np == 16) return false;
        }
        groups = (wide + np - 1) / np;
    }
    CUtensorMap map;
    if (!encode_rows_map(&map, x, n, h, w, cin)) return false;
    switch (np) {
        case 16: *err = launch_tc<16>(map, n, h, w, cin, wt, bias, cout, relu, y, s, groups, fewest); break;
        case 32: *err = launch_tc<32>(map, n, h, w, cin, wt, bias, cout, relu, y, s, groups, fewest); break;
        case 48: *err = launch_tc<48>(map, n, h, w, cin, wt, bias, cout, relu, y, s, groups, fewest); break;
        case 64: *err = launch_tc<64>(map, n, h, w, cin, wt, bias, cout, relu, y, s, groups, fewest); break;
        case 80: *err = launch_tc<80>(map, n, h, w, cin, wt, bias, cout, relu, y, s, groups, fewest); break;
        case 96: *err = launch_tc<96>(map, n, h, w, cin, wt, bias, cout, relu, y, s, groups, fewest); break;
        default: return false;
    }
    return true;
}

}  // namespace nn
}  // namespace vv

using namespace vv::nn;

extern "C" vv_status vv_nn_conv3x3_tc(const void* x, int n, int h, int w, int cin, const void* weights,
                                      const float* bias, int cout, int relu, void* y, void* stream) {
    if (!x || !weights || !y || n <= 0 || h <= 0 || w <= 0 || w % 16 || cin <= 0 || cin % 16 || cout <= 0 ||
        cout % 8 || cout > 176)
        return VV_ERR_ARG;
    cudaError_t e = cudaSuccess;
    if (!conv3x3_tc((const __half*)x, n, h, w, cin, (const __half*)weights, bias, cout, relu, (__half*)y,
                    (cudaStream_t)stream, false, &e))
        return VV_ERR_ARG;
    return e == cudaSuccess ? VV_OK : VV_ERR_CUDA;
}

extern "C" vv_status vv_nn_tc_status(int* failed, int clear) {
    if (!failed) return VV_ERR_ARG;
    if (cudaMemcpyFromSymbol(failed, g_tc_status, sizeof(int)) != cudaSuccess) return VV_ERR_CUDA;
    if (clear) {
        int zero = 0;
        if (cudaMemcpyToSymbol(g_tc_status, &zero, sizeof(int)) != cudaSuccess) return VV_ERR_CUDA;
    }
    return VV_OK;
}
