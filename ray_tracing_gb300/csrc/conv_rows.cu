// The denoiser's 3x3 convolution by image rows (k_conv_rows): the same layer as
// k_conv3x3 (denoiser.cu), the same products summed in the same order (dy, dx,
// then 16 input channels a step), so the same bits.
//
// k_conv3x3 issues one tcgen05.mma of N = c_out per tap and 16 channels, and
// each re-reads a 4 KB A tile (128 pixels x 16 channels) from shared memory for
// c_out <= 64 columns of work: 32 of the ~45 clocks an instruction takes at
// c_out = 32 are that read, the tensor pipe is 15-26 % busy. Here M = 128 is 128
// consecutive pixels of ONE image row, and an input row r contributes to three
// output rows: r - 1 with dy = 2, r with dy = 1 and r + 1 with dy = 0. Their
// accumulators are neighbours in TMEM and the three dy slices of a (dx, 16
// channels) weight block are neighbours in shared memory, so one instruction of
// N = 3 c_out reads the A tile once for all three: a third of the instructions,
// at ~56 clocks each for c_out = 32. Going down the image row by row each output
// row still receives dy = 0, 1, 2 in that order.
//
//   * A CTA runs two or four groups, each a producer warp, an issuing warp and
//     epilogue warps over a run of output rows of one 128-pixel column (a run
//     may continue in the next column); weights are shared. One issuing warp
//     alone reaches half the instruction rate.
//   * Input rows arrive by cp.async.bulk, one copy of up to 130 x 16 bytes per
//     8-channel block (contiguous in the blocked layout), into a ring of row
//     stages; the pixels left of 0 and at w are zeroed by the producer's lanes
//     (pixels further right only feed outputs that are not stored), rows outside
//     the image are skipped.
//   * Output rows live in a ring of TMEM slots of c_out columns, zero before their
//     first product (the epilogue clears what it has read), so every instruction
//     accumulates; one that would cross the ring's end is issued in two parts.
//     Within an input row all instructions of a part have one accumulator and
//     shape and so execute in order; the next row's accumulators overlap them at
//     another base, so it waits for the row before (its commit), while the other
//     group's instructions run.
//   * The epilogue is k_conv3x3's (bias, ReLU or mask, BF16 stores of 512
//     contiguous bytes a warp and block, fused 2x2 pooling and nearest
//     upsampling); pooling keeps the even row's outputs in registers, so runs
//     start and end on even rows.
// Every wait is bounded and a failed role stops the others.
//
// The U-Net at 4 x 640x480 (eleven layers, packing, unpacking): 502 us by tiles,
// 337 us here (d1a, 80 -> 32 channels: 97 -> 54 us; e1a 42 -> 25; the 48 -> 48 layer
// with upsampling 52 -> 32 with whole-sector stores). d1a issues 242,000
// instructions (every second row's go in two parts around the slot ring's end), 58
// clocks apiece an SM: the shared-memory reads of their operands (4 KB of pixels and
// up to 3 KB of weights at 128 bytes a clock) and the DRAM stream (62 % of its peak)
// are what is left near a limit, the tensor pipe is at 48 %. The same loop run by
// one lane, its descriptors moved to uniform registers one by one, took 570 us, two
// groups instead of four 414 us.
// conv_rows_fits says which layers take this form; a frame of 1 x 128 x 128 or
// 1 x 160 x 120, too small to fill the SMs with rows, took 106 and 116 us of
// denoising by rows alone, 92 by tiles.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "denoiser.cuh"
#include "per_device.h"
#include "tc_primitives.cuh"

namespace rtgb {
namespace {

constexpr int kCols = 128;                 // output pixels of a row strip (M)
constexpr int kHaloCols = kCols + 2;
constexpr int kPitch = kHaloCols * 16;     // one 8-channel block of a staged row: 2080 bytes
constexpr int kMaxRowStages = 8;
constexpr int kMaxSlots = 8;
constexpr int kMaxGroups = 4;
// Groups of a CTA: a row of products waits for the row before, and the other
// groups' instructions fill that wait; up to 32 output channels four groups have
// the four TMEM slots each needs, beyond that two. Epilogue warps: four a set (a
// quarter of the pixels each), two sets sharing a row's channels beside two groups.
__host__ __device__ constexpr int rows_groups(int chunks) { return chunks > 2 ? 2 : 4; }
__host__ __device__ constexpr int epilogue_sets(int chunks) { return chunks > 2 ? 2 : 1; }
__host__ __device__ constexpr int rows_threads(int chunks) { return 32 * rows_groups(chunks) * (2 + 4 * epilogue_sets(chunks)); }
constexpr int kSpin = 1 << 22;
constexpr int kBiasAt = 1152;              // the bias, after barriers, TMEM address and stop flag
constexpr int kBarBytes = kBiasAt + 256;
constexpr int kSmemMax = 227 * 1024;
constexpr int kSmemMin = 116 * 1024;       // one CTA per SM: each takes all of TMEM

struct RowsArgs {
    const __nv_bfloat16* x;
    int n, h, w, cin, cout;
    int y_channels, y_offset, relu;
    const uint4* weight;   // packed [tap][cin/8][cout][8] BF16
    const float* bias;
    __nv_bfloat16* y;
    __nv_bfloat16* pool;
    const __nv_bfloat16* mask;
    int up;
    int* err;
    int stages, slots;
    int strips, pairs;     // 128-pixel columns of an image, row pairs of a column
    int run;               // row pairs of a group's run
    long long units;       // n * strips * pairs
    int cta_step, group_step;  // runs from a CTA's first to the next one's, from a group to the next
};

struct GroupBars {
    uint64_t full[kMaxRowStages];    // row landed
    uint64_t empty[kMaxRowStages];   // row consumed (commit)
    uint64_t acc_full[kMaxSlots];    // output row complete (commit)
    uint64_t acc_empty[kMaxSlots];   // output row drained (every epilogue warp)
};
static_assert(sizeof(GroupBars) * kMaxGroups + 16 <= kBiasAt, "barrier block");

__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     tc::smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(tc::smem_u32(bar))
                 : "memory");
}

// A place in a ring of barriers and the parity of its current use.
struct Cursor {
    int at = 0;
    uint32_t parity = 0;
    __device__ __forceinline__ void next(int size) {
        if (++at == size) {
            at = 0;
            parity ^= 1u;
        }
    }
};

// A piece of a group's run inside one column: output rows [y0, y1) of strip
// `strip` of image `img`, and the input rows [r0, r1) inside the image.
struct Segment {
    int img, x0, y0, y1, r0, r1;
};

__device__ __forceinline__ bool next_segment(const RowsArgs& a, long long& unit, long long end, Segment& s) {
    if (unit >= end) return false;
    const long long column = unit / a.pairs;
    const int p0 = static_cast<int>(unit - column * a.pairs);
    const long long left = end - unit;
    const int count = left < a.pairs - p0 ? static_cast<int>(left) : a.pairs - p0;
    s.img = static_cast<int>(column / a.strips);
    s.x0 = static_cast<int>(column - static_cast<long long>(s.img) * a.strips) * kCols;
    s.y0 = 2 * p0;
    s.y1 = min(2 * (p0 + count), a.h);
    s.r0 = max(s.y0 - 1, 0);
    s.r1 = min(s.y1 + 1, a.h);
    unit += count;
    return true;
}

__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}

// 2x2 average of one packed channel pair: `top` and `bottom` are this lane's
// outputs in the even and the odd row, the neighbour column comes from the next
// lane; sums in k_conv3x3's order (the two columns of a row, then the rows).
__device__ __forceinline__ uint32_t pool_pair(uint32_t top, uint32_t bottom, bool inside, bool has_bottom, float inv) {
    const __nv_bfloat162 t2 = *reinterpret_cast<const __nv_bfloat162*>(&top);
    const __nv_bfloat162 b2 = *reinterpret_cast<const __nv_bfloat162*>(&bottom);
    float tl = inside ? __low2float(t2) : 0.0f, th = inside ? __high2float(t2) : 0.0f;
    float bl = inside && has_bottom ? __low2float(b2) : 0.0f, bh = inside && has_bottom ? __high2float(b2) : 0.0f;
    tl += __shfl_down_sync(0xffffffffu, tl, 1);
    th += __shfl_down_sync(0xffffffffu, th, 1);
    bl += __shfl_down_sync(0xffffffffu, bl, 1);
    bh += __shfl_down_sync(0xffffffffu, bh, 1);
    return pack2((tl + bl) * inv, (th + bh) * inv);
}

__device__ __forceinline__ void store_twice(__nv_bfloat16* p, const uint4& q) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %1, %2, %3, %4};" ::"l"(p), "r"(q.x), "r"(q.y), "r"(q.z), "r"(q.w)
                 : "memory");
}

__device__ __forceinline__ uint32_t pack_biased(uint32_t lo, uint32_t hi, float2 bias, uint32_t relu) {
    // two FP32 sums plus their bias as one packed add, rounded to BF16; the
    // ReLU after the rounding (it commutes with it)
    unsigned long long v, b;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "r"(lo), "r"(hi));
    asm("mov.b64 %0, {%1, %2};" : "=l"(b) : "f"(bias.x), "f"(bias.y));
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(v), "l"(b));
    float x, y;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v));
    __nv_bfloat162 r = __floats2bfloat162_rn(x, y);
    if (relu) r = __hmax2(r, __floats2bfloat162_rn(0.0f, 0.0f));
    return *reinterpret_cast<const uint32_t*>(&r);
}

// Output channels [16 c0, 16 (c0 + kPer)) (as far as `chunks` goes) of this
// lane's pixel of output row `oy`, accumulated from TMEM column `acc` on.
template <int kPer, bool kPool>
__device__ __forceinline__ void rows_epilogue(const RowsArgs& a, const Segment& s, int oy, int quarter, int lane,
    uint32_t acc, uint64_t* drained, const float* bias, int c0, int chunks, uint32_t (&even)[kPer][8]) {
    const int xx = s.x0 + quarter * 32 + lane;
    const bool inside = xx < a.w;
    const int oh = a.up ? 2 * a.h : a.h, ow = a.up ? 2 * a.w : a.w;
    const int py = a.up ? 2 * oy : oy, px = a.up ? 2 * xx : xx;
    const long long oplane = static_cast<long long>(oh) * ow * 8;
    __nv_bfloat16* out = a.y + ((static_cast<long long>(s.img) * (a.y_channels >> 3) + (a.y_offset >> 3) + 2 * c0) * oh + py) * ow * 8 +
                         static_cast<long long>(px) * 8;
    const uint32_t mine = acc + (static_cast<uint32_t>(quarter * 32) << 16) + static_cast<uint32_t>(c0 * 16);
    uint32_t v[kPer][16];
#pragma unroll
    for (int g = 0; g < kPer; ++g) {
        if (c0 + g < chunks) tc::tmem_ld16(mine + static_cast<uint32_t>(g * 16), v[g]);
    }
    tc::tmem_wait_ld();
#pragma unroll
    for (int g = 0; g < kPer; ++g) {
        if (c0 + g < chunks) tc::tmem_zero16(mine + static_cast<uint32_t>(g * 16));
    }
    tc::tmem_wait_st();
    tc::tc_fence_before();
    __syncwarp();
    if (lane == 0) tc::mbar_arrive(drained);  // this warp's part of the slot is read and zero again
    const bool odd = (oy & 1) != 0, last = oy + 1 == a.h;
    const int ph = (a.h + 1) >> 1, pw = (a.w + 1) >> 1;
    const long long pplane = static_cast<long long>(ph) * pw * 8;
    float inv = 0.0f;
    if constexpr (kPool) {
        const float n0 = inside ? 1.0f : 0.0f;
        const float n1 = n0 + __shfl_down_sync(0xffffffffu, n0, 1);
        const float cnt = odd ? n1 + n1 : n1;
        inv = cnt > 0.0f ? 1.0f / cnt : 0.0f;
    }
#pragma unroll
    for (int g = 0; g < kPer; ++g) {
        if (c0 + g >= chunks) break;
        uint32_t packed[8];
        const float4* b4 = reinterpret_cast<const float4*>(bias + (c0 + g) * 16);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float4 b = b4[k];
            packed[2 * k] = pack_biased(v[g][4 * k], v[g][4 * k + 1], make_float2(b.x, b.y), static_cast<uint32_t>(a.relu));
            packed[2 * k + 1] = pack_biased(v[g][4 * k + 2], v[g][4 * k + 3], make_float2(b.z, b.w), static_cast<uint32_t>(a.relu));
        }
        __nv_bfloat16* blk = out + 2 * g * oplane;
        if (a.mask != nullptr && inside) {
            const __nv_bfloat16* mb = a.mask + (blk - a.y);
            const uint4 m0 = __ldg(reinterpret_cast<const uint4*>(mb));
            const uint4 m1 = __ldg(reinterpret_cast<const uint4*>(mb + oplane));
            const uint32_t m[8] = {m0.x, m0.y, m0.z, m0.w, m1.x, m1.y, m1.z, m1.w};
            const __nv_bfloat162 zero = __floats2bfloat162_rn(0.0f, 0.0f);
#pragma unroll
            for (int k = 0; k < 8; ++k) packed[k] &= __hgt2_mask(*reinterpret_cast<const __nv_bfloat162*>(&m[k]), zero);
        }
        if (inside) {
            const uint4 q0 = make_uint4(packed[0], packed[1], packed[2], packed[3]);
            const uint4 q1 = make_uint4(packed[4], packed[5], packed[6], packed[7]);
            if (a.up) {
                for (int dy = 0; dy < 2; ++dy) {  // both pixels of a row at once: whole 32-byte sectors
                    store_twice(blk + static_cast<long long>(dy) * ow * 8, q0);
                    store_twice(blk + oplane + static_cast<long long>(dy) * ow * 8, q1);
                }
            } else {
                *reinterpret_cast<uint4*>(blk) = q0;
                *reinterpret_cast<uint4*>(blk + oplane) = q1;
            }
        }
        if constexpr (kPool) {
            if (odd || last) {
                uint32_t pooled[8];
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const uint32_t top = odd ? even[g][k] : packed[k];
                    pooled[k] = pool_pair(top, packed[k], inside, odd, inv);
                }
                if (inside && (xx & 1) == 0) {
                    __nv_bfloat16* pblk = a.pool +
                        ((static_cast<long long>(s.img) * (a.cout >> 3) + 2 * (c0 + g)) * ph + (oy >> 1)) * pw * 8 +
                        static_cast<long long>(xx >> 1) * 8;
                    *reinterpret_cast<uint4*>(pblk) = make_uint4(pooled[0], pooled[1], pooled[2], pooled[3]);
                    *reinterpret_cast<uint4*>(pblk + pplane) = make_uint4(pooled[4], pooled[5], pooled[6], pooled[7]);
                }
            }
#pragma unroll
            for (int k = 0; k < 8; ++k) even[g][k] = packed[k];
        }
    }
}

template <int kChunks, bool kPool>
__global__ void __launch_bounds__(rows_threads(kChunks), 1) k_conv_rows(RowsArgs a) {
    constexpr int kCout = 16 * kChunks;
    constexpr int kGroups = rows_groups(kChunks), kTmemCols = 512 / kGroups;
    constexpr int kSets = epilogue_sets(kChunks), kPer = (kChunks + kSets - 1) / kSets;
    extern __shared__ __align__(1024) uint8_t smem[];
    GroupBars* bars = reinterpret_cast<GroupBars*>(smem);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + sizeof(GroupBars) * kMaxGroups);
    volatile int* stop = reinterpret_cast<volatile int*>(smem + sizeof(GroupBars) * kMaxGroups + 8);
    const int cb = a.cin >> 3;
    const int row_bytes = cb * kPitch;
    uint8_t* sw = smem + kBarBytes;                          // [dx][cin/8][dy = 2, 1, 0][cout][8]
    uint8_t* rows = sw + 9 * a.cin * kCout * 2;              // [group][stage][cin/8][130 pixels][8]
    // the warp's index from one lane: what derives from it is then known to be equal across the warp
    const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int g = 0; g < kGroups; ++g) {
            for (int i = 0; i < a.stages; ++i) {
                tc::mbar_init(bars[g].full + i, 1);
                tc::mbar_init(bars[g].empty + i, 1);
            }
            for (int i = 0; i < a.slots; ++i) {
                tc::mbar_init(bars[g].acc_full + i, 1);
                tc::mbar_init(bars[g].acc_empty + i, 4 * kSets);
            }
        }
        *stop = 0;
        tc::mbar_fence_init();
    }
    if (warp == 0) {
        tc::tmem_alloc(tmem_slot, 512);
        tc::tmem_relinquish();
    }
    float* bias = reinterpret_cast<float*>(smem + kBiasAt);
    if (threadIdx.x < kCout) bias[threadIdx.x] = a.bias[threadIdx.x];
    const int wvec = 9 * cb * kCout;  // 16-byte pieces
    for (int i = threadIdx.x; i < wvec; i += blockDim.x) {
        const int o = i % kCout, b = i / kCout % cb, tap = i / kCout / cb;
        const int dy = tap / 3, dx = tap - 3 * dy;
        reinterpret_cast<uint4*>(sw)[((dx * cb + b) * 3 + 2 - dy) * kCout + o] = a.weight[i];
    }
    tc::fence_proxy_async_smem();
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const int role = warp < kGroups ? 0 : (warp < 2 * kGroups ? 1 : 2);
    const int group = role == 0 ? warp : (role == 1 ? warp - kGroups : (warp - 2 * kGroups) / (4 * kSets));
    if (role == 2) {  // accumulators start at zero
        const uint32_t lanes = *tmem_slot + static_cast<uint32_t>(group * kTmemCols) + (static_cast<uint32_t>((warp & 3) * 32) << 16);
        for (int c = 0; c < kTmemCols; c += 16) tc::tmem_zero16(lanes + static_cast<uint32_t>(c));
        tc::tmem_wait_st();
    }
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    GroupBars& bar = bars[group];
    uint8_t* ring = rows + group * a.stages * row_bytes;
    const uint32_t tmem = *tmem_slot + static_cast<uint32_t>(group * kTmemCols);
    // every group's run of row pairs
    const long long first = static_cast<long long>(static_cast<int>(blockIdx.x) * a.cta_step + group * a.group_step) * a.run;
    const long long end = first + a.run < a.units ? first + a.run : a.units;
    auto fail = [&](int code) {
        *stop = 1;
        if (a.err != nullptr) atomicExch(a.err, code);
    };

    if (role == 0) {
        // ---- producer: input rows in order, one bulk copy per channel block
        Cursor st;
        int issued = 0;
        bool ok = true;
        Segment s;
        long long unit = first;
        while (ok && next_segment(a, unit, end, s)) {
            const int xs = s.x0 > 0 ? s.x0 - 1 : 0;
            const int xe = min(s.x0 + kCols + 1, a.w);
            const int at = xs - (s.x0 - 1);        // first staged pixel: 0, or 1 left of the image's edge
            const uint32_t bytes = static_cast<uint32_t>(xe - xs) * 16u;
            const int right = a.w - (s.x0 - 1);    // staged place of pixel w
            const __nv_bfloat16* src = a.x + (static_cast<long long>(s.img) * cb * a.h) * a.w * 8 + static_cast<long long>(xs) * 8;
            for (int r = s.r0; r < s.r1; ++r) {
                bool free_stage = true;
                if (issued >= a.stages) free_stage = tc::mbar_wait_or_abort(bar.empty + st.at, st.parity ^ 1u, kSpin, stop);
                if (!__all_sync(0xffffffffu, free_stage)) {
                    if (lane == 0) fail(21);
                    ok = false;
                    break;
                }
                uint8_t* dst = ring + st.at * row_bytes;
                if (lane < cb) {
                    uint8_t* blk = dst + lane * kPitch;
                    if (at == 1) *reinterpret_cast<uint4*>(blk) = make_uint4(0, 0, 0, 0);
                    if (right < kHaloCols) *reinterpret_cast<uint4*>(blk + right * 16) = make_uint4(0, 0, 0, 0);
                    if (at == 1 || right < kHaloCols) tc::fence_proxy_async_smem();
                }
                __syncwarp();
                if (lane == 0) tc::mbar_arrive_expect_tx(bar.full + st.at, bytes * static_cast<uint32_t>(cb));
                __syncwarp();
                if (lane < cb) {
                    bulk_load(dst + lane * kPitch + at * 16, src + (static_cast<long long>(lane) * a.h + r) * a.w * 8, bytes, bar.full + st.at);
                }
                ++issued;
                st.next(a.stages);
            }
        }
        // every copy has landed before shared memory is released
        for (int j = issued > a.stages ? issued - a.stages : 0; j < issued; ++j) {
            tc::mbar_wait(bar.full + j % a.stages, static_cast<uint32_t>(j / a.stages) & 1u, kSpin);
        }
        __syncwarp();
    } else if (role == 1) {
        // ---- issuer: the whole warp runs it with equal values, lane 0 issues
        {
            const uint32_t leader = lane == 0 ? 1u : 0u;
            const uint64_t b_first = tc::smem_desc(tc::smem_u32(sw), 3 * kCout * 16, 128);
            const int ksteps = cb >> 1;
            Cursor st;           // the input row's stage
            Cursor open;         // the slot of the next output row to begin
            Cursor prev;         // the input row before
            int opened = 0;      // output rows begun, over all segments
            int first_slot = 0;  // the slot of the oldest unfinished output row
            int complete = 0;    // output rows whose last product is issued
            bool ok = true, later = false;
            Segment s;
            long long unit = first;
            while (ok && next_segment(a, unit, end, s)) {
                const int base = opened - s.y0;  // output row o is number base + o
                for (int r = s.r0; r < s.r1; ++r) {
                    const int ob = min(r + 1, s.y1 - 1);
                    // the slots of the rows this one begins (one, two at the image's first row) are drained
                    for (; ok && opened <= base + ob; ++opened) {
                        if (opened >= a.slots) ok = tc::mbar_wait_or_abort(bar.acc_empty + open.at, open.parity ^ 1u, kSpin, stop);
                        open.next(a.slots);
                    }
                    ok = ok && tc::mbar_wait_or_abort(bar.full + st.at, st.parity, kSpin, stop);
                    // the row before has left the accumulators this one shares with it
                    if (later) ok = ok && tc::mbar_wait_or_abort(bar.empty + prev.at, prev.parity, kSpin, stop);
                    if (!ok) {
                        if (lane == 0) fail(22);
                        break;
                    }
                    tc::tc_fence_after();
                    // products of the unfinished output rows up to ob: one part, or two around the slot ring's end
                    const int count = opened - complete;
                    const int head = count < a.slots - first_slot ? count : a.slots - first_slot, tail = count - head;
                    const uint32_t d_head = tmem + static_cast<uint32_t>(first_slot * kCout);
                    const uint32_t i_head = tc::idesc_bf16_f32(128, head * kCout), i_tail = tc::idesc_bf16_f32(128, tail * kCout);
                    // weight rows: dy = 2 for output row r - 1, 1 for r, 0 for r + 1
                    const uint64_t b_head = b_first + static_cast<uint64_t>((complete - base - (r - 1)) * kCout);
                    const uint64_t b_tail = b_head + static_cast<uint64_t>(head * kCout);
                    const uint64_t a_first = tc::smem_desc(tc::smem_u32(ring + st.at * row_bytes), kPitch, 128);
#pragma unroll
                    for (int dx = 0; dx < 3; ++dx) {
                        uint64_t ad = a_first + static_cast<uint64_t>(dx);
                        uint64_t bd = static_cast<uint64_t>(dx * cb * 3 * kCout);
                        for (int k = 0; k < ksteps; ++k) {
                            tc::umma_bf16_if(leader, d_head, ad, b_head + bd, i_head);
                            if (tail > 0) tc::umma_bf16_if(leader, tmem, ad, b_tail + bd, i_tail);
                            ad += static_cast<uint64_t>(2 * kPitch / 16);
                            bd += static_cast<uint64_t>(2 * 3 * kCout);
                        }
                    }
                    tc::umma_commit_if(leader, bar.empty + st.at);
                    prev = st;
                    later = true;
                    st.next(a.stages);
                    // rows that received their last input row: r - 1, and at the image's last row r too
                    const int done = r == a.h - 1 ? opened : base + r;
                    for (; complete < done; ++complete) {
                        tc::umma_commit_if(leader, bar.acc_full + first_slot);
                        if (++first_slot == a.slots) first_slot = 0;
                    }
                }
            }
            // every UMMA this warp issued has completed before TMEM is released
            if (later) tc::mbar_wait(bar.empty + prev.at, prev.parity, kSpin);
        }
        __syncwarp();
    } else {
        // ---- epilogue: output rows in order, this warp the quarter of the pixels and the channels its index selects
        const int quarter = warp & 3;
        const int c0 = ((warp - 2 * kGroups) >> 2) % kSets * kPer;  // this set's first 16 channels
        uint32_t even[kPer][8];
#pragma unroll
        for (int g = 0; g < kPer; ++g) {
#pragma unroll
            for (int k = 0; k < 8; ++k) even[g][k] = 0;
        }
        Cursor slot;
        bool ok = true;
        Segment s;
        long long unit = first;
        while (ok && next_segment(a, unit, end, s)) {
            for (int oy = s.y0; oy < s.y1; ++oy, slot.next(a.slots)) {
                const bool ready = tc::mbar_wait_or_abort(bar.acc_full + slot.at, slot.parity, kSpin, stop);
                if (!__all_sync(0xffffffffu, ready)) {
                    if (lane == 0) fail(24);
                    ok = false;
                    break;
                }
                tc::tc_fence_after();
                rows_epilogue<kPer, kPool>(a, s, oy, quarter, lane, tmem + static_cast<uint32_t>(slot.at * kCout),
                    bar.acc_empty + slot.at, bias, c0, kChunks, even);
            }
        }
    }
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    if (warp == 0) tc::tmem_dealloc(*tmem_slot, 512);
}

int row_stages(int cin, int cout) {
    const int fixed = kBarBytes + 9 * cin * cout * 2;
    const int s = (kSmemMax - fixed) / (rows_groups(cout / 16) * (cin / 8) * kPitch);
    return s < kMaxRowStages ? s : kMaxRowStages;
}

using RowsKernel = void (*)(RowsArgs);
RowsKernel rows_kernel(int cout, bool pool) {
    static const RowsKernel kernels[2][4] = {
        {k_conv_rows<1, false>, k_conv_rows<2, false>, k_conv_rows<3, false>, k_conv_rows<4, false>},
        {k_conv_rows<1, true>, k_conv_rows<2, true>, k_conv_rows<3, true>, k_conv_rows<4, true>}};
    return kernels[pool ? 1 : 0][cout / 16 - 1];
}

}  // namespace

// Row pairs of a group's run when every SM's groups share the image's.
static int rows_run(int n, int h, int w, int cout, int sms) {
    const long long units = static_cast<long long>(n) * ((w + kCols - 1) / kCols) * ((h + 1) / 2);
    const long long groups = static_cast<long long>(sms) * rows_groups(cout / 16);
    return static_cast<int>((units + groups - 1) / groups);
}

// By rows a layer takes a start of 6-8 us and 2-6 us for each row pair of a run
// (the groups' runs proceed side by side), by tiles 5-7 us and 0.004-0.018 us a
// tile of 8 x 16 pixels, both in proportion to the channels; so rows pay from so
// many tiles on per SM and per row pair of a run, and that counts a width that
// fills its strips badly as well as a small image. Measured on 152 SMs, tiles
// against rows: 80 -> 32 channels 10.5 : 11.7 us at 1 x 256 x 256 (3.4 tiles an SM,
// runs of one), 14.8 : 13.1 at 16 x 64 x 128 (6.7, one), 22.7 : 15.9 at
// 1 x 360 x 640 (12.1, two), 97 : 53 at 4 x 480 x 640 (63, eight); 48 -> 48 7.7 : 9.4
// at 1 x 120 x 160 (1.1, one), 13.7 : 14.8 at 2 x 240 x 320 (7.9, three), 17.6 : 15.2
// at 1 x 360 x 640 (12.1, three); 112 -> 48 15.9 : 17.2 at 1 x 240 x 320 (3.9, two),
// 26.0 : 22.8 at 2 x 240 x 320; 48 -> 64 10.2 : 9.9 at 2 x 120 x 160 (2.1, one); 32 -> 32
// in 16 images 256 high equal at a width of 76 (16.8, four), 1.30x by rows at 128, 0.94x
// at 130 (two strips), 1.06x at 160. Layers with `fused` pooling or upsampling gain
// more (rows store both pixels of an upsampled pair at once) and take rows from three
// quarters of that on: the network at 2 x 640 x 480 takes 2 us less with it, from half
// of it on the one at 1 x 640 x 480 4 us more.
bool conv_rows_fits(int n, int h, int w, int cin, int cout, int sms, bool fused) {
    if (row_stages(cin, cout) < 2) return false;  // two staged rows a group do not fit beside the weights
    const long long tiles = static_cast<long long>(n) * ((w + 7) / 8) * ((h + 15) / 16);
    const long long run = rows_run(n, h, w, cout, sms);
    // hundredths of a tile per SM
    const long long least = rows_groups(cout / 16) == 4 ? 130 + 420 * run : (cin <= 48 && cout <= 48 ? 275 : 210) * run;
    return 100 * tiles > sms * (fused ? least * 3 / 4 : least);
}

// Opts every instance into its shared memory (once per device; call outside
// stream capture).
cudaError_t conv_rows_init() {
    static OncePerDevice once;
    return once.run([](int) {
        cudaError_t e = cudaSuccess;
        for (int k = 0; k < 8 && e == cudaSuccess; ++k) {
            e = cudaFuncSetAttribute(rows_kernel(16 * (k / 2 + 1), k % 2 != 0), cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax);
        }
        return e;
    });
}

cudaError_t launch_conv_rows(const void* x, int n, int h, int w, int cin, const void* weight, const float* bias, int cout,
    int relu, void* y, int y_channels, int y_offset, int* err, int sms, cudaStream_t stream, void* pool, int up,
    const void* mask) {
    // a row's bulk copies start on 16-byte boundaries (k_conv3x3's tensor map refuses such an input itself)
    if ((reinterpret_cast<uintptr_t>(x) & 15u) != 0) return cudaErrorInvalidValue;
    const cudaError_t attr = conv_rows_init();
    if (attr != cudaSuccess) return attr;
    RowsArgs a{};
    a.x = static_cast<const __nv_bfloat16*>(x);
    a.n = n;
    a.h = h;
    a.w = w;
    a.cin = cin;
    a.cout = cout;
    a.y_channels = y_channels;
    a.y_offset = y_offset;
    a.relu = relu;
    a.weight = static_cast<const uint4*>(weight);
    a.bias = bias;
    a.y = static_cast<__nv_bfloat16*>(y);
    a.pool = static_cast<__nv_bfloat16*>(pool);
    a.mask = static_cast<const __nv_bfloat16*>(mask);
    a.up = up;
    a.err = err;
    a.stages = row_stages(cin, cout);
    const int cta_groups = rows_groups(cout / 16), columns = 512 / cta_groups;
    a.slots = columns / cout < kMaxSlots ? columns / cout : kMaxSlots;
    a.strips = (w + kCols - 1) / kCols;
    a.pairs = (h + 1) / 2;
    a.units = static_cast<long long>(n) * a.strips * a.pairs;
    a.run = rows_run(n, h, w, cout, sms);
    // Runs that leave every SM a group free go to all SMs in turn, a group of each
    // (640 x 360 pixels 159 -> 154 us of denoising); else neighbouring runs fill a CTA's
    // groups, which is 1 % faster than runs in turn (1920 x 1080: 504 against 508 us).
    const long long runs = (a.units + a.run - 1) / a.run;
    const bool in_turn = runs <= static_cast<long long>(cta_groups - 1) * sms;
    const long long ctas = in_turn ? (runs < sms ? runs : sms) : (runs + cta_groups - 1) / cta_groups;
    const int grid = static_cast<int>(ctas);
    a.cta_step = in_turn ? 1 : cta_groups;
    a.group_step = in_turn ? grid : 1;
    int smem = kBarBytes + 9 * cin * cout * 2 + cta_groups * a.stages * (cin / 8) * kPitch;
    smem = smem > kSmemMin ? smem : kSmemMin;
    rows_kernel(cout, pool != nullptr)<<<grid, rows_threads(cout / 16), smem, stream>>>(a);
    return cudaGetLastError();
}

}  // namespace rtgb
