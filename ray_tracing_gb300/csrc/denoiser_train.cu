// Training kernels of the denoiser's 3x3 convolution on the sm_103a tensor
// cores (the backward pass of k_conv3x3; the input gradient is k_conv3x3 itself
// with flipped, transposed weights).
//
// k_conv3x3_wgrad: dW[o][i][dy][dx] = sum over pixels p of
// dY[p][o] * X[p + (dy - 1, dx - 1)][i], an implicit GEMM with the pixels as the
// reduction dimension:
//   * a CTA owns every 8 x 16-pixel tile j with j % gridDim.x == blockIdx.x (and
//     the tap rows dy of blockIdx.y's group). Per 8-channel block of X three
//     TMA boxes of 8 x 18 pixels arrive, one per horizontal tap dx, and per
//     block of dY one of 8 x 16, through up to kMaxStages stages;
//   * the rows of the GEMM's M = 128 are (dx, input channel): the three shifted
//     copies lie one box apart like the channel blocks, so one tcgen05.mma
//     covers up to 16 blocks of them. An instruction costs about the same
//     whatever it holds (a fresh 4 KB A tile, ~45 clocks with several issuing
//     threads), and 32 input channels alone fill a quarter of it: three taps an
//     instruction instead of one are a third of the instructions for up to 40
//     channels, two thirds up to 80. N = c_out, K = 16 pixels (two tile rows);
//   * both operands are MN-major straight from the blocked layout: a core matrix
//     is 8 pixels x 8 channels = 128 contiguous bytes; the next 8 pixels along K
//     are one row, 128 bytes, on (the descriptor's leading byte offset) and the
//     next 8 channels along M or N one box on (its stride byte offset) -- for
//     MN-major no-swizzle operands, as for K-major ones, the leading offset
//     steps along K (checked against all four assignments on this GPU; only
//     this one is exact). Rows past the last block read whatever lies there and
//     are not stored;
//   * the block after the last holds ones, so that its row of the product is the
//     sum of dY over the pixels: the bias gradient (c_in = 128 leaves no room
//     for it and runs k_bias_grad);
//   * one warp per tap row dy issues (one thread reaches a third of the rate),
//     into per-(dy, 16 blocks) FP32 accumulators that stay in TMEM for the CTA's
//     whole run; at the end four warps write them to a per-CTA partial buffer,
//     which k_wgrad_reduce sums in a fixed order (no atomics).
// One training step's eleven weight gradients at 16 x 256 x 256 took 1560 us
// with one tap an instruction and one issuing thread (8-16 % of the tensor
// pipe), plus 267 for the reduction, 124 for the bias sums and 33 for a gather.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>
#include <cstring>

#include "denoiser.cuh"
#include "per_device.h"
#include "rtgb.h"
#include "tc_primitives.cuh"

namespace rtgb {
namespace {

constexpr int kTileW = 8;
constexpr int kTileH = 16;
constexpr int kHaloH = kTileH + 2;
constexpr int kRow = kTileW * 16;                    // 128: next pixel row of a box
constexpr int kXBox = kHaloH * kRow;                 // 2304: 8 channels of one shifted copy
constexpr int kYBox = kTileH * kRow;                 // 2048: 8 channels of dY
constexpr int kMBlocks = 16;                         // 8-channel blocks of an instruction's M = 128
constexpr int kMaxStages = 4;
constexpr int kWgradSmemMax = 227 * 1024;
constexpr int kIssuers = 3;                          // one warp per tap row dy
constexpr int kWgradThreads = 32 * (1 + kIssuers + 4);  // producer, issuers, four epilogue warps
constexpr int kSpin = 1 << 22;

// How a layer maps onto the kernel (host and device).
struct WgradShape {
    int xboxes, blocks, groups;  // X blocks, (dx, block) rows, instructions per dy and K step
    bool ones;                   // room for the row of ones
    int stage_bytes, stages, smem;
    int dys;                     // tap rows per CTA: their accumulators fit 512 TMEM columns
};

WgradShape wgrad_shape(int cin, int cout) {
    WgradShape w{};
    w.xboxes = cin / 8;
    w.blocks = 3 * w.xboxes;
    w.groups = (w.blocks + kMBlocks - 1) / kMBlocks;
    w.ones = w.blocks < w.groups * kMBlocks;
    w.stage_bytes = (w.blocks + (w.ones ? 1 : 0)) * kXBox + (cout / 8) * kYBox;
    // an instruction reads all 16 blocks of its group, also past the last stage's end
    const int tail = w.groups * kMBlocks * kXBox;
    for (w.stages = kMaxStages; w.stages > 1; --w.stages) {
        if (256 + (w.stages - 1) * w.stage_bytes + (w.stage_bytes > tail ? w.stage_bytes : tail) <= kWgradSmemMax) break;
    }
    w.smem = 256 + (w.stages - 1) * w.stage_bytes + (w.stage_bytes > tail ? w.stage_bytes : tail);
    const int fit = 512 / (w.groups * cout);
    w.dys = fit < 3 ? fit : 3;
    return w;
}

struct WgradArgs {
    int n, h, w, cin, cout;
    int blocks, groups, ones, stages, stage_bytes, dys;
    uint32_t tmem_cols;    // power of two >= dys * groups * cout
    float* partial;        // [gridDim.x][9 * cin rows (tap, input channel), then the bias row][cout]
    int* err;
};

// Instruction descriptor of kind::f16 with both operands MN-major.
__host__ __device__ constexpr uint32_t idesc_bf16_f32_mn(int m, int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) | (static_cast<uint32_t>(n >> 3) << 17) |
           (static_cast<uint32_t>(m >> 4) << 24);
}

__global__ void __launch_bounds__(kWgradThreads, 1) k_conv3x3_wgrad(const __grid_constant__ CUtensorMap xmap,
    const __grid_constant__ CUtensorMap ymap, WgradArgs a) {
    extern __shared__ __align__(1024) uint8_t smem[];
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem);  // [kMaxStages] stage landed
    uint64_t* empty_bar = full_bar + kMaxStages;              // [kMaxStages] stage consumed (each issuer's commit)
    uint64_t* done_bar = empty_bar + kMaxStages;              // every UMMA of the CTA completed
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + 128);
    volatile int* stop = reinterpret_cast<volatile int*>(smem + 136);
    uint8_t* stage0 = smem + 256;
    const int xboxes = a.cin >> 3, yboxes = a.cout >> 3;
    const int ybase = (a.blocks + a.ones) * kXBox;  // dY's place in a stage
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int dy0 = static_cast<int>(blockIdx.y) * a.dys;
    const int dys = 3 - dy0 < a.dys ? 3 - dy0 : a.dys;  // tap rows (and issuers) of this CTA

    // the row of ones of every stage (TMA never writes there)
    if (a.ones) {
        const uint32_t one2 = 0x3f803f80u;
        for (int i = threadIdx.x; i < a.stages * (kXBox / 16); i += blockDim.x) {
            const int s = i / (kXBox / 16), k = i - s * (kXBox / 16);
            reinterpret_cast<uint4*>(stage0 + s * a.stage_bytes + a.blocks * kXBox)[k] = make_uint4(one2, one2, one2, one2);
        }
    }
    if (threadIdx.x == 0) {
        for (int i = 0; i < kMaxStages; ++i) {
            tc::mbar_init(full_bar + i, 1);
            tc::mbar_init(empty_bar + i, static_cast<uint32_t>(dys));
        }
        tc::mbar_init(done_bar, static_cast<uint32_t>(dys));
        *stop = 0;
        tc::mbar_fence_init();
    }
    if (warp == 0) {
        tc::tmem_alloc(tmem_slot, a.tmem_cols);
        tc::tmem_relinquish();
    }
    tc::fence_proxy_async_smem();
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    const int tiles_x = (a.w + kTileW - 1) / kTileW;
    const int tiles_y = (a.h + kTileH - 1) / kTileH;
    const int per_image = tiles_x * tiles_y;
    const int total = per_image * a.n;
    const int count = static_cast<int>(blockIdx.x) < total ? (total - 1 - static_cast<int>(blockIdx.x)) / static_cast<int>(gridDim.x) + 1 : 0;
    auto fail = [&](int code) {
        *stop = 1;
        if (a.err != nullptr) atomicExch(a.err, code);
    };

    if (warp == 0) {
        // ---- producer
        if (lane == 0) {
            int issued = 0;
            for (int j = 0; j < count; ++j) {
                const int s = j % a.stages;
                if (j >= a.stages &&
                    !tc::mbar_wait_or_abort(empty_bar + s, static_cast<uint32_t>(j / a.stages - 1) & 1u, kSpin, stop)) {
                    fail(11);
                    break;
                }
                const int tile = static_cast<int>(blockIdx.x) + j * static_cast<int>(gridDim.x);
                const int img = tile / per_image;
                const int t = tile - img * per_image;
                const int ty = t / tiles_x;
                const int x0 = (t - ty * tiles_x) * kTileW;
                const int y0 = ty * kTileH;
                uint8_t* st = stage0 + s * a.stage_bytes;
                tc::mbar_arrive_expect_tx(full_bar + s, static_cast<uint32_t>(a.blocks * kXBox + yboxes * kYBox));
                for (int dx = 0; dx < 3; ++dx) {
                    for (int b = 0; b < xboxes; ++b) {
                        tc::tma_load_3d(st + (dx * xboxes + b) * kXBox, &xmap, full_bar + s, 8 * (x0 - 1 + dx), y0 - 1,
                            img * xboxes + b);
                    }
                }
                for (int b = 0; b < yboxes; ++b) {
                    tc::tma_load_3d(st + ybase + b * kYBox, &ymap, full_bar + s, 8 * x0, y0, img * yboxes + b);
                }
                issued = j + 1;
            }
            // every load has landed before shared memory is released
            for (int j = issued > a.stages ? issued - a.stages : 0; j < issued; ++j) {
                tc::mbar_wait(full_bar + j % a.stages, static_cast<uint32_t>(j / a.stages) & 1u, kSpin);
            }
        }
        __syncwarp();
    } else if (warp <= kIssuers) {
        // ---- issuers: warp 1 + q takes tap row dy0 + q; per tile and 16-block group, 8 UMMAs of 16 pixels
        const int q = warp - 1;
        if (lane == 0 && q < dys) {
            const uint32_t idesc = idesc_bf16_f32_mn(128, a.cout);
            bool committed = false;
            for (int j = 0; j < count; ++j) {
                const int s = j % a.stages;
                if (!tc::mbar_wait_or_abort(full_bar + s, static_cast<uint32_t>(j / a.stages) & 1u, kSpin, stop)) {
                    fail(12);
                    break;
                }
                tc::tc_fence_after();
                const uint32_t xs = tc::smem_u32(stage0 + s * a.stage_bytes) + static_cast<uint32_t>((dy0 + q) * kRow);
                const uint32_t ys = tc::smem_u32(stage0 + s * a.stage_bytes) + static_cast<uint32_t>(ybase);
                const uint64_t b_first = tc::smem_desc(ys, kRow, kYBox);
                for (int g = 0; g < a.groups; ++g) {
                    const uint32_t acc = tmem + static_cast<uint32_t>((q * a.groups + g) * a.cout);
                    // pixels of tile rows 2k, 2k + 1: box rows 2k + dy, 2k + dy + 1. The descriptors step by
                    // constant adds (their address field is the address / 16 and never carries out of it)
                    uint64_t ad = tc::smem_desc(xs + static_cast<uint32_t>(g * kMBlocks * kXBox), kRow, kXBox);
                    uint64_t bd = b_first;
#pragma unroll
                    for (int k = 0; k < kTileH / 2; ++k) {
                        tc::umma_bf16(acc, ad, bd, idesc, (j > 0 || k > 0) ? 1u : 0u);
                        ad += 2 * kRow / 16;
                        bd += 2 * kRow / 16;
                    }
                }
                tc::umma_commit(empty_bar + s);
                committed = true;
            }
            if (committed) tc::umma_commit(done_bar);
            else tc::mbar_arrive(done_bar);  // nothing issued: the epilogue writes zeros
        }
        __syncwarp();
    } else {
        // ---- epilogue: TMEM lane = (dx, input channel) row of a group, columns = output channels
        const int quarter = warp & 3;
        const bool done = tc::mbar_wait_or_abort(done_bar, 0u, kSpin, stop);
        if (__all_sync(0xffffffffu, done)) {
            tc::tc_fence_after();
            const int m = quarter * 32 + lane;
            float* mine = a.partial + static_cast<long long>(blockIdx.x) * (9 * a.cin + 1) * a.cout;
            for (int q = 0; q < dys; ++q) {
                for (int g = 0; g < a.groups; ++g) {
                    const int block = g * kMBlocks + (m >> 3);
                    const int dx = block / xboxes;
                    int row = -1;  // of the partial buffer
                    if (block < a.blocks) row = ((dy0 + q) * 3 + dx) * a.cin + (block - dx * xboxes) * 8 + (m & 7);
                    else if (a.ones && block == a.blocks && (m & 7) == 0 && dy0 + q == 0) row = 9 * a.cin;
                    for (int c = 0; c < (a.cout >> 4); ++c) {
                        uint32_t v[16];
                        tc::tmem_ld16(tmem + (static_cast<uint32_t>(quarter * 32) << 16) +
                                          static_cast<uint32_t>((q * a.groups + g) * a.cout + c * 16), v);
                        tc::tmem_wait_ld();
                        if (row < 0) continue;
                        float4* dst = reinterpret_cast<float4*>(mine + static_cast<long long>(row) * a.cout + c * 16);
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            dst[e] = count > 0 ? make_float4(__uint_as_float(v[4 * e]), __uint_as_float(v[4 * e + 1]),
                                                     __uint_as_float(v[4 * e + 2]), __uint_as_float(v[4 * e + 3]))
                                               : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                        }
                    }
                }
            }
        } else if (lane == 0) {
            fail(13);
        }
    }
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    if (warp == 0) tc::tmem_dealloc(tmem, a.tmem_cols);
}

// dW[o][i][tap] (PyTorch's out x in x 3 x 3 order, the used channels only) and,
// from the row of ones, db[o] = sums over the CTAs' partials: a block sums 32
// runs of four output channels, eight threads a run, each every eighth CTA in
// order and the eight sums in order; a warp reads 512 contiguous bytes. (A thread
// per element walking all CTAs with neighbours in other taps' rows took 24 us a
// layer of a training step.)
constexpr int kReduceRuns = 32;
constexpr int kReduceSlices = 8;
__device__ __forceinline__ void wgrad_reduce(const WgradReduce& t) {
    const float* __restrict__ partial = t.partial;
    const int ctas = t.ctas, cin = t.cin, cout = t.cout, cin_used = t.cin_used, cout_used = t.cout_used;
    const int bias_row = t.bias_row;
    float* __restrict__ dw = t.dw;
    float* __restrict__ db = t.db;
    __shared__ float4 sums[kReduceSlices][kReduceRuns];
    const int run = threadIdx.x % kReduceRuns, slice = threadIdx.x / kReduceRuns;
    const int quads = cout >> 2;
    const int rows = 9 * cin + 1;
    const long long e = static_cast<long long>(blockIdx.x) * kReduceRuns + run;
    const int row = static_cast<int>(e / quads), o0 = static_cast<int>(e % quads) * 4;
    const bool inside = row < 9 * cin || (row == 9 * cin && bias_row != 0);
    float4 s = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (inside) {
        const float4* src = reinterpret_cast<const float4*>(partial) + e;
        const long long stride = static_cast<long long>(rows) * quads;
#pragma unroll 4
        for (int c = slice; c < ctas; c += kReduceSlices) {
            const float4 v = src[c * stride];
            s.x += v.x;
            s.y += v.y;
            s.z += v.z;
            s.w += v.w;
        }
    }
    sums[slice][run] = s;
    __syncthreads();
    if (slice != 0 || !inside) return;
    for (int k = 1; k < kReduceSlices; ++k) {
        const float4 v = sums[k][run];
        s.x += v.x;
        s.y += v.y;
        s.z += v.z;
        s.w += v.w;
    }
    const float out[4] = {s.x, s.y, s.z, s.w};
    const int tap = row / cin, i = row - tap * cin;
    for (int k = 0; k < 4; ++k) {
        const int o = o0 + k;
        if (o >= cout_used) break;
        if (row == 9 * cin) {
            if (db != nullptr) db[o] = out[k];
        } else if (i < cin_used) {
            dw[(static_cast<long long>(o) * cin_used + i) * 9 + tap] = out[k];
        }
    }
}

__global__ void __launch_bounds__(kReduceRuns * kReduceSlices) k_wgrad_reduce(WgradReduce task) { wgrad_reduce(task); }

// Every layer of a training step, blockIdx.y the layer (blocks past a layer's end do nothing).
__global__ void __launch_bounds__(kReduceRuns * kReduceSlices) k_wgrad_reduce_all(const WgradReduce* __restrict__ tasks) {
    wgrad_reduce(tasks[blockIdx.y]);
}

// db[o] += sum over pixels of dY (blocked layout, `hw` pixels per image); a
// block sums a run of pixels of one 8-channel block: each thread a strided
// slice of 16-byte loads, then warp shuffles and a shared-memory pass across
// the block's warps, so each block adds one value per channel (atomics on the
// few bias words used to come from every warp and serialised in L2).
constexpr int kBiasThreads = 256;
constexpr int kBiasLoadsPerThread = 16;

__global__ void __launch_bounds__(kBiasThreads) k_bias_grad(const __nv_bfloat16* __restrict__ dy, long long hw,
    int cout, int cout_used, float* __restrict__ db) {
    __shared__ float part[kBiasThreads / 32][8];
    const int blocks = cout >> 3;
    const int cb = blockIdx.y % blocks, img = blockIdx.y / blocks;
    const __nv_bfloat16* base = dy + (static_cast<long long>(img) * blocks + cb) * hw * 8;
    float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (long long p = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; p < hw;
         p += static_cast<long long>(gridDim.x) * blockDim.x) {
        const uint4 q = *reinterpret_cast<const uint4*>(base + p * 8);
        const __nv_bfloat16* v = reinterpret_cast<const __nv_bfloat16*>(&q);
#pragma unroll
        for (int k = 0; k < 8; ++k) acc[k] += __bfloat162float(v[k]);
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        float v = acc[k];
        for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
        if (lane == 0) part[warp][k] = v;
    }
    __syncthreads();
    if (threadIdx.x < 8 && cb * 8 + static_cast<int>(threadIdx.x) < cout_used) {
        float v = 0.0f;
        for (int w = 0; w < kBiasThreads / 32; ++w) v += part[w][threadIdx.x];
        atomicAdd(db + cb * 8 + threadIdx.x, v);
    }
}

// Where the single-layer entry point takes its partials from, in stream order and
// one allocation per call: calls on several streams and devices share nothing.
// The pool keeps up to the largest layer's partials between calls (45 MB on 152
// SMs), as a buffer kept for the process would: a call alone takes 4 us more than
// with such a buffer (64 x 64, 16 -> 16 channels 25 against 21 us), one among
// others 1 us (16 x 256 x 256, 32 -> 32 channels 73.4 against 71.9).
constexpr uint64_t kKeptPartials = 64u << 20;

cudaError_t partials_pool(cudaMemPool_t* out) {
    static OncePerDevice once;
    static cudaMemPool_t pools[kMaxDevices] = {};
    int device = 0;
    cudaError_t e = once.run([](int dev) {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaError_t made = cudaMemPoolCreate(&pools[dev], &props);
        uint64_t keep = kKeptPartials;
        if (made == cudaSuccess) made = cudaMemPoolSetAttribute(pools[dev], cudaMemPoolAttrReleaseThreshold, &keep);
        return made;
    });
    if (e == cudaSuccess) e = cudaGetDevice(&device);
    if (e == cudaSuccess) *out = pools[device];
    return e;
}

void set_message(char* msg, size_t cap, const char* text) {
    if (msg != nullptr && cap > 0) std::snprintf(msg, cap, "%s", text);
}

}  // namespace

static int reduce_blocks(int cin, int cout) {
    const int runs = (9 * cin + 1) * (cout / 4);
    return (runs + kReduceRuns - 1) / kReduceRuns;
}

cudaError_t launch_wgrad_reduce_all(const WgradReduce* tasks, int count, int blocks, cudaStream_t stream) {
    k_wgrad_reduce_all<<<dim3(static_cast<unsigned>(blocks), static_cast<unsigned>(count)), kReduceRuns * kReduceSlices, 0,
        stream>>>(tasks);
    return cudaGetLastError();
}

int wgrad_reduce_blocks(int cin, int cout) { return reduce_blocks(cin, cout); }

cudaError_t launch_conv3x3_wgrad(const void* x, int n, int h, int w, int cin, const void* dy, int cout, int cin_used,
    int cout_used, float* dweight, float* dbias, int* err, int sms, cudaStream_t stream, float* partial,
    size_t partial_bytes, WgradReduce* later) {
    static OncePerDevice once;
    const cudaError_t attr = once.run([](int) {
        return cudaFuncSetAttribute(k_conv3x3_wgrad, cudaFuncAttributeMaxDynamicSharedMemorySize, kWgradSmemMax);
    });
    if (attr != cudaSuccess) return attr;
    CUtensorMap xmap, ymap;
    if (!blocked_tensor_map(&xmap, x, n, h, w, cin, kTileW, kHaloH) ||
        !blocked_tensor_map(&ymap, dy, n, h, w, cout, kTileW, kTileH)) {
        return cudaErrorInvalidValue;
    }
    const long long tiles = static_cast<long long>((w + kTileW - 1) / kTileW) * ((h + kTileH - 1) / kTileH) * n;
    const int gx = static_cast<int>(tiles < sms ? tiles : sms);
    const WgradShape sh = wgrad_shape(cin, cout);
    const int gy = (3 + sh.dys - 1) / sh.dys;
    if (sh.smem > kWgradSmemMax || wgrad_partial_bytes(gx, cin, cout) > partial_bytes) return cudaErrorInvalidValue;
    uint32_t cols = 32;
    while (cols < static_cast<uint32_t>(sh.dys * sh.groups * cout)) cols <<= 1;
    const WgradArgs a{n, h, w, cin, cout, sh.blocks, sh.groups, sh.ones ? 1 : 0, sh.stages, sh.stage_bytes, sh.dys, cols,
        partial, err};
    k_conv3x3_wgrad<<<dim3(gx, gy), kWgradThreads, sh.smem, stream>>>(xmap, ymap, a);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const WgradReduce task{partial, gx, cin, cout, cin_used, cout_used, a.ones, dweight, dbias};
    if (later != nullptr) {
        *later = task;
    } else {
        k_wgrad_reduce<<<reduce_blocks(cin, cout), kReduceRuns * kReduceSlices, 0, stream>>>(task);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    if (dbias != nullptr && !sh.ones) {
        if ((e = cudaMemsetAsync(dbias, 0, static_cast<size_t>(cout_used) * sizeof(float), stream)) != cudaSuccess) return e;
        const long long hw = static_cast<long long>(h) * w;
        constexpr long long kPerBlock = static_cast<long long>(kBiasThreads) * kBiasLoadsPerThread;
        long long bx = (hw + kPerBlock - 1) / kPerBlock;
        bx = bx < 64 ? bx : 64;
        k_bias_grad<<<dim3(static_cast<unsigned>(bx), static_cast<unsigned>(n * (cout >> 3))), kBiasThreads, 0, stream>>>(
            static_cast<const __nv_bfloat16*>(dy), hw, cout, cout_used, dbias);
        e = cudaGetLastError();
    }
    return e;
}

size_t wgrad_partial_bytes(int ctas, int cin, int cout) {
    return static_cast<size_t>(ctas) * (9 * static_cast<size_t>(cin) + 1) * cout * sizeof(float);
}

}  // namespace rtgb

extern "C" rtgb_status rtgb_conv3x3_wgrad_bf16(const void* x, int32_t n, int32_t h, int32_t w, int32_t c_in,
    const void* dy, int32_t c_out, float* dweight, float* dbias, int32_t* device_error, void* stream, char* message,
    size_t message_size) {
    using namespace rtgb;
    set_message(message, message_size, "");
    if (x == nullptr || dy == nullptr || dweight == nullptr || n <= 0 || h <= 0 || w <= 0) {
        set_message(message, message_size, "null pointer or empty extent");
        return RTGB_INVALID_ARGUMENT;
    }
    if (c_in < 16 || c_in > 128 || c_in % 16 != 0 || c_out < 16 || c_out > 64 || c_out % 16 != 0) {
        set_message(message, message_size, "c_in must be a multiple of 16 in [16, 128], c_out a multiple of 16 in [16, 64]");
        return RTGB_INVALID_ARGUMENT;
    }
    if ((reinterpret_cast<uintptr_t>(x) & 15u) != 0 || (reinterpret_cast<uintptr_t>(dy) & 15u) != 0) {
        set_message(message, message_size, "tensors must be 16-byte aligned");
        return RTGB_INVALID_ARGUMENT;
    }
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    sms = sms > 0 ? sms : 1;
    const cudaStream_t st = static_cast<cudaStream_t>(stream);
    const size_t bytes = wgrad_partial_bytes(sms, c_in, c_out);
    cudaMemPool_t pool = nullptr;
    void* partial = nullptr;
    cudaError_t e = partials_pool(&pool);
    if (e == cudaSuccess) e = cudaMallocFromPoolAsync(&partial, bytes, pool, st);
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        set_message(message, message_size, "out of device memory for the weight-gradient partials");
        return RTGB_RUNTIME_ERROR;
    }
    e = launch_conv3x3_wgrad(x, n, h, w, c_in, dy, c_out, c_in, c_out, dweight, dbias, device_error, sms, st,
        static_cast<float*>(partial), bytes);
    const cudaError_t freed = cudaFreeAsync(partial, st);
    if (e == cudaSuccess) e = freed;
    if (e != cudaSuccess) {
        set_message(message, message_size, cudaGetErrorString(e));
        return RTGB_RUNTIME_ERROR;
    }
    return RTGB_OK;
}
