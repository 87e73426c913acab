// Native training of the denoiser U-Net: forward, log-space L1 loss,
// backward and Adam, all on this library's kernels (no framework):
//   * forward: k_conv3x3 per layer with the fused pooling / upsampling, every
//     activation kept (BF16, channel-blocked);
//   * input gradients: k_conv3x3 itself with flipped, transposed weights
//     (dX = conv(dZ, W^T flipped)), split into launches of <= 64 output
//     channels;
//   * weight and bias gradients: k_conv3x3_wgrad (denoiser_train.cu);
//   * ReLU masks: in the input-gradient convolutions' epilogue;
//   * the backward of 2 x 2 average pooling and of nearest upsampling (with
//     their ReLU masks), the loss gradient, weight packing and Adam:
//     elementwise kernels below.
// Gradients flow in BF16 between layers and accumulate in FP32 inside each
// GEMM; the master parameters and Adam moments are FP32. Batches are n crops
// of h x w with h and w multiples of 4 (the pooled sizes then halve exactly).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <new>
#include <string>
#include <vector>

#include "denoiser.cuh"
#include "rtgb.h"

#include <initializer_list>

namespace rtgb {
namespace {

__device__ __forceinline__ float bf2f(__nv_bfloat16 v) { return __bfloat162float(v); }

// Loss gradient of mean |out - target| over n x h x w x 3 (log1p radiance):
// sign / count into channels 0..2 of a 16-channel gradient, 0 elsewhere; the
// loss sum goes to *loss. A thread moves a pixel's 16 channels as two 16-byte
// stores (`hw` pixels per image), a block adds one value to the sum (2-byte
// stores and an atomic per warp took 58 us for 16 x 256 x 256 pixels).
__global__ void __launch_bounds__(256) k_loss_grad(const __nv_bfloat16* __restrict__ out16, const float* __restrict__ target,
    long long px, int hw, __nv_bfloat16* __restrict__ g16, double* loss) {
    __shared__ double part[8];
    const float inv = 1.0f / static_cast<float>(px * 3);
    double local = 0.0;
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < px;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        const long long img = i / hw, p = i - img * hw;
        const long long at = (img * 2 * hw + p) * 8;  // the pixel in channel block 0; block 1 is hw pixels on
        const uint2 q = *reinterpret_cast<const uint2*>(out16 + at);
        const __nv_bfloat16* e = reinterpret_cast<const __nv_bfloat16*>(&q);
        __align__(16) __nv_bfloat16 g[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            float v = 0.0f;
            if (c < 3) {
                const float d = bf2f(e[c]) - target[i * 3 + c];
                local += fabsf(d);
                v = d > 0.0f ? inv : (d < 0.0f ? -inv : 0.0f);
            }
            g[c] = __float2bfloat16_rn(v);
        }
        *reinterpret_cast<uint4*>(g16 + at) = *reinterpret_cast<const uint4*>(g);
        *reinterpret_cast<uint4*>(g16 + at + 8ll * hw) = make_uint4(0, 0, 0, 0);
    }
    for (int off = 16; off > 0; off >>= 1) local += __shfl_down_sync(0xffffffffu, local, off);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = local;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) local += part[w];
        atomicAdd(loss, local);
    }
}

// Backward passes on whole 8-channel blocks (every channel count and offset of
// the U-Net is a multiple of 8): a thread moves one pixel's 8 channels as one
// 16-byte load per operand, and the index arithmetic is 32-bit on (image,
// channel block, pixel). (A ReLU alone needs no pass: the input-gradient
// convolution stores its output masked.)
__device__ __forceinline__ void unpack8(const uint4& q, float f[8]) {
    const __nv_bfloat16* v = reinterpret_cast<const __nv_bfloat16*>(&q);
#pragma unroll
    for (int k = 0; k < 8; ++k) f[k] = bf2f(v[k]);
}
__device__ __forceinline__ uint4 pack8(const float f[8]) {
    uint4 q;
    __nv_bfloat16* v = reinterpret_cast<__nv_bfloat16*>(&q);
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = __float2bfloat16_rn(f[k]);
    return q;
}
// 16-byte unit of channel block `cb` (of `cbs`) at pixel p of image img, hw pixels
__device__ __forceinline__ long long unit(int img, int cbs, int cb, int hw, int p) {
    return (static_cast<long long>(img) * cbs + cb) * hw + p;
}

// Backward of nearest 2x upsampling followed by the ReLU of the layer that
// produced it: out (h x w, dense channel blocks) = (sum of the 2 x 2 gradient
// block of g) * (y > 0), y being the upsampled output itself (any pixel of
// its 2 x 2 block holds the value).
__global__ void k_up_backward_mask8(const uint4* __restrict__ g, int g_cbs, int g_cb0, const uint4* __restrict__ y,
    int y_cbs, int y_cb0, uint4* __restrict__ out, int blocks, int n, int h, int w) {
    const int hw = h * w, w2 = 2 * w, hw2 = 4 * hw;
    const long long total = static_cast<long long>(n) * blocks * hw;
    for (long long j = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; j < total;
         j += static_cast<long long>(gridDim.x) * blockDim.x) {
        const int p = static_cast<int>(j % hw);
        const int t = static_cast<int>(j / hw);
        const int cb = t % blocks, img = t / blocks;
        const int yy = p / w, x = p - yy * w;
        float s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        for (int dy = 0; dy < 2; ++dy) {
            for (int dx = 0; dx < 2; ++dx) {
                float v[8];
                unpack8(g[unit(img, g_cbs, g_cb0 + cb, hw2, (2 * yy + dy) * w2 + 2 * x + dx)], v);
#pragma unroll
                for (int k = 0; k < 8; ++k) s[k] += v[k];
            }
        }
        float yv[8], o[8];
        unpack8(y[unit(img, y_cbs, y_cb0 + cb, hw2, 2 * yy * w2 + 2 * x)], yv);
#pragma unroll
        for (int k = 0; k < 8; ++k) o[k] = yv[k] > 0.0f ? s[k] : 0.0f;
        out[unit(img, blocks, cb, hw, p)] = pack8(o);
    }
}

// Gradient of a layer whose output feeds both a skip connection (gradient g)
// and a 2 x 2 average pooling (gradient gp at half size): out = (g + gp / 4) *
// (y > 0) into a dense tensor (h, w even).
__global__ void k_pool_backward_mask8(const uint4* __restrict__ g, int g_cbs, int g_cb0, const uint4* __restrict__ gp,
    const uint4* __restrict__ y, int y_cbs, int y_cb0, uint4* __restrict__ out, int blocks, int n, int h, int w) {
    const int hw = h * w, wh = w / 2, hwh = (h / 2) * wh;
    const long long total = static_cast<long long>(n) * blocks * hw;
    for (long long j = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; j < total;
         j += static_cast<long long>(gridDim.x) * blockDim.x) {
        const int p = static_cast<int>(j % hw);
        const int t = static_cast<int>(j / hw);
        const int cb = t % blocks, img = t / blocks;
        const int yy = p / w, x = p - yy * w;
        float gv[8], pv[8], yv[8], o[8];
        unpack8(g[unit(img, g_cbs, g_cb0 + cb, hw, p)], gv);
        unpack8(gp[unit(img, blocks, cb, hwh, (yy / 2) * wh + x / 2)], pv);
        unpack8(y[unit(img, y_cbs, y_cb0 + cb, hw, p)], yv);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const float sv = gv[k] + 0.25f * pv[k];
            o[k] = yv[k] > 0.0f ? sv : 0.0f;
        }
        out[unit(img, blocks, cb, hw, p)] = pack8(o);
    }
}

// One tensor of a step's weight packing: FP32 weights (cout_used x cin_used x
// 3 x 3, then the bias, at params + src) as rtgb_conv3x3_pack_weights packs
// them, [tap][cin/8][cout][8] BF16 with zero padding; with `transposed` the
// packed kernel is the input-gradient one, W'[i][o][2 - dy][2 - dx], for output
// channels [o0, o0 + cout) of it (i.e. layer input channels) and input channels
// = the layer's cout. With `bias` set instead of `packed`, the bias padded to cout.
struct PackTask {
    long long src;
    int cout_used, cin_used, transposed, o0, cout, cin;
    __nv_bfloat16* packed;
    float* bias;
};

// Every layer's packed tensors in one launch, blockIdx.y the task (24 launches
// and 22 copies of a few KB each were 70 us of device time and most of a small
// step's launches).
__global__ void k_pack_weights(const float* __restrict__ params, const PackTask* __restrict__ tasks) {
    const PackTask t = tasks[blockIdx.y];
    const float* __restrict__ wsrc = params + t.src;
    const int total = t.packed != nullptr ? 9 * t.cin * t.cout : t.cout;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < total; e += gridDim.x * blockDim.x) {
        if (t.packed == nullptr) {
            t.bias[e] = e < t.cout_used ? wsrc[static_cast<long long>(t.cout_used) * t.cin_used * 9 + e] : 0.0f;
            continue;
        }
        const int j = e & 7;
        const int o = (e >> 3) % t.cout;
        const int b = (e >> 3) / t.cout % (t.cin >> 3);
        const int tap = (e >> 3) / t.cout / (t.cin >> 3);
        const int i = b * 8 + j;
        float v = 0.0f;
        if (!t.transposed) {
            if (o < t.cout_used && i < t.cin_used) v = wsrc[(static_cast<long long>(o) * t.cin_used + i) * 9 + tap];
        } else {
            // packed output channel o = layer input channel o0 + o, packed input i = layer output channel
            const int li = t.o0 + o, lo = i;
            if (li < t.cin_used && lo < t.cout_used) v = wsrc[(static_cast<long long>(lo) * t.cin_used + li) * 9 + (8 - tap)];
        }
        t.packed[e] = __float2bfloat16_rn(v);
    }
}

// Adam (Kingma & Ba 2015) on the FP32 master parameters, bias-corrected.
__global__ void k_adam(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m, float* __restrict__ v,
    long long count, float lr, float b1, float b2, float eps, float c1, float c2) {
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < count;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        const float gi = g[i];
        const float mi = b1 * m[i] + (1.0f - b1) * gi;
        const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    }
}

int grid_of(long long work) {
    long long g = (work + 255) / 256;
    return static_cast<int>(g < 1 ? 1 : (g < 4096 ? g : 4096));
}

}  // namespace

struct Trainer {
    int n = 0, h = 0, w = 0, sms = 1;
    long long count = 0;                 // parameters
    cudaStream_t stream = nullptr;
    std::vector<void*> allocations;
    // FP32 master parameters (flat, layer order: weight out x in x 3 x 3, then bias), gradients, Adam moments
    float *params = nullptr, *grads = nullptr, *m = nullptr, *v = nullptr;
    long long offset[kLayerCount] = {};  // of each layer's weight in the flat vector
    // packed BF16 weights: forward per layer, input-gradient per layer and 64-channel chunk
    __nv_bfloat16* wf[kLayerCount] = {};
    __nv_bfloat16* wb[kLayerCount][2] = {};
    float* bias[kLayerCount] = {};       // FP32 bias (forward), padded to cout
    PackTask* pack_tasks = nullptr;      // device: what k_pack_weights writes
    int pack_count = 0;
    float* zero_bias = nullptr;          // 128 zeros for the input-gradient convolutions
    float* partial = nullptr;
    size_t partial_bytes = 0;
    size_t partial_at[kLayerCount] = {};
    WgradReduce reduce_list[kLayerCount] = {};  // what the step's reduction launch sums; the same every step
    WgradReduce* reduce_tasks = nullptr;        // device copy
    bool reduce_listed = false;
    int reduce_blocks = 0;
    // activations (channel-blocked BF16)
    __nv_bfloat16 *t1, *cat1, *p1, *t2, *cat2, *p2, *t3, *t4, *t5, *t6, *out16;
    // gradients
    __nv_bfloat16 *g_out16, *g_t6, *g_t5, *g_cat1, *g_u7, *g_t4, *g_cat2, *g_u5, *g_t3, *g_p2, *g3, *g_t2, *g_p1, *g1,
        *g_t1;
    double* loss = nullptr;
    int* err = nullptr;
    int steps = 0;
    std::string error;

    template <typename T>
    T* alloc(size_t count_elems) {
        void* p = nullptr;
        if (cudaMalloc(&p, count_elems * sizeof(T)) != cudaSuccess) throw std::string("out of device memory");
        allocations.push_back(p);
        cudaMemset(p, 0, count_elems * sizeof(T));
        return static_cast<T*>(p);
    }

    ~Trainer() {
        if (stream) cudaStreamSynchronize(stream);
        for (void* p : allocations) cudaFree(p);
        if (stream) cudaStreamDestroy(stream);
    }

    void init(int n_, int h_, int w_, const float* host_params, long long count_) {
        n = n_;
        h = h_;
        w = w_;
        if (cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking) != cudaSuccess) throw std::string("stream");
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        long long off = 0;
        for (int l = 0; l < kLayerCount; ++l) {
            offset[l] = off;
            off += static_cast<long long>(kLayers[l].cout_used) * kLayers[l].cin_used * 9 + kLayers[l].cout_used;
        }
        if (count_ != off) throw std::string("parameter count mismatch");
        count = off;
        params = alloc<float>(count);
        grads = alloc<float>(count);
        m = alloc<float>(count);
        v = alloc<float>(count);
        cudaMemcpy(params, host_params, count * sizeof(float), cudaMemcpyHostToDevice);
        for (int l = 0; l < kLayerCount; ++l) {
            const LayerSpec& L = kLayers[l];
            wf[l] = alloc<__nv_bfloat16>(9 * static_cast<size_t>(L.cin) * L.cout);
            for (int k = 0; k < 2; ++k) wb[l][k] = alloc<__nv_bfloat16>(9 * static_cast<size_t>(L.cout) * 64);
            bias[l] = alloc<float>(L.cout);
        }
        zero_bias = alloc<float>(128);
        list_pack_tasks();
        // a partial buffer per layer: one launch at the end of the backward pass reduces them all
        for (int l = 0; l < kLayerCount; ++l) {
            partial_at[l] = partial_bytes / sizeof(float);
            partial_bytes += (wgrad_partial_bytes(sms, kLayers[l].cin, kLayers[l].cout) + 255) & ~size_t(255);
            reduce_blocks = std::max(reduce_blocks, wgrad_reduce_blocks(kLayers[l].cin, kLayers[l].cout));
        }
        reduce_tasks = alloc<WgradReduce>(kLayerCount);
        partial = alloc<float>(partial_bytes / sizeof(float));
        const size_t full = static_cast<size_t>(n) * h * w, half = full / 4, quarter = full / 16;
        t1 = alloc<__nv_bfloat16>(full * 32);
        cat1 = alloc<__nv_bfloat16>(full * 80);
        p1 = alloc<__nv_bfloat16>(half * 32);
        t2 = alloc<__nv_bfloat16>(half * 48);
        cat2 = alloc<__nv_bfloat16>(half * 112);
        p2 = alloc<__nv_bfloat16>(quarter * 48);
        t3 = alloc<__nv_bfloat16>(quarter * 64);
        t4 = alloc<__nv_bfloat16>(half * 48);
        t5 = alloc<__nv_bfloat16>(full * 32);
        t6 = alloc<__nv_bfloat16>(full * 32);
        out16 = alloc<__nv_bfloat16>(full * 16);
        g_out16 = alloc<__nv_bfloat16>(full * 16);
        g_t6 = alloc<__nv_bfloat16>(full * 32);
        g_t5 = alloc<__nv_bfloat16>(full * 32);
        g_cat1 = alloc<__nv_bfloat16>(full * 80);
        g_u7 = alloc<__nv_bfloat16>(half * 48);
        g_t4 = alloc<__nv_bfloat16>(half * 48);
        g_cat2 = alloc<__nv_bfloat16>(half * 112);
        g_u5 = alloc<__nv_bfloat16>(quarter * 64);
        g_t3 = alloc<__nv_bfloat16>(quarter * 64);
        g_p2 = alloc<__nv_bfloat16>(quarter * 48);
        g3 = alloc<__nv_bfloat16>(half * 48);
        g_t2 = alloc<__nv_bfloat16>(half * 48);
        g_p1 = alloc<__nv_bfloat16>(half * 32);
        g1 = alloc<__nv_bfloat16>(full * 32);
        g_t1 = alloc<__nv_bfloat16>(full * 32);
        loss = alloc<double>(2);  // the sum, then the error word: cleared and read as one
        err = reinterpret_cast<int*>(loss + 1);
        if (conv_init() != cudaSuccess || conv_rows_init() != cudaSuccess) throw std::string("conv_init");
        cudaDeviceSynchronize();
    }

    void check(cudaError_t e, const char* what) {
        if (e != cudaSuccess) throw std::string(what) + ": " + cudaGetErrorString(e);
    }

    // packs every layer's forward and input-gradient weights and copies the biases
    void pack() {
        k_pack_weights<<<dim3(16, static_cast<unsigned>(pack_count)), 256, 0, stream>>>(params, pack_tasks);
        check(cudaGetLastError(), "pack");
    }

    void list_pack_tasks() {
        std::vector<PackTask> tasks;
        for (int l = 0; l < kLayerCount; ++l) {
            const LayerSpec& L = kLayers[l];
            tasks.push_back({offset[l], L.cout_used, L.cin_used, 0, 0, L.cout, L.cin, wf[l], nullptr});
            for (int k = 0; k * 64 < L.cin; ++k) {
                const int oc = L.cin - 64 * k < 64 ? L.cin - 64 * k : 64;
                tasks.push_back({offset[l], L.cout_used, L.cin_used, 1, 64 * k, oc, L.cout, wb[l][k], nullptr});
            }
            tasks.push_back({offset[l], L.cout_used, L.cin_used, 0, 0, L.cout, L.cin, nullptr, bias[l]});
        }
        pack_tasks = alloc<PackTask>(tasks.size());
        pack_count = static_cast<int>(tasks.size());
        check(cudaMemcpy(pack_tasks, tasks.data(), tasks.size() * sizeof(PackTask), cudaMemcpyHostToDevice), "pack tasks");
    }

    // one convolution: input x (cin channels) at hh x ww
    void conv(const void* x, int cin, int hh, int ww, const void* wts, const float* b, int cout, int relu, void* y,
        int ych, int yoff, void* pool = nullptr, int up = 0, const void* relu_of = nullptr) {
        if (conv_rows_fits(n, hh, ww, cin, cout, sms, pool != nullptr || up != 0)) {
            check(launch_conv_rows(x, n, hh, ww, cin, wts, b, cout, relu, y, ych, yoff, err, sms, stream, pool, up, relu_of),
                "conv");
            return;
        }
        CUtensorMap map;
        if (!conv_input_map(&map, x, n, hh, ww, cin)) throw std::string("tensor map");
        check(launch_conv3x3(map, n, hh, ww, cin, wts, b, cout, relu, y, ych, yoff, err, sms, stream, pool, up, 0, relu_of),
            "conv");
    }

    void forward(const void* in16) {
        const int h2 = h / 2, w2 = w / 2, h4 = h / 4, w4 = w / 4;
        conv(in16, 16, h, w, wf[0], bias[0], 32, 1, t1, 32, 0);
        conv(t1, 32, h, w, wf[1], bias[1], 32, 1, cat1, 80, 0, p1);
        conv(p1, 32, h2, w2, wf[2], bias[2], 48, 1, t2, 48, 0);
        conv(t2, 48, h2, w2, wf[3], bias[3], 48, 1, cat2, 112, 0, p2);
        conv(p2, 48, h4, w4, wf[4], bias[4], 64, 1, t3, 64, 0);
        conv(t3, 64, h4, w4, wf[5], bias[5], 64, 1, cat2, 112, 48, nullptr, 1);
        conv(cat2, 112, h2, w2, wf[6], bias[6], 48, 1, t4, 48, 0);
        conv(t4, 48, h2, w2, wf[7], bias[7], 48, 1, cat1, 80, 32, nullptr, 1);
        conv(cat1, 80, h, w, wf[8], bias[8], 32, 1, t5, 32, 0);
        conv(t5, 32, h, w, wf[9], bias[9], 32, 1, t6, 32, 0);
        conv(t6, 32, h, w, wf[10], bias[10], 16, 0, out16, 16, 0);
    }

    // weight/bias gradients of layer l (x: its input, dz: its masked output gradient) into its partials;
    // reduce_gradients sums every layer's into the flat vector
    void wgrad(int l, const void* x, int hh, int ww, const void* dz) {
        const LayerSpec& L = kLayers[l];
        float* dw = grads + offset[l];
        check(launch_conv3x3_wgrad(x, n, hh, ww, L.cin, dz, L.cout, L.cin_used, L.cout_used, dw,
                  dw + static_cast<long long>(L.cout_used) * L.cin_used * 9, err, sms, stream, partial + partial_at[l],
                  wgrad_partial_bytes(sms, L.cin, L.cout), &reduce_list[l]),
            "wgrad");
    }

    void reduce_gradients() {
        if (!reduce_listed) {
            check(cudaMemcpyAsync(reduce_tasks, reduce_list, sizeof reduce_list, cudaMemcpyHostToDevice, stream), "reduce");
            reduce_listed = true;
        }
        check(launch_wgrad_reduce_all(reduce_tasks, kLayerCount, reduce_blocks, stream), "reduce");
    }

    // input gradient of layer l: dX (cin channels, written at channel xoff of an xcs tensor) from dz (cout
    // channels); with `relu_of`, the layer's input after its ReLU, already masked by that ReLU
    void dgrad(int l, const void* dz, int hh, int ww, void* dx, int xcs, int xoff, const void* relu_of = nullptr) {
        const LayerSpec& L = kLayers[l];
        for (int k = 0; k * 64 < L.cin; ++k) {
            const int oc = L.cin - 64 * k < 64 ? L.cin - 64 * k : 64;
            conv(dz, L.cout, hh, ww, wb[l][k], zero_bias, oc, 0, dx, xcs, xoff + 64 * k, nullptr, 0, relu_of);
        }
    }

    void backward(const void* in16) {
        const int h2 = h / 2, w2 = w / 2, h4 = h / 4, w4 = w / 4;
        const long long full = static_cast<long long>(n) * h * w, half = full / 4, quarter = full / 16;
        // head (no ReLU): dZ = loss gradient
        wgrad(10, t6, h, w, g_out16);
        dgrad(10, g_out16, h, w, g_t6, 32, 0, t6);
        // d1b, d1a
        wgrad(9, t5, h, w, g_t6);
        dgrad(9, g_t6, h, w, g_t5, 32, 0, t5);
        wgrad(8, cat1, h, w, g_t5);
        dgrad(8, g_t5, h, w, g_cat1, 80, 0);
        // d2b: its output was upsampled into cat1[32:80]
        k_up_backward_mask8<<<grid_of(half * 6), 256, 0, stream>>>(reinterpret_cast<const uint4*>(g_cat1), 10, 4,
            reinterpret_cast<const uint4*>(cat1), 10, 4, reinterpret_cast<uint4*>(g_u7), 6, n, h2, w2);
        check(cudaGetLastError(), "up backward");
        wgrad(7, t4, h2, w2, g_u7);
        dgrad(7, g_u7, h2, w2, g_t4, 48, 0, t4);
        // d2a
        wgrad(6, cat2, h2, w2, g_t4);
        dgrad(6, g_t4, h2, w2, g_cat2, 112, 0);
        // e3b: its output was upsampled into cat2[48:112]
        k_up_backward_mask8<<<grid_of(quarter * 8), 256, 0, stream>>>(reinterpret_cast<const uint4*>(g_cat2), 14, 6,
            reinterpret_cast<const uint4*>(cat2), 14, 6, reinterpret_cast<uint4*>(g_u5), 8, n, h4, w4);
        check(cudaGetLastError(), "up backward");
        wgrad(5, t3, h4, w4, g_u5);
        dgrad(5, g_u5, h4, w4, g_t3, 64, 0, t3);
        // e3a
        wgrad(4, p2, h4, w4, g_t3);
        dgrad(4, g_t3, h4, w4, g_p2, 48, 0);
        // e2b: output in cat2[0:48] (skip) and pooled into p2
        k_pool_backward_mask8<<<grid_of(half * 6), 256, 0, stream>>>(reinterpret_cast<const uint4*>(g_cat2), 14, 0,
            reinterpret_cast<const uint4*>(g_p2), reinterpret_cast<const uint4*>(cat2), 14, 0, reinterpret_cast<uint4*>(g3), 6, n, h2,
            w2);
        check(cudaGetLastError(), "pool backward");
        wgrad(3, t2, h2, w2, g3);
        dgrad(3, g3, h2, w2, g_t2, 48, 0, t2);
        // e2a
        wgrad(2, p1, h2, w2, g_t2);
        dgrad(2, g_t2, h2, w2, g_p1, 32, 0);
        // e1b: output in cat1[0:32] (skip) and pooled into p1
        k_pool_backward_mask8<<<grid_of(full * 4), 256, 0, stream>>>(reinterpret_cast<const uint4*>(g_cat1), 10, 0,
            reinterpret_cast<const uint4*>(g_p1), reinterpret_cast<const uint4*>(cat1), 10, 0, reinterpret_cast<uint4*>(g1), 4, n, h,
            w);
        check(cudaGetLastError(), "pool backward");
        wgrad(1, t1, h, w, g1);
        dgrad(1, g1, h, w, g_t1, 32, 0, t1);
        // e1a (its input needs no gradient)
        wgrad(0, in16, h, w, g_t1);
        reduce_gradients();
    }

    // forward, loss, backward; then Adam when lr > 0. Returns the mean loss.
    float step(const void* in16, const float* target, float lr) {
        check(cudaMemsetAsync(loss, 0, 2 * sizeof(double), stream), "loss");
        pack();
        forward(in16);
        const long long full = static_cast<long long>(n) * h * w;
        k_loss_grad<<<std::min(grid_of(full), 4 * sms), 256, 0, stream>>>(out16, target, full, h * w, g_out16, loss);
        check(cudaGetLastError(), "loss");
        backward(in16);
        if (lr > 0.0f) {
            ++steps;
            const float c1 = 1.0f - std::pow(0.9f, static_cast<float>(steps));
            const float c2 = 1.0f - std::pow(0.999f, static_cast<float>(steps));
            k_adam<<<grid_of(count), 256, 0, stream>>>(params, grads, m, v, count, lr, 0.9f, 0.999f, 1e-8f, c1, c2);
            check(cudaGetLastError(), "adam");
        }
        double h_result[2] = {0.0, 0.0};
        check(cudaMemcpyAsync(h_result, loss, sizeof h_result, cudaMemcpyDeviceToHost, stream), "loss");
        check(cudaStreamSynchronize(stream), "step");
        const double h_loss = h_result[0];
        int h_err = 0;
        std::memcpy(&h_err, &h_result[1], sizeof h_err);
        if (h_err != 0) throw std::string("a bounded wait inside a training kernel ran out (code ") + std::to_string(h_err) + ")";
        return static_cast<float>(h_loss / static_cast<double>(full * 3));
    }
};

}  // namespace rtgb

struct rtgb_trainer_s {
    rtgb::Trainer t;
};

extern "C" {

rtgb_status rtgb_trainer_create(int32_t n, int32_t h, int32_t w, const float* params, int64_t count, rtgb_trainer* out) {
    if (out == nullptr || params == nullptr || n <= 0 || h <= 0 || w <= 0 || h % 4 != 0 || w % 4 != 0) {
        return RTGB_INVALID_ARGUMENT;
    }
    *out = nullptr;
    auto* tr = new (std::nothrow) rtgb_trainer_s();
    if (tr == nullptr) return RTGB_RUNTIME_ERROR;
    try {
        tr->t.init(n, h, w, params, count);
    } catch (const std::string&) {
        delete tr;
        return RTGB_RUNTIME_ERROR;
    } catch (const std::bad_alloc&) {  // the packing list, an error's text
        delete tr;
        return RTGB_RUNTIME_ERROR;
    }
    *out = tr;
    return RTGB_OK;
}

void rtgb_trainer_destroy(rtgb_trainer t) { delete t; }

rtgb_status rtgb_trainer_step(rtgb_trainer t, const void* input, const float* target, float learning_rate, float* loss) {
    if (t == nullptr || input == nullptr || target == nullptr || !(learning_rate >= 0.0f)) return RTGB_INVALID_ARGUMENT;
    try {
        const float l = t->t.step(input, target, learning_rate);
        if (loss != nullptr) *loss = l;
    } catch (const std::string& e) {
        t->t.error = e;
        return RTGB_RUNTIME_ERROR;
    } catch (const std::bad_alloc&) {
        t->t.error.clear();
        return RTGB_RUNTIME_ERROR;
    }
    return RTGB_OK;
}

rtgb_status rtgb_trainer_gradients(rtgb_trainer t, float* grads) {
    if (t == nullptr || grads == nullptr) return RTGB_INVALID_ARGUMENT;
    return cudaMemcpy(grads, t->t.grads, t->t.count * sizeof(float), cudaMemcpyDeviceToHost) == cudaSuccess
               ? RTGB_OK
               : RTGB_RUNTIME_ERROR;
}

rtgb_status rtgb_trainer_params(rtgb_trainer t, float* params) {
    if (t == nullptr || params == nullptr) return RTGB_INVALID_ARGUMENT;
    return cudaMemcpy(params, t->t.params, t->t.count * sizeof(float), cudaMemcpyDeviceToHost) == cudaSuccess
               ? RTGB_OK
               : RTGB_RUNTIME_ERROR;
}

const char* rtgb_trainer_last_error(rtgb_trainer t) { return t != nullptr ? t->t.error.c_str() : ""; }

}  // extern "C"
