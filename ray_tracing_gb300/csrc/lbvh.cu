// Device LBVH build (Karras 2012, "Maximizing parallelism in the construction
// of BVHs, octrees, and k-d trees"): Morton codes of primitive centroids,
// a stable LSD radix sort (4-bit digits, warp-match ranking), one thread per
// internal node for the hierarchy, and an atomic bottom-up pass for bounds.
//
// Ties between equal Morton codes break by primitive index (the sort is
// stable over index-ordered input, and the Karras prefix length falls back to
// the index when keys are equal), so the leaf order is a pure function of the
// input and oracle/lbvh.py reproduces it bit for bit.
#include "lbvh.cuh"

#include <algorithm>

namespace rtgb {
namespace {

// The loops over a tile's rounds end with the input: a scene of 1024 primitives
// fills four rounds of eight, and the empty ones cost a rebuild about 10 of its
// 315 us (eighteen launches walk such tiles).
constexpr int kSortThreads = 256;
constexpr int kSortItems = 8;
constexpr int kSortTile = kSortThreads * kSortItems;
constexpr int kDigits = 16;

size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

int sort_blocks(int n) { return (n + kSortTile - 1) / kSortTile; }

RTGB_D unsigned int float_to_ordered(float f) {
    const unsigned int u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
RTGB_D float ordered_to_float(unsigned int u) {
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

__global__ void k_init_bounds(unsigned int* bits) {
    if (threadIdx.x < 3) bits[threadIdx.x] = 0xffffffffu;          // min: ordered max
    else if (threadIdx.x < 6) bits[threadIdx.x] = 0u;             // max: ordered min
}

// Centroid bounds via ordered-int atomics (one warp-reduced update per warp).
__global__ void k_centroid_bounds(const float4* __restrict__ lo, const float4* __restrict__ hi, int n,
    unsigned int* bits) {
    unsigned int mn[3] = {0xffffffffu, 0xffffffffu, 0xffffffffu}, mx[3] = {0u, 0u, 0u};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float4 a = lo[i], b = hi[i];
        const float c[3] = {(a.x + b.x) * 0.5f, (a.y + b.y) * 0.5f, (a.z + b.z) * 0.5f};
        for (int k = 0; k < 3; ++k) {
            const unsigned int o = float_to_ordered(c[k]);
            mn[k] = min(mn[k], o);
            mx[k] = max(mx[k], o);
        }
    }
    for (int k = 0; k < 3; ++k) {
        for (int off = 16; off > 0; off >>= 1) {
            mn[k] = min(mn[k], __shfl_xor_sync(0xffffffffu, mn[k], off));
            mx[k] = max(mx[k], __shfl_xor_sync(0xffffffffu, mx[k], off));
        }
    }
    if ((threadIdx.x & 31) == 0) {
        for (int k = 0; k < 3; ++k) {
            atomicMin(bits + k, mn[k]);
            atomicMax(bits + 3 + k, mx[k]);
        }
    }
}

__global__ void k_morton(const float4* __restrict__ lo, const float4* __restrict__ hi, int n,
    const unsigned int* __restrict__ bits, uint32_t* keys, int* vals) {
    float blo[3], bhi[3];
    for (int k = 0; k < 3; ++k) {
        blo[k] = ordered_to_float(bits[k]);
        bhi[k] = ordered_to_float(bits[3 + k]);
    }
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float4 a = lo[i], b = hi[i];
        keys[i] = morton30((a.x + b.x) * 0.5f, (a.y + b.y) * 0.5f, (a.z + b.z) * 0.5f, blo, bhi);
        vals[i] = i;
    }
}

// Per-tile digit histogram (digit-major layout: hist[d * blocks + b]).
__global__ void __launch_bounds__(kSortThreads) k_sort_hist(const uint32_t* __restrict__ keys, int n, int shift,
    uint32_t* hist) {
    __shared__ uint32_t counts[kDigits];
    if (threadIdx.x < kDigits) counts[threadIdx.x] = 0;
    __syncthreads();
    const int base = blockIdx.x * kSortTile;
    for (int r = 0; r < kSortItems && base + r * kSortThreads < n; ++r) {
        const int i = base + r * kSortThreads + threadIdx.x;
        if (i < n) atomicAdd(&counts[(keys[i] >> shift) & (kDigits - 1)], 1u);
    }
    __syncthreads();
    if (threadIdx.x < kDigits) hist[threadIdx.x * gridDim.x + blockIdx.x] = counts[threadIdx.x];
}

// Exclusive scan of the digit-major histogram (one block, any length).
__global__ void __launch_bounds__(1024) k_sort_scan(uint32_t* hist, int len) {
    __shared__ uint32_t warp_sums[32];
    __shared__ uint32_t carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int base = 0; base < len; base += 1024) {
        const int i = base + threadIdx.x;
        const uint32_t v = i < len ? hist[i] : 0u;
        uint32_t x = v;
        for (int off = 1; off < 32; off <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, off);
            if ((threadIdx.x & 31) >= off) x += y;
        }
        if ((threadIdx.x & 31) == 31) warp_sums[threadIdx.x >> 5] = x;
        __syncthreads();
        if (threadIdx.x < 32) {
            uint32_t w = warp_sums[threadIdx.x];
            for (int off = 1; off < 32; off <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, w, off);
                if (threadIdx.x >= off) w += y;
            }
            warp_sums[threadIdx.x] = w;
        }
        __syncthreads();
        const uint32_t warp_prefix = (threadIdx.x >= 32) ? warp_sums[(threadIdx.x >> 5) - 1] : 0u;
        if (i < len) hist[i] = carry + warp_prefix + x - v;
        __syncthreads();
        if (threadIdx.x == 1023) carry += warp_prefix + x;
        __syncthreads();
    }
}

// Stable scatter: items of a tile are ranked in input order (round by round,
// warp by warp, lane by lane) with __match_any_sync.
__global__ void __launch_bounds__(kSortThreads) k_sort_scatter(const uint32_t* __restrict__ keys_in,
    const int* __restrict__ vals_in, int n, int shift, const uint32_t* __restrict__ hist, uint32_t* keys_out,
    int* vals_out) {
    constexpr int kWarps = kSortThreads / 32;
    __shared__ uint32_t running[kDigits];
    __shared__ uint32_t warp_counts[kWarps][kDigits];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x < kDigits) running[threadIdx.x] = hist[threadIdx.x * gridDim.x + blockIdx.x];
    const int base = blockIdx.x * kSortTile;
    for (int r = 0; r < kSortItems && base + r * kSortThreads < n; ++r) {
        for (int k = threadIdx.x; k < kWarps * kDigits; k += kSortThreads) (&warp_counts[0][0])[k] = 0;
        __syncthreads();
        const int i = base + r * kSortThreads + threadIdx.x;
        const bool valid = i < n;
        const uint32_t key = valid ? keys_in[i] : 0u;
        const int digit = valid ? static_cast<int>((key >> shift) & (kDigits - 1)) : kDigits;  // invalid: own group
        const unsigned int peers = __match_any_sync(0xffffffffu, digit);
        const int rank_in_warp = __popc(peers & ((1u << lane) - 1u));
        if (valid && rank_in_warp == 0) warp_counts[warp][digit] = __popc(peers);
        __syncthreads();
        if (valid) {
            uint32_t offset = running[digit];
            for (int w = 0; w < warp; ++w) offset += warp_counts[w][digit];
            const uint32_t dst = offset + static_cast<uint32_t>(rank_in_warp);
            keys_out[dst] = key;
            vals_out[dst] = vals_in[i];
        }
        __syncthreads();
        if (threadIdx.x < kDigits) {
            uint32_t total = 0;
            for (int w = 0; w < kWarps; ++w) total += warp_counts[w][threadIdx.x];
            running[threadIdx.x] += total;
        }
        __syncthreads();
    }
}

// Karras prefix length with index tie-break for equal keys.
RTGB_D int delta(const uint32_t* __restrict__ keys, int n, int i, int j) {
    if (j < 0 || j >= n) return -1;
    const uint32_t a = keys[i], b = keys[j];
    if (a == b) return 32 + __clz(static_cast<uint32_t>(i ^ j));
    return __clz(a ^ b);
}

__global__ void k_karras(const uint32_t* __restrict__ keys, int n, int* children, int* parent) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n - 1) return;
    const int d = (delta(keys, n, i, i + 1) - delta(keys, n, i, i - 1)) >= 0 ? 1 : -1;
    const int dmin = delta(keys, n, i, i - d);
    int lmax = 2;
    while (delta(keys, n, i, i + lmax * d) > dmin) lmax <<= 1;
    int l = 0;
    for (int t = lmax >> 1; t >= 1; t >>= 1) {
        if (delta(keys, n, i, i + (l + t) * d) > dmin) l += t;
    }
    const int j = i + l * d;
    const int dnode = delta(keys, n, i, j);
    int s = 0;
    int t = l;
    do {
        t = (t + 1) >> 1;
        if (delta(keys, n, i, i + (s + t) * d) > dnode) s += t;
    } while (t > 1);
    const int gamma = i + s * d + min(d, 0);
    const int lo = min(i, j), hi = max(i, j);
    const int left = (lo == gamma) ? ~gamma : gamma;            // leaf slot gamma or internal node gamma
    const int right = (hi == gamma + 1) ? ~(gamma + 1) : gamma + 1;
    children[2 * i] = left;
    children[2 * i + 1] = right;
    // parent[] holds internal parents for internal nodes [0, n-1) and leaves [n-1, 2n-1)
    parent[left >= 0 ? left : (n - 1 + ~left)] = i;
    parent[right >= 0 ? right : (n - 1 + ~right)] = i;
    if (i == 0) parent[0] = -1;
}

// Bottom-up bounds: each leaf walks to the root; the second arrival at a node
// unions both children and writes the node record.
__global__ void k_bounds(const float4* __restrict__ aabb_lo, const float4* __restrict__ aabb_hi,
    const int* __restrict__ sorted_vals, int n, const int* __restrict__ children, const int* __restrict__ parent,
    int* flags, float4* node_lo, float4* node_hi, BvhNode* nodes) {
    const int leaf = blockIdx.x * blockDim.x + threadIdx.x;
    if (leaf >= n) return;
    int node = parent[n - 1 + leaf];
    for (int guard = 0; guard < 2 * n && node >= 0; ++guard) {
        __threadfence();
        if (atomicAdd(flags + node, 1) == 0) return;  // first arrival: sibling finishes this node
        __threadfence();
        float4 lo[2], hi[2];
        for (int k = 0; k < 2; ++k) {
            const int c = children[2 * node + k];
            if (c < 0) {
                const int src = sorted_vals[~c];
                lo[k] = aabb_lo[src];
                hi[k] = aabb_hi[src];
            } else {
                lo[k] = __ldcg(node_lo + c);
                hi[k] = __ldcg(node_hi + c);
            }
        }
        const int c0 = children[2 * node], c1 = children[2 * node + 1];
        BvhNode out;
        out.a = make_float4(lo[0].x, lo[0].y, lo[0].z, __int_as_float(c0));
        out.b = make_float4(hi[0].x, hi[0].y, hi[0].z, __int_as_float(c1));
        out.c = make_float4(lo[1].x, lo[1].y, lo[1].z, 0.0f);
        out.d = make_float4(hi[1].x, hi[1].y, hi[1].z, 0.0f);
        nodes[node] = out;
        __stcg(node_lo + node, make_float4(fminf(lo[0].x, lo[1].x), fminf(lo[0].y, lo[1].y), fminf(lo[0].z, lo[1].z), 0.0f));
        __stcg(node_hi + node, make_float4(fmaxf(hi[0].x, hi[1].x), fmaxf(hi[0].y, hi[1].y), fmaxf(hi[0].z, hi[1].z), 0.0f));
        node = parent[node];
    }
}

}  // namespace

size_t lbvh_scratch_bytes(int n) {
    const size_t nn = static_cast<size_t>(std::max(n, 2));
    const size_t blocks = static_cast<size_t>(sort_blocks(static_cast<int>(nn)));
    size_t b = 0;
    b += 2 * align256(nn * sizeof(float4));          // aabb lo/hi
    b += 2 * align256(nn * sizeof(uint32_t));        // keys
    b += 2 * align256(nn * sizeof(int));             // vals
    b += align256(kDigits * blocks * sizeof(uint32_t));
    b += align256(2 * nn * sizeof(int));             // parent
    b += align256(nn * sizeof(int));                 // flags
    b += 2 * align256(nn * sizeof(float4));          // node bounds
    b += align256(2 * nn * sizeof(int));             // children
    b += align256(8 * sizeof(unsigned int));
    return b;
}

LbvhScratch lbvh_carve(void* base, int n) {
    const size_t nn = static_cast<size_t>(std::max(n, 2));
    const size_t blocks = static_cast<size_t>(sort_blocks(static_cast<int>(nn)));
    char* p = static_cast<char*>(base);
    auto take = [&](size_t bytes) {
        char* r = p;
        p += align256(bytes);
        return r;
    };
    LbvhScratch s;
    s.aabb_lo = reinterpret_cast<float4*>(take(nn * sizeof(float4)));
    s.aabb_hi = reinterpret_cast<float4*>(take(nn * sizeof(float4)));
    s.keys[0] = reinterpret_cast<uint32_t*>(take(nn * sizeof(uint32_t)));
    s.keys[1] = reinterpret_cast<uint32_t*>(take(nn * sizeof(uint32_t)));
    s.vals[0] = reinterpret_cast<int*>(take(nn * sizeof(int)));
    s.vals[1] = reinterpret_cast<int*>(take(nn * sizeof(int)));
    s.block_hist = reinterpret_cast<uint32_t*>(take(kDigits * blocks * sizeof(uint32_t)));
    s.parent = reinterpret_cast<int*>(take(2 * nn * sizeof(int)));
    s.flags = reinterpret_cast<int*>(take(nn * sizeof(int)));
    s.node_lo = reinterpret_cast<float4*>(take(nn * sizeof(float4)));
    s.node_hi = reinterpret_cast<float4*>(take(nn * sizeof(float4)));
    s.children = reinterpret_cast<int*>(take(2 * nn * sizeof(int)));
    s.bounds_bits = reinterpret_cast<unsigned int*>(take(8 * sizeof(unsigned int)));
    return s;
}

cudaError_t lbvh_build(LbvhScratch& s, int n, BvhNode* nodes, int** sorted_vals, uint32_t** sorted_keys,
    cudaStream_t stream) {
    if (n < 2) return cudaErrorInvalidValue;
    // An error left on this thread by earlier work is returned unchanged (and
    // not cleared) before anything is launched, so the launch check at the end
    // sees this build's launches only.
    if (const cudaError_t pending = cudaPeekAtLastError(); pending != cudaSuccess) return pending;
    const int threads = 256;
    const int grid = std::min((n + threads - 1) / threads, 4096);
    k_init_bounds<<<1, 32, 0, stream>>>(s.bounds_bits);
    k_centroid_bounds<<<grid, threads, 0, stream>>>(s.aabb_lo, s.aabb_hi, n, s.bounds_bits);
    k_morton<<<grid, threads, 0, stream>>>(s.aabb_lo, s.aabb_hi, n, s.bounds_bits, s.keys[0], s.vals[0]);
    const int blocks = sort_blocks(n);
    int cur = 0;
    for (int shift = 0; shift < 30; shift += 4) {
        k_sort_hist<<<blocks, kSortThreads, 0, stream>>>(s.keys[cur], n, shift, s.block_hist);
        k_sort_scan<<<1, 1024, 0, stream>>>(s.block_hist, kDigits * blocks);
        k_sort_scatter<<<blocks, kSortThreads, 0, stream>>>(s.keys[cur], s.vals[cur], n, shift, s.block_hist,
            s.keys[cur ^ 1], s.vals[cur ^ 1]);
        cur ^= 1;
    }
    k_karras<<<(n - 1 + threads - 1) / threads, threads, 0, stream>>>(s.keys[cur], n, s.children, s.parent);
    if (const cudaError_t e = cudaMemsetAsync(s.flags, 0, static_cast<size_t>(n) * sizeof(int), stream); e != cudaSuccess) {
        return e;
    }
    k_bounds<<<(n + threads - 1) / threads, threads, 0, stream>>>(s.aabb_lo, s.aabb_hi, s.vals[cur], n, s.children,
        s.parent, s.flags, s.node_lo, s.node_hi, nodes);
    *sorted_vals = s.vals[cur];
    *sorted_keys = s.keys[cur];
    return cudaGetLastError();
}

namespace {

// The collapse keeps the binary nodes of even depth (the root is depth 0) in
// breadth-first order: by depth, and within a depth from left to right, which
// is the order of their indices (a Karras node's index lies inside the leaf
// range it covers, and ranges of one depth are disjoint). So the numbering is
// one stable counting-sort pass over half depths.
constexpr int kLevels = 64;  // prefix lengths grow by at least one a step: depth <= 64, half depth <= 32

// Half the depth of each internal node, -1 at odd depths.
__global__ void k_half_depth(const int* __restrict__ parent, int nodes, int* __restrict__ level) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nodes) return;
    int d = 0;
    for (int p = parent[i]; p >= 0 && d < 2 * kLevels - 1; p = parent[p]) ++d;
    level[i] = (d & 1) != 0 ? -1 : d >> 1;
}

// Per-tile counts of each level (level-major), the word past them zeroed so
// that the scan leaves the total there.
__global__ void __launch_bounds__(kSortThreads) k_level_hist(const int* __restrict__ level, int nodes, uint32_t* hist) {
    __shared__ uint32_t counts[kLevels];
    if (threadIdx.x < kLevels) counts[threadIdx.x] = 0;
    __syncthreads();
    const int base = blockIdx.x * kSortTile;
    for (int r = 0; r < kSortItems && base + r * kSortThreads < nodes; ++r) {
        const int i = base + r * kSortThreads + threadIdx.x;
        if (i < nodes && level[i] >= 0) atomicAdd(&counts[level[i]], 1u);
    }
    __syncthreads();
    if (threadIdx.x < kLevels) hist[threadIdx.x * gridDim.x + blockIdx.x] = counts[threadIdx.x];
    if (blockIdx.x == 0 && threadIdx.x == 0) hist[kLevels * gridDim.x] = 0;
}

// The BVH4 number of every even-depth node (ranked in index order as
// k_sort_scatter ranks equal digits), -1 for the others.
__global__ void __launch_bounds__(kSortThreads) k_level_rank(const int* __restrict__ level, int nodes,
    const uint32_t* __restrict__ hist, int* __restrict__ number) {
    constexpr int kWarps = kSortThreads / 32;
    __shared__ uint32_t running[kLevels];
    __shared__ uint32_t warp_counts[kWarps][kLevels];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x < kLevels) running[threadIdx.x] = hist[threadIdx.x * gridDim.x + blockIdx.x];
    const int base = blockIdx.x * kSortTile;
    for (int r = 0; r < kSortItems && base + r * kSortThreads < nodes; ++r) {
        for (int k = threadIdx.x; k < kWarps * kLevels; k += kSortThreads) (&warp_counts[0][0])[k] = 0;
        __syncthreads();
        const int i = base + r * kSortThreads + threadIdx.x;
        const int l = i < nodes ? level[i] : -1;
        const unsigned int peers = __match_any_sync(0xffffffffu, l);
        const int rank = __popc(peers & ((1u << lane) - 1u));
        if (l >= 0 && rank == 0) warp_counts[warp][l] = __popc(peers);
        __syncthreads();
        if (i < nodes) {
            int id = -1;
            if (l >= 0) {
                uint32_t at = running[l];
                for (int w = 0; w < warp; ++w) at += warp_counts[w][l];
                id = static_cast<int>(at) + rank;
            }
            number[i] = id;
        }
        __syncthreads();
        if (threadIdx.x < kLevels) {
            uint32_t total = 0;
            for (int w = 0; w < kWarps; ++w) total += warp_counts[w][threadIdx.x];
            running[threadIdx.x] += total;
        }
        __syncthreads();
    }
}

// Children and box references of each BVH4 node: the binary node's children,
// an internal one replaced by its own two.
__global__ void k_write_bvh4(const int* __restrict__ children, const int* __restrict__ number, int nodes,
    int4* __restrict__ child4, int4* __restrict__ ref4) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nodes || number[i] < 0) return;
    int c4[4], r4[4];
    int slot = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        c4[k] = kEmptyChild;
        r4[k] = -1;
    }
    for (int k = 0; k < 2; ++k) {
        const int c = children[2 * i + k];
        for (int kk = 0; kk < 2; ++kk) {
            if (c < 0 && kk == 1) break;
            const int ref = c < 0 ? 2 * i + k : 2 * c + kk;
            const int g = c < 0 ? c : children[2 * c + kk];
            const int id = g < 0 ? g : number[g];
#pragma unroll
            for (int t = 0; t < 4; ++t) {  // registers: no dynamic indexing
                if (t == slot) {
                    c4[t] = id;
                    r4[t] = ref;
                }
            }
            ++slot;
        }
    }
    child4[number[i]] = make_int4(c4[0], c4[1], c4[2], c4[3]);
    ref4[number[i]] = make_int4(r4[0], r4[1], r4[2], r4[3]);
}

}  // namespace

size_t collapse_scratch_bytes(int n) {
    const size_t nn = static_cast<size_t>(std::max(n, 2));
    const size_t blocks = static_cast<size_t>(sort_blocks(static_cast<int>(nn)));
    return 2 * align256(nn * sizeof(int)) + align256((kLevels * blocks + 1) * sizeof(uint32_t));
}

cudaError_t number_bvh4(const int* parent, int n, void* scratch, const int** count, cudaStream_t stream) {
    if (n < 2) return cudaErrorInvalidValue;
    const int nodes = n - 1, blocks = sort_blocks(nodes), threads = 256;
    int* level = static_cast<int*>(scratch);
    int* number = reinterpret_cast<int*>(static_cast<char*>(scratch) + align256(static_cast<size_t>(n) * sizeof(int)));
    uint32_t* hist = reinterpret_cast<uint32_t*>(reinterpret_cast<char*>(number) + align256(static_cast<size_t>(n) * sizeof(int)));
    k_half_depth<<<(nodes + threads - 1) / threads, threads, 0, stream>>>(parent, nodes, level);
    k_level_hist<<<blocks, kSortThreads, 0, stream>>>(level, nodes, hist);
    k_sort_scan<<<1, 1024, 0, stream>>>(hist, kLevels * blocks + 1);
    k_level_rank<<<blocks, kSortThreads, 0, stream>>>(level, nodes, hist, number);
    *count = reinterpret_cast<const int*>(hist + static_cast<size_t>(kLevels) * blocks);
    return cudaGetLastError();
}

cudaError_t write_bvh4(const int* children, int n, const void* scratch, int* child4, int* ref4, cudaStream_t stream) {
    const int nodes = n - 1, threads = 256;
    const int* number = reinterpret_cast<const int*>(static_cast<const char*>(scratch) + align256(static_cast<size_t>(n) * sizeof(int)));
    k_write_bvh4<<<(nodes + threads - 1) / threads, threads, 0, stream>>>(children, number, nodes,
        reinterpret_cast<int4*>(child4), reinterpret_cast<int4*>(ref4));
    return cudaGetLastError();
}

namespace {

__global__ void k_fill_bvh4(const BvhNode* __restrict__ nodes2, const int* __restrict__ child4,
    const int* __restrict__ ref4, int n4, float4* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n4) return;
    float lo[3][4], hi[3][4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int r = ref4[4 * i + k];
        float4 a = make_float4(0.0f, 0.0f, 0.0f, 0.0f), b = a;
        if (r >= 0) {
            const BvhNode& nd = nodes2[r >> 1];
            a = (r & 1) ? nd.c : nd.a;
            b = (r & 1) ? nd.d : nd.b;
        }
        lo[0][k] = a.x; lo[1][k] = a.y; lo[2][k] = a.z;
        hi[0][k] = b.x; hi[1][k] = b.y; hi[2][k] = b.z;
    }
    float4* o = out + static_cast<long long>(kNode4) * i;
    for (int ax = 0; ax < 3; ++ax) {
        o[ax] = make_float4(lo[ax][0], lo[ax][1], lo[ax][2], lo[ax][3]);
        o[3 + ax] = make_float4(hi[ax][0], hi[ax][1], hi[ax][2], hi[ax][3]);
    }
    o[6] = make_float4(__int_as_float(child4[4 * i]), __int_as_float(child4[4 * i + 1]), __int_as_float(child4[4 * i + 2]),
        __int_as_float(child4[4 * i + 3]));
    o[7] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
}

}  // namespace

cudaError_t fill_bvh4(const BvhNode* nodes2, const int* child4, const int* ref4, int n4, float4* nodes4,
    cudaStream_t stream) {
    if (n4 <= 0) return cudaSuccess;
    k_fill_bvh4<<<(n4 + 127) / 128, 128, 0, stream>>>(nodes2, child4, ref4, n4, nodes4);
    return cudaGetLastError();
}

cudaError_t lbvh_refit(LbvhScratch& s, int n, const int* sorted_vals, const int* children, const int* parent,
    BvhNode* nodes, cudaStream_t stream) {
    if (n < 2) return cudaErrorInvalidValue;
    const int threads = 256;
    if (const cudaError_t e = cudaMemsetAsync(s.flags, 0, static_cast<size_t>(n) * sizeof(int), stream); e != cudaSuccess) {
        return e;
    }
    k_bounds<<<(n + threads - 1) / threads, threads, 0, stream>>>(s.aabb_lo, s.aabb_hi, sorted_vals, n, children,
        parent, s.flags, s.node_lo, s.node_hi, nodes);
    return cudaGetLastError();
}

}  // namespace rtgb
