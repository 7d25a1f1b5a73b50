// std::sort's exact permutation of (radius, voxel) items by descending radius, on the device.
//
// The reference orders its maximum balls with std::sort (PoreAndThroatComputer.cpp:121-122), and
// the order among equal radii decides seeds and pore ids. libstdc++'s std::sort is an introsort
// (Musser, "Introspective sorting and selection algorithms", 1997): ranges of more than 16 elements
// are partitioned (Hoare) around the median of their second, middle and last elements, a range
// that is 2 log2(n) partitions deep goes to a heap sort, and an insertion sort ends it; a
// comparator that records its calls shows which elements these are. Here the steps run in parallel:
//  * Partition of [first + 1, last) around the pivot P at first. The scan from the left stops at
//    elements that do not come before P, the scan from the right at elements that P does not come
//    before. With L_k and R_k the k-th stops from the two ends, the pairs with L_k < R_k, a prefix
//    k < m, change places, because the elements between the scans are still those of the start; then
//    the left scan ends the partition at the next stop L_m, or at R_{m-1} if that is nearer (it holds
//    an element from the left by then). So the stops and their ranks are prefix counts, m a search,
//    and the exchanges are independent of each other.
//  * The insertion sort is a stable sort of each range of at most 16 elements: no element comes
//    before an element of the ranges in front of its own, so none leaves its range.
// Ranges of more than kBlockSort elements are partitioned by the whole grid, all ranges of a depth
// at once; a block takes each smaller one through all its partitions in shared memory, a warp per
// subrange. A range that reaches the depth limit ends the call with false (the caller then sorts on
// the host with the library's own routines).
//
// What bounds it: the launches and the read-back of the large depths (six launches each), then in
// each block the first partitions, on one to eight warps. Measured: 1.8 ms for the maximum balls of
// a 512^3 random field, where the library's routines on 16 threads were waited for 30 ms behind
// the plateau kernels; 0.87 against 5 ms (spinodal 256^3); 0.1 ms for a few thousand balls.
#pragma once

#include <algorithm>
#include <mutex>
#include <vector>

#include "devutil.cuh"

namespace pma {
namespace {

constexpr uint32_t kLeaf = 16;          // libstdc++ partitions while more than this many are left
constexpr uint32_t kBlockSort = 8192;   // elements sorted by one block: 100 KB, two blocks an SM
constexpr int kBlockSortThreads = 512;
constexpr uint32_t kPartChunk = 2048;   // elements of a block of the large partitions
constexpr int kPartThreads = 256;
constexpr uint32_t kBlockList = kBlockSort / (kLeaf + 1) + 1;  // subranges above kLeaf at once

struct SortRange {
    uint32_t first, last, depth;  // partitions left before the heap sort
};

struct SortChunk {
    uint32_t range, from, to;
};

__device__ __forceinline__ uint32_t sort_key(unsigned long long v) { return static_cast<uint32_t>(v >> 32); }

// The median of the elements first + 1, middle, last - 1 changes places with the first. Descending
// order: x comes before y when its key is larger.
__device__ __forceinline__ void sort_median(unsigned long long* a, uint32_t first, uint32_t last) {
    const uint32_t ia = first + 1, ib = first + (last - first) / 2, ic = last - 1;
    const uint32_t ka = sort_key(a[ia]), kb = sort_key(a[ib]), kc = sort_key(a[ic]);
    uint32_t m;
    if (ka > kb) m = kb > kc ? ib : (ka > kc ? ic : ia);
    else m = ka > kc ? ia : (kb > kc ? ic : ib);
    const unsigned long long t = a[first];
    a[first] = a[m];
    a[m] = t;
}

__global__ void sort_pivots(unsigned long long* __restrict__ a, const SortRange* __restrict__ ranges, uint32_t n) {
    PMA_GRID_STRIDE(r, n) sort_median(a, ranges[r].first, ranges[r].last);
}

// Left and right stops of each chunk.
__global__ void __launch_bounds__(kPartThreads) sort_count(const unsigned long long* __restrict__ a, const SortRange* __restrict__ ranges,
                                                           const SortChunk* __restrict__ chunks, uint32_t* __restrict__ left,
                                                           uint32_t* __restrict__ right) {
    __shared__ uint32_t sl, sr;
    const SortChunk c = chunks[blockIdx.x];
    const uint32_t P = sort_key(a[ranges[c.range].first]);
    if (threadIdx.x == 0) sl = sr = 0;
    __syncthreads();
    uint32_t l = 0, r = 0;
    for (uint32_t i = c.from + threadIdx.x; i < c.to; i += kPartThreads) {
        const uint32_t k = sort_key(a[i]);
        l += k <= P ? 1u : 0u;
        r += k >= P ? 1u : 0u;
    }
    l = __reduce_add_sync(0xFFFFFFFFu, l);
    r = __reduce_add_sync(0xFFFFFFFFu, r);
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&sl, l);
        atomicAdd(&sr, r);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        left[blockIdx.x] = sl;
        right[blockIdx.x] = sr;
    }
}

// Per range: the stops before (left) and after (right) each of its chunks, and in all. One warp a range.
__global__ void sort_scan(const uint32_t* __restrict__ chunk0, uint32_t n, uint32_t* __restrict__ left, uint32_t* __restrict__ right,
                          uint2* __restrict__ total) {
    const unsigned lane = threadIdx.x & 31;
    const uint32_t r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (r >= n) return;
    const uint32_t c0 = chunk0[r], c1 = chunk0[r + 1];
    uint32_t l = 0, q = 0;
    for (uint32_t b = 0; b < c1 - c0; b += 32) {
        const bool in = b + lane < c1 - c0;
        const uint32_t cl = c0 + b + lane, cr = c1 - 1 - b - lane;
        const uint32_t vl = in ? left[cl] : 0u, vr = in ? right[cr] : 0u;
        uint32_t il = vl, ir = vr;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t tl = __shfl_up_sync(0xFFFFFFFFu, il, o), tr = __shfl_up_sync(0xFFFFFFFFu, ir, o);
            if (lane >= static_cast<unsigned>(o)) {
                il += tl;
                ir += tr;
            }
        }
        if (in) {
            left[cl] = l + il - vl;
            right[cr] = q + ir - vr;
        }
        l += __shfl_sync(0xFFFFFFFFu, il, 31);
        q += __shfl_sync(0xFFFFFFFFu, ir, 31);
    }
    if (lane == 0) total[r] = make_uint2(l, q);
}

// Positions of the stops by rank, at lpos / rpos [first + rank].
__global__ void __launch_bounds__(kPartThreads) sort_positions(const unsigned long long* __restrict__ a,
                                                               const SortRange* __restrict__ ranges, const SortChunk* __restrict__ chunks,
                                                               const uint32_t* __restrict__ left, const uint32_t* __restrict__ right,
                                                               uint32_t* __restrict__ lpos, uint32_t* __restrict__ rpos) {
    constexpr int kWarps = kPartThreads / 32, kRows = kPartChunk / kPartThreads;
    __shared__ uint32_t wl[kWarps], wr[kWarps];
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5, lt = (1u << lane) - 1u;
    const SortChunk c = chunks[blockIdx.x];
    const uint32_t first = ranges[c.range].first, P = sort_key(a[first]);
    unsigned ml[kRows], mr[kRows];
    uint32_t nl = 0, nr = 0;
#pragma unroll
    for (int r = 0; r < kRows; ++r) {  // a warp's rows are contiguous
        const uint32_t i = c.from + (warp * kRows + r) * 32 + lane;
        const uint32_t k = i < c.to ? sort_key(a[i]) : 0u;
        ml[r] = __ballot_sync(0xFFFFFFFFu, i < c.to && k <= P);
        mr[r] = __ballot_sync(0xFFFFFFFFu, i < c.to && k >= P);
        nl += __popc(ml[r]);
        nr += __popc(mr[r]);
    }
    if (lane == 0) {
        wl[warp] = nl;
        wr[warp] = nr;
    }
    __syncthreads();
    uint32_t l = first + left[blockIdx.x], q = first + right[blockIdx.x];
    for (unsigned w = 0; w < kWarps; ++w) {
        if (w < warp) l += wl[w];
        if (w > warp) q += wr[w];
    }
    q += nr;  // the warp's right stops are ranked from its last row down
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
        const uint32_t i = c.from + (warp * kRows + r) * 32 + lane;
        if ((ml[r] >> lane) & 1u) lpos[l + __popc(ml[r] & lt)] = i;
        l += __popc(ml[r]);
        q -= __popc(mr[r]);
        if ((mr[r] >> lane) & 1u) rpos[q + __popc(mr[r] & ~lt & ~(1u << lane))] = i;
    }
}

// Per range: the number m of swaps (pairs with L < R, a prefix of the ranks) and the cut. One warp a range.
__global__ void sort_cuts(const SortRange* __restrict__ ranges, uint32_t n, const uint2* __restrict__ total,
                          const uint32_t* __restrict__ lpos, const uint32_t* __restrict__ rpos, uint32_t* __restrict__ swaps,
                          uint32_t* __restrict__ cut) {
    const unsigned lane = threadIdx.x & 31;
    const uint32_t r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (r >= n) return;
    const SortRange g = ranges[r];
    const uint2 t = total[r];
    const uint32_t* L = lpos + g.first;
    const uint32_t* R = rpos + g.first;
    uint32_t lo = 0, hi = min(t.x, t.y);  // pairs [0, lo) are swapped, pair hi is not (or does not exist)
    while (lo < hi) {
        const uint32_t step = (hi - lo + 31) / 32, k = lo + lane * step;
        const unsigned yes = __ballot_sync(0xFFFFFFFFu, k < hi && L[k] < R[k]);
        const uint32_t c = __popc(yes);  // lanes 0 .. c - 1
        if (c == 0) {
            hi = lo;
        } else {
            const uint32_t from = lo;
            lo = from + (c - 1) * step + 1;
            hi = min(hi, from + c * step);
        }
    }
    if (lane == 0) {
        const uint32_t last_r = lo ? R[lo - 1] : g.last;
        swaps[r] = lo;
        cut[r] = lo < t.x && L[lo] < last_r ? L[lo] : last_r;
    }
}

__global__ void __launch_bounds__(kPartThreads) sort_swap(unsigned long long* __restrict__ a, const SortRange* __restrict__ ranges,
                                                          const SortChunk* __restrict__ chunks, const uint32_t* __restrict__ swaps,
                                                          const uint32_t* __restrict__ lpos, const uint32_t* __restrict__ rpos) {
    const SortChunk c = chunks[blockIdx.x];
    const uint32_t first = ranges[c.range].first, m = swaps[c.range];
    const uint32_t k1 = min(c.to - first - 1, m);  // the chunk's share of the ranks
    for (uint32_t k = c.from - first - 1 + threadIdx.x; k < k1; k += kPartThreads) {
        const uint32_t i = lpos[first + k], j = rpos[first + k];
        const unsigned long long t = a[i];
        a[i] = a[j];
        a[j] = t;
    }
}

struct BlockSortShared {
    unsigned long long a[kBlockSort];
    uint16_t lpos[kBlockSort], rpos[kBlockSort];
    uint32_t range[2][kBlockList];  // first | last << 16
    uint32_t count[2];
};

// Stable sort of at most kLeaf elements by one warp.
__device__ __forceinline__ void sort_leaf(unsigned long long* a, uint32_t first, uint32_t last) {
    const unsigned lane = threadIdx.x & 31;
    const uint32_t n = last - first;
    const unsigned long long v = lane < n ? a[first + lane] : 0ull;
    uint32_t rank = 0;
    for (uint32_t j = 0; j < n; ++j) {
        const uint32_t k = __shfl_sync(0xFFFFFFFFu, sort_key(v), j);
        rank += k > sort_key(v) || (k == sort_key(v) && j < lane) ? 1u : 0u;
    }
    __syncwarp();
    if (lane < n) a[first + rank] = v;
    __syncwarp();
}

// One warp partitions [first, last); returns the cut.
__device__ __forceinline__ uint32_t sort_partition(BlockSortShared& sh, uint32_t first, uint32_t last) {
    const unsigned lane = threadIdx.x & 31, lt = (1u << lane) - 1u;
    if (lane == 0) sort_median(sh.a, first, last);
    __syncwarp();
    const uint32_t P = sort_key(sh.a[first]);
    uint32_t nl = 0, nr = 0;
    for (uint32_t b = 0; b < last - first - 1; b += 32) {
        const bool in = b + lane < last - first - 1;
        const uint32_t i = first + 1 + b + lane, j = last - 1 - b - lane;
        const bool l = in && sort_key(sh.a[i]) <= P, r = in && sort_key(sh.a[j]) >= P;
        const unsigned ml = __ballot_sync(0xFFFFFFFFu, l), mr = __ballot_sync(0xFFFFFFFFu, r);
        if (l) sh.lpos[first + nl + __popc(ml & lt)] = static_cast<uint16_t>(i);
        if (r) sh.rpos[first + nr + __popc(mr & lt)] = static_cast<uint16_t>(j);
        nl += __popc(ml);
        nr += __popc(mr);
    }
    __syncwarp();
    const uint32_t pairs = min(nl, nr);
    uint32_t m = 0;
    for (uint32_t b = 0; b < pairs; b += 32) {
        uint32_t i = 0, j = 0;
        if (b + lane < pairs) {
            i = sh.lpos[first + b + lane];
            j = sh.rpos[first + b + lane];
        }
        const unsigned yes = __ballot_sync(0xFFFFFFFFu, i < j);
        if (i < j) {
            const unsigned long long t = sh.a[i];
            sh.a[i] = sh.a[j];
            sh.a[j] = t;
        }
        m += __popc(yes);
        if (yes != 0xFFFFFFFFu) break;
    }
    __syncwarp();
    const uint32_t last_r = m ? sh.rpos[first + m - 1] : last;
    return m < nl && sh.lpos[first + m] < last_r ? sh.lpos[first + m] : last_r;
}

// A block per range of at most kBlockSort elements: all its partitions, level by level, and leaves.
__global__ void __launch_bounds__(kBlockSortThreads) sort_block(unsigned long long* __restrict__ items, const SortRange* __restrict__ ranges,
                                                                unsigned int* __restrict__ failed) {
    extern __shared__ __align__(16) unsigned char dynamic[];
    BlockSortShared& sh = *reinterpret_cast<BlockSortShared*>(dynamic);
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = kBlockSortThreads / 32;
    const SortRange g = ranges[blockIdx.x];
    const uint32_t n = g.last - g.first;
    for (uint32_t i = threadIdx.x; i < n; i += kBlockSortThreads) sh.a[i] = items[g.first + i];
    if (threadIdx.x == 0) {
        sh.count[0] = n > kLeaf ? 1u : 0u;
        sh.range[0][0] = n << 16;
    }
    __syncthreads();
    if (n <= kLeaf && warp == 0) sort_leaf(sh.a, 0, n);
    int side = 0;
    uint32_t depth = g.depth;
    for (; sh.count[side]; side ^= 1, --depth) {
        const uint32_t k = sh.count[side];
        if (depth == 0) {  // a heap sort would follow
            if (threadIdx.x == 0) atomicExch(failed, 1u);
            break;
        }
        __syncthreads();
        if (threadIdx.x == 0) sh.count[side ^ 1] = 0;
        __syncthreads();
        for (uint32_t q = warp; q < k; q += warps) {
            const uint32_t first = sh.range[side][q] & 0xFFFFu, last = sh.range[side][q] >> 16;
            const uint32_t cut = sort_partition(sh, first, last);
#pragma unroll
            for (int part = 0; part < 2; ++part) {
                const uint32_t f = part ? cut : first, l = part ? last : cut;
                if (l - f <= kLeaf) sort_leaf(sh.a, f, l);
                else if (lane == 0) sh.range[side ^ 1][atomicAdd(&sh.count[side ^ 1], 1u)] = f | l << 16;
            }
        }
        __syncthreads();
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < n; i += kBlockSortThreads) items[g.first + i] = sh.a[i];
}

// Sorts n < 2^32 items in place; false when a range reached the depth limit (the items are then in no
// particular order). lpos and rpos are n words of scratch each.
inline bool ordered_sort_device(pma_ctx* ctx, unsigned long long* items, int64_t n, uint32_t* lpos, uint32_t* rpos) {
    if (n < 2) return true;
    cudaStream_t s = ctx->stream;
    {
        static std::mutex mutex;  // the limit is a process-wide attribute of the kernel: once per device
        static std::vector<int> devices;
        int dev = 0;
        PMA_CUDA(cudaGetDevice(&dev));
        std::lock_guard<std::mutex> lock(mutex);
        if (std::find(devices.begin(), devices.end(), dev) == devices.end()) {
            PMA_CUDA(cudaFuncSetAttribute(sort_block, cudaFuncAttributeMaxDynamicSharedMemorySize, sizeof(BlockSortShared)));
            devices.push_back(dev);
        }
    }
    auto scratch = [&](const char* tag, size_t bytes) { return ctx->scratch(tag, std::max<size_t>(bytes, 16)); };
    uint32_t log2n = 0;
    while ((n >> (log2n + 1)) != 0) ++log2n;
    std::vector<SortRange> large, small, next;
    std::vector<SortChunk> chunks;
    std::vector<uint32_t> chunk0, cuts;
    auto sort_out = [&](uint32_t first, uint32_t last, uint32_t depth, std::vector<SortRange>& to) {
        if (last - first > kBlockSort) to.push_back({first, last, depth});
        else if (last - first > 1) small.push_back({first, last, depth});
    };
    sort_out(0, static_cast<uint32_t>(n), 2 * log2n, large);
    while (!large.empty()) {
        chunks.clear();
        chunk0.assign(1, 0);
        for (uint32_t r = 0; r < large.size(); ++r) {
            if (large[r].depth == 0) return false;
            for (uint32_t f = large[r].first + 1; f < large[r].last; f += std::min(kPartChunk, large[r].last - f))
                chunks.push_back({r, f, std::min(f + std::min(kPartChunk, large[r].last - f), large[r].last)});
            chunk0.push_back(static_cast<uint32_t>(chunks.size()));
        }
        const uint32_t nr = static_cast<uint32_t>(large.size()), nc = static_cast<uint32_t>(chunks.size());
        auto* d_ranges = static_cast<SortRange*>(scratch("sort.ranges", nr * sizeof(SortRange)));
        auto* d_chunks = static_cast<SortChunk*>(scratch("sort.chunks", nc * sizeof(SortChunk)));
        auto* d_chunk0 = static_cast<uint32_t*>(scratch("sort.chunk0", (nr + 1) * 4ull));
        auto* d_left = static_cast<uint32_t*>(scratch("sort.left", nc * 4ull));
        auto* d_right = static_cast<uint32_t*>(scratch("sort.right", nc * 4ull));
        auto* d_total = static_cast<uint2*>(scratch("sort.total", nr * sizeof(uint2)));
        auto* d_swaps = static_cast<uint32_t*>(scratch("sort.swaps", nr * 4ull));
        auto* d_cut = static_cast<uint32_t*>(scratch("sort.cut", nr * 4ull));
        PMA_CUDA(cudaMemcpyAsync(d_ranges, large.data(), nr * sizeof(SortRange), cudaMemcpyHostToDevice, s));
        PMA_CUDA(cudaMemcpyAsync(d_chunks, chunks.data(), nc * sizeof(SortChunk), cudaMemcpyHostToDevice, s));
        PMA_CUDA(cudaMemcpyAsync(d_chunk0, chunk0.data(), (nr + 1) * 4ull, cudaMemcpyHostToDevice, s));
        sort_pivots<<<div_up(nr, 128), 128, 0, s>>>(items, d_ranges, nr);
        sort_count<<<nc, kPartThreads, 0, s>>>(items, d_ranges, d_chunks, d_left, d_right);
        sort_scan<<<div_up(nr, 4), 128, 0, s>>>(d_chunk0, nr, d_left, d_right, d_total);
        sort_positions<<<nc, kPartThreads, 0, s>>>(items, d_ranges, d_chunks, d_left, d_right, lpos, rpos);
        sort_cuts<<<div_up(nr, 4), 128, 0, s>>>(d_ranges, nr, d_total, lpos, rpos, d_swaps, d_cut);
        sort_swap<<<nc, kPartThreads, 0, s>>>(items, d_ranges, d_chunks, d_swaps, lpos, rpos);
        ctx->count_launch(5);
        ctx->check_launch("sort_partition");
        cuts.resize(nr);
        PMA_CUDA(cudaMemcpyAsync(cuts.data(), d_cut, nr * 4ull, cudaMemcpyDeviceToHost, s));
        ctx->sync();
        next.clear();
        for (uint32_t r = 0; r < nr; ++r) {
            const SortRange g = large[r];
            PMA_REQUIRE(cuts[r] > g.first && cuts[r] < g.last, PMA_ERR_INTERNAL, "pma_pores: a partition left its range");
            sort_out(g.first, cuts[r], g.depth - 1, next);
            sort_out(cuts[r], g.last, g.depth - 1, next);
        }
        large.swap(next);
    }
    auto* failed = static_cast<unsigned int*>(scratch("sort.failed", 4));
    PMA_CUDA(cudaMemsetAsync(failed, 0, 4, s));
    auto* d_small = static_cast<SortRange*>(scratch("sort.small", small.size() * sizeof(SortRange)));
    PMA_CUDA(cudaMemcpyAsync(d_small, small.data(), small.size() * sizeof(SortRange), cudaMemcpyHostToDevice, s));
    if (!small.empty()) {
        sort_block<<<static_cast<unsigned>(small.size()), kBlockSortThreads, sizeof(BlockSortShared), s>>>(items, d_small, failed);
        ctx->check_launch("sort_block");
    }
    auto* h = static_cast<unsigned int*>(ctx->host_staging(64));
    ReadBack rb;
    rb.add(h, failed, 4);
    read_back(ctx, rb);
    return h[0] == 0;
}

}  // namespace
}  // namespace pma
