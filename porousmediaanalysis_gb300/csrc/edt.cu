// Squared Euclidean distance transform (EuclideanDistanceComputer.cpp:149-343).
//
// The reference runs a two-scan along X with virtual solids at x = -SX and x = 2SX-1
// (BOUNDARIES_ARE_SOLID = false), then brute-force windowed minima along Y and along Z.
// Both windowed minima compute exactly h(y) = min_{y'} g(y') + (y - y')^2, so any exact
// 1-D minimisation gives identical integers. Here:
//   pass X: columns packed into bitmasks in shared memory; the nearest solid on both sides is
//           read off the bits, and the distance (not its square) goes out in 16 bits, into the
//           first half of the voxel's row of the result. HBM: 1 B read + 2 B written per voxel.
//   pass Y: a block per eight rows; reads their distances, writes squares over them. 2 B + 4 B.
//   pass Z: tiles of 16 consecutive y by all z staged in shared memory, fused with the running
//           maximum and the histogram of balls that do not cross the image boundary
//           (EDC.cpp:310-327). 4 B + 4 B.
// In passes Y and Z a thread takes eight consecutive outputs and walks outward from them, two
// inputs a step (one add-and-minimum per output and input), until the squared distance of the
// step reaches the warp's largest minimum. An input past the end of the line is replaced by the
// last one: it then counts with a distance larger than its own, which never lowers a minimum.
// What bounds them: instructions, about two per output and step, as many steps as the largest
// distance of the warp's outputs. 1024^3 spinodal, before (32-bit squares throughout, one output
// a thread, both inputs read again for each) and after, ms: X 2.3 -> 1.2, Y 8.0 -> 5.1,
// Z 10.9 -> 4.6 (1.9 TB/s).
// Extents for which a square or a sum could pass 2^32 go through the general kernels.
#include <algorithm>
#include <mutex>
#include <vector>

#include "devutil.cuh"

namespace pma {
namespace {

constexpr int kHistSmall = 2048;  // histogram bins kept in shared memory per block

// ---------------------------------------------------------------------------------------
// General passes (any extents): one output a thread, 32-bit squares throughout.
// ---------------------------------------------------------------------------------------
__global__ void edt_general_x(const uint8_t* __restrict__ solid, uint32_t* __restrict__ g, int SX,
                           int SY, int SZ, int words) {
    extern __shared__ uint32_t bits[];  // [words][blockDim.x]
    const int col = blockIdx.x * blockDim.x + threadIdx.x;  // over SY * SZ columns
    const int ncols = SY * SZ;
    const bool active = col < ncols;
    const int y = active ? col % SY : 0;
    const int z = active ? col / SY : 0;
    const size_t base = static_cast<size_t>(z) * SX * SY + y;
    const int T = blockDim.x;
    uint32_t* mybits = bits + threadIdx.x;

    // Forward: pack solid flags, 32 rows per word. Loads of a word are independent.
    for (int w = 0; w < words; ++w) {
        uint32_t word = 0;
        if (active) {
            const int x0 = w * 32;
            const int n = min(32, SX - x0);
            uint8_t v[32];
#pragma unroll
            for (int i = 0; i < 32; ++i)
                v[i] = (i < n) ? __ldg(solid + base + static_cast<size_t>(x0 + i) * SY) : 0;
#pragma unroll
            for (int i = 0; i < 32; ++i) word |= (v[i] != 0 ? 1u : 0u) << i;
        }
        mybits[w * T] = word;
    }
    if (!active) return;

    // Backward: nearest solid at or after x (running) and at or before x (bit search).
    int next_solid = -1;  // -1: none yet (virtual solid at 2SX-1)
    int prev_solid = -2;  // -2: not searched yet
    for (int x = SX - 1; x >= 0; --x) {
        const uint32_t word = mybits[(x >> 5) * T];
        const bool s = (word >> (x & 31)) & 1u;
        uint32_t out;
        if (s) {
            next_solid = x;
            prev_solid = x;
            out = 0;
        } else {
            if (prev_solid == -2 || prev_solid > x) {
                // highest set bit at index <= x
                int wi = x >> 5;
                uint32_t m = word & (0xFFFFFFFFu >> (31 - (x & 31)));
                prev_solid = -1;
                while (true) {
                    if (m) {
                        prev_solid = wi * 32 + 31 - __clz(m);
                        break;
                    }
                    if (--wi < 0) break;
                    m = mybits[wi * T];
                }
            }
            const uint32_t dl = prev_solid >= 0 ? static_cast<uint32_t>(x - prev_solid)
                                                : static_cast<uint32_t>(x + SX);
            const uint32_t dr = next_solid >= 0 ? static_cast<uint32_t>(next_solid - x)
                                                : static_cast<uint32_t>(2 * SX - 1 - x);
            const uint32_t dmin = dl < dr ? dl : dr;
            out = dmin * dmin;
        }
        g[base + static_cast<size_t>(x) * SY] = out;
    }
}

// Exact 1-D lower envelope at position i of a staged line: min_j f[j] + (i-j)^2.
__device__ __forceinline__ uint32_t scan_line(const uint32_t* f, int stride, int n, int i) {
    uint32_t best = f[i * stride];
    if (best == 0) return 0;
    for (int d = 1;; ++d) {
        const uint32_t dd = static_cast<uint32_t>(d) * static_cast<uint32_t>(d);
        if (dd >= best) break;
        if (i - d >= 0) {
            const uint32_t c = f[(i - d) * stride] + dd;
            best = c < best ? c : best;
        }
        if (i + d < n) {
            const uint32_t c = f[(i + d) * stride] + dd;
            best = c < best ? c : best;
        }
        if (i - d < 0 && i + d >= n) break;
    }
    return best;
}

// One warp per row of SY elements.
__global__ void edt_general_y(uint32_t* __restrict__ g, int SY, size_t nrows) {
    extern __shared__ uint32_t rows[];  // [warps][SY]
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int warps = blockDim.x >> 5;
    uint32_t* line = rows + static_cast<size_t>(warp) * SY;
    for (size_t r = static_cast<size_t>(blockIdx.x) * warps + warp; r < nrows;
         r += static_cast<size_t>(gridDim.x) * warps) {
        uint32_t* p = g + r * SY;
        for (int i = lane; i < SY; i += 32) line[i] = p[i];
        __syncwarp();
        for (int i = lane; i < SY; i += 32) p[i] = scan_line(line, 1, SY, i);
        __syncwarp();
    }
}

// With maximum and histogram.
constexpr int kTileY = 16;

__global__ void edt_general_z(uint32_t* __restrict__ g, int SX, int SY, int SZ,
                           unsigned long long* __restrict__ hist, size_t hist_len,
                           unsigned int* __restrict__ max_out) {
    extern __shared__ uint32_t smem[];
    uint32_t* tile = smem;                                  // [SZ][kTileY]
    unsigned int* h_small = smem + static_cast<size_t>(SZ) * kTileY;  // [kHistSmall]
    const int tiles_y = (SY + kTileY - 1) / kTileY;
    const int x = blockIdx.x / tiles_y;
    const int y0 = (blockIdx.x % tiles_y) * kTileY;
    const int ny = min(kTileY, SY - y0);
    const size_t plane = static_cast<size_t>(SX) * SY;
    const size_t base = static_cast<size_t>(x) * SY + y0;

    for (int i = threadIdx.x; i < kHistSmall; i += blockDim.x) h_small[i] = 0;
    for (int i = threadIdx.x; i < SZ * kTileY; i += blockDim.x) {
        const int z = i / kTileY, yy = i % kTileY;
        tile[i] = (yy < ny) ? g[base + z * plane + yy] : 0;
    }
    __syncthreads();

    unsigned int local_max = 0;
    const int mx = min(x, SX - 1 - x);
    for (int i = threadIdx.x; i < SZ * kTileY; i += blockDim.x) {
        const int z = i / kTileY, yy = i % kTileY;
        if (yy >= ny) continue;
        const uint32_t e = scan_line(tile + yy, kTileY, SZ, z);
        g[base + z * plane + yy] = e;
        if (e == 0) continue;
        local_max = e > local_max ? e : local_max;
        const int y = y0 + yy;
        int m = min(mx, min(min(y, SY - 1 - y), min(z, SZ - 1 - z)));
        // e <= m^2 <=> the ball of radius sqrt(e) stays inside the image (EDC.cpp:316-327).
        if (static_cast<unsigned long long>(e) <= static_cast<unsigned long long>(m) * m) {
            if (e < kHistSmall) atomicAdd(&h_small[e], 1u);
            else if (e < hist_len) atomicAdd(&hist[e], 1ull);
        }
    }
    // block maximum
    for (int o = 16; o > 0; o >>= 1) {
        unsigned int v = __shfl_xor_sync(0xFFFFFFFFu, local_max, o);
        local_max = v > local_max ? v : local_max;
    }
    if ((threadIdx.x & 31) == 0 && local_max) atomicMax(max_out, local_max);
    __syncthreads();
    for (int i = threadIdx.x; i < kHistSmall && i < static_cast<int>(hist_len); i += blockDim.x)
        if (h_small[i]) atomicAdd(&hist[i], static_cast<unsigned long long>(h_small[i]));
}

// ---------------------------------------------------------------------------------------
// Pass X: V adjacent columns a thread (V = 4: 4-byte loads, 8-byte stores).
// ---------------------------------------------------------------------------------------
constexpr int kXThreads = 128;

template <int V>
__global__ void __launch_bounds__(kXThreads) edt_pass_x(const uint8_t* __restrict__ solid, uint32_t* __restrict__ g,
                                                        int SX, int SY, int SZ, int words,
                                                        unsigned long long* __restrict__ clear, size_t nclear) {
    extern __shared__ uint32_t bits[];  // [word][column of the thread][thread]
    const size_t tid = blockIdx.x * static_cast<size_t>(kXThreads) + threadIdx.x;
    for (size_t i = tid; i < nclear; i += static_cast<size_t>(gridDim.x) * kXThreads) clear[i] = 0;  // pass Z's statistics
    const int per_row = SY / V;
    if (tid >= static_cast<size_t>(per_row) * SZ) return;
    const int z = static_cast<int>(tid / per_row);
    const int y = static_cast<int>(tid - static_cast<size_t>(z) * per_row) * V;
    const size_t row0 = static_cast<size_t>(z) * SX;
    const uint8_t* in = solid + row0 * SY + y;
    uint32_t* mine = bits + threadIdx.x;
    for (int w = 0; w < words; ++w) {  // 32 rows a word, their loads in flight together
        const int n = min(32, SX - w * 32);
        uint32_t word[V];
#pragma unroll
        for (int c = 0; c < V; ++c) word[c] = 0;
        uint32_t v[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) {
            const uint8_t* p = in + static_cast<size_t>(w * 32 + i) * SY;
            v[i] = i >= n ? 0u : V == 4 ? __ldg(reinterpret_cast<const uint32_t*>(p)) : __ldg(p);
        }
#pragma unroll
        for (int i = 0; i < 32; ++i)
#pragma unroll
            for (int c = 0; c < V; ++c) word[c] |= ((v[i] >> (8 * c)) & 0xFFu ? 1u : 0u) << i;
#pragma unroll
        for (int c = 0; c < V; ++c) mine[(w * V + c) * kXThreads] = word[c];
    }
    // Words from the last to the first. after[c]: the nearest solid row behind the word (virtual at
    // 2 SX - 1), before[c]: the nearest in front of it (virtual at -SX), searched when it is needed.
    int after[V], before[V];
    bool known[V];
#pragma unroll
    for (int c = 0; c < V; ++c) {
        after[c] = 2 * SX - 1;
        before[c] = -SX;
        known[c] = false;
    }
    for (int w = words - 1; w >= 0; --w) {
        uint32_t word[V];
#pragma unroll
        for (int c = 0; c < V; ++c) {
            word[c] = mine[(w * V + c) * kXThreads];
            // the last solid row of an earlier word: still the same while no solid word was passed
            if (!known[c] || before[c] >= w * 32) {
                known[c] = true;
                before[c] = -SX;
                for (int q = w - 1; q >= 0; --q) {
                    const uint32_t b = mine[(q * V + c) * kXThreads];
                    if (b) {
                        before[c] = q * 32 + 31 - __clz(b);
                        break;
                    }
                }
            }
        }
        const int n = min(32, SX - w * 32);
#pragma unroll 4
        for (int i = n - 1; i >= 0; --i) {
            const int x = w * 32 + i;
            uint32_t d[V];
#pragma unroll
            for (int c = 0; c < V; ++c) {
                const uint32_t at_or_before = word[c] << (31 - i), at_or_after = word[c] >> i;
                const int p = at_or_before ? x - __clz(at_or_before) : before[c];
                const int q = at_or_after ? x + __ffs(at_or_after) - 1 : after[c];
                d[c] = static_cast<uint32_t>(min(x - p, q - x));
            }
            uint16_t* out = reinterpret_cast<uint16_t*>(g + (row0 + x) * SY) + y;
            if (V == 4) {
                *reinterpret_cast<uint2*>(out) = make_uint2(d[0] | (d[1 % V] << 16), d[2 % V] | (d[3 % V] << 16));
            } else {
                *out = static_cast<uint16_t>(d[0]);
            }
        }
#pragma unroll
        for (int c = 0; c < V; ++c)
            if (word[c]) after[c] = w * 32 + __ffs(word[c]) - 1;
    }
}

// ---------------------------------------------------------------------------------------
// The outward walk: outputs i0 .. i0 + 7 of a line of n inputs, f(j) = input j for 0 <= j < n.
// live: outputs that exist. All 32 lanes call.
// ---------------------------------------------------------------------------------------
constexpr int kOut = 8;

template <class F>
__device__ __forceinline__ void walk_line(F f, int n, int i0, int live, uint32_t* best) {
    uint32_t c[kOut];
#pragma unroll
    for (int k = 0; k < kOut; ++k) c[k] = f(min(i0 + k, n - 1));
#pragma unroll
    for (int k = 0; k < kOut; ++k) {
        best[k] = k < live ? c[k] : 0u;
#pragma unroll
        for (int q = 0; q < kOut; ++q)
            if (q != k) best[k] = __viaddmin_u32(c[q], static_cast<uint32_t>((k - q) * (k - q)), best[k]);
    }
    for (int t = 1; t < n; t += 2) {
        uint32_t most = best[0];
#pragma unroll
        for (int k = 1; k < kOut; ++k) most = max(most, best[k]);
        if (!__any_sync(0xFFFFFFFFu, static_cast<uint32_t>(t) * static_cast<uint32_t>(t) < most)) break;
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int s = t + u;
            const uint32_t a = f(max(i0 - s, 0)), b = f(min(i0 + kOut - 1 + s, n - 1));
#pragma unroll
            for (int k = 0; k < kOut; ++k) {
                const uint32_t da = static_cast<uint32_t>((s + k) * (s + k));
                const uint32_t db = static_cast<uint32_t>((s + kOut - 1 - k) * (s + kOut - 1 - k));
                best[k] = __viaddmin_u32(a, da, best[k]);
                best[k] = __viaddmin_u32(b, db, best[k]);
            }
        }
    }
}

// ---------------------------------------------------------------------------------------
// Pass Y: a block takes as many rows as it has warps (eight, fewer where the rows are long), a warp a
// stretch of all of them: 32 y of eight rows, not 256 y of one, because the longest walk of the warp
// counts for all its lanes, and near outputs are alike (spinodal of wavelength 48: 16.3 steps on average,
// not 24.5; 5.9 -> 5.1 ms). The rows' distances lie in shared memory with two elements skipped after every
// eight and rows 4 (mod 8) words apart, so that the lanes' inputs fall on different banks.
// Walks on 16-bit pairs (6.2 ms) and on floats with three-input minima (4.8, but pass Z 4.9) gave nothing.
// ---------------------------------------------------------------------------------------
constexpr int kYPad = kOut + 1;  // outputs of a lane, staged for coalesced stores

__global__ void edt_pass_y(uint32_t* __restrict__ g, int SY, size_t nrows, int row_words) {
    extern __shared__ uint32_t smem[];  // per warp: row_words words of distances; then 32 * kYPad outputs
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5, wb = __ffs(warps) - 1;
    const int per_row = 32 >> wb, span = per_row * kOut;  // lanes and outputs of a row in a warp's stretch
    const int mine = lane >> (5 - wb);
    uint32_t* dist = smem + static_cast<size_t>(warp) * row_words;
    uint32_t* stage = smem + static_cast<size_t>(warps) * row_words + warp * (32 * kYPad);
    const uint16_t* d16 = reinterpret_cast<const uint16_t*>(smem + static_cast<size_t>(mine) * row_words);
    auto f = [&](int j) {
        const uint32_t d = d16[j + 2 * (j / kOut)];
        return d * d;
    };
    for (size_t r0 = static_cast<size_t>(blockIdx.x) * warps; r0 < nrows; r0 += static_cast<size_t>(gridDim.x) * warps) {
        uint32_t* rows = g + r0 * SY;
        if (r0 + warp < nrows)
            for (int i = lane; i < (SY + 1) / 2; i += 32) dist[i + 2 * i / kOut] = rows[static_cast<size_t>(warp) * SY + i];
        __syncthreads();
        for (int y0 = warp * span; y0 < SY; y0 += warps * span) {
            const int i0 = y0 + (lane - mine * per_row) * kOut;
            uint32_t best[kOut];
            walk_line(f, SY, min(i0, SY - 1), r0 + mine < nrows ? min(max(SY - i0, 0), kOut) : 0, best);
#pragma unroll
            for (int k = 0; k < kOut; ++k) stage[lane * kYPad + k] = best[k];
            __syncwarp();
#pragma unroll
            for (int k = 0; k < kOut; ++k) {
                const int i = k * 32 + lane, row = i >> (8 - wb), y = y0 + i - row * span;
                if (y < SY && r0 + row < nrows) rows[static_cast<size_t>(row) * SY + y] = stage[i + i / kOut];
            }
            __syncwarp();
        }
        __syncthreads();  // before the next rows are staged
    }
}

// ---------------------------------------------------------------------------------------
// Pass Z with maximum and histogram. pitch: 18 words a z-slice of the tile (the two halves of a
// warp are eight slices apart: 144 words, other banks), 16 where that does not fit.
// Up to kZShort slices 128 threads a block, which cover 64 slices at once (512 would mostly be idle), and
// short_bins of the histogram in shared memory, as many as the extents allow (balls that do not cross
// the boundary): clearing 2048 for 16 lines of a few voxels was as much again. 1000 x 1000 planes, solid
// 1 %, ms with 512 threads / 128: 2 planes 0.33 / 0.08, 7 0.39 / 0.11, 64 0.53 / 0.30, 128 0.68 / 0.41 (one
// output a thread: 0.12, 0.17, 0.40, 0.68). Longer lines take so much shared memory that few blocks fit
// an SM: 700 x 700 spinodals of 300 planes 0.75 / 0.67, 512 1.03 / 1.16, 1024 2.17 / 3.98.
// ---------------------------------------------------------------------------------------
constexpr int kZShort = 128;

template <int kZThreads>
__global__ void __launch_bounds__(kZThreads) edt_pass_z(uint32_t* __restrict__ g, int SX, int SY, int SZ, int pitch, int short_bins,
                                                        unsigned long long* __restrict__ hist, size_t hist_len,
                                                        unsigned int* __restrict__ max_out) {
    extern __shared__ uint32_t smem[];
    const int bins = kZThreads == 512 ? kHistSmall : short_bins;
    unsigned int* h_small = smem;   // [bins]
    uint32_t* tile = smem + bins;   // [SZ][pitch]
    const int tiles_y = (SY + kTileY - 1) / kTileY;
    const int x = blockIdx.x / tiles_y;
    const int y0 = (blockIdx.x % tiles_y) * kTileY;
    const int ny = min(kTileY, SY - y0);
    const size_t plane = static_cast<size_t>(SX) * SY;
    uint32_t* base = g + static_cast<size_t>(x) * SY + y0;
    const int yy = threadIdx.x % kTileY, z0 = threadIdx.x / kTileY;
    constexpr int kRows = kZThreads / kTileY;  // z-slices the block loads at a time

    for (int i = threadIdx.x; i < bins; i += kZThreads) h_small[i] = 0;
#pragma unroll 8
    for (int z = z0; z < SZ; z += kRows) tile[z * pitch + yy] = yy < ny ? base[z * plane + yy] : 0u;
    __syncthreads();

    unsigned int local_max = 0;
    const int y = y0 + yy;
    const int mxy = min(min(x, SX - 1 - x), min(y, SY - 1 - y));
    auto f = [&](int j) { return tile[j * pitch + yy]; };
    for (int zb = 0; zb < SZ; zb += kRows * kOut) {
        const int i0 = zb + z0 * kOut;
        const int live = yy < ny ? min(max(SZ - i0, 0), kOut) : 0;
        uint32_t best[kOut];
        walk_line(f, SZ, min(i0, SZ - 1), live, best);
#pragma unroll
        for (int k = 0; k < kOut; ++k) {
            if (k >= live) continue;
            const int z = i0 + k;
            const uint32_t e = best[k];
            base[z * plane + yy] = e;
            if (e == 0) continue;
            local_max = max(local_max, e);
            const int m = min(mxy, min(z, SZ - 1 - z));
            // e <= m^2 <=> the ball of radius sqrt(e) stays inside the image (EDC.cpp:316-327).
            if (e <= static_cast<uint32_t>(m) * static_cast<uint32_t>(m)) {  // m < 2^15 here
                if (e < static_cast<uint32_t>(bins)) atomicAdd(&h_small[e], 1u);
                else if (e < hist_len) atomicAdd(&hist[e], 1ull);
            }
        }
    }
    local_max = __reduce_max_sync(0xFFFFFFFFu, local_max);
    if ((threadIdx.x & 31) == 0 && local_max) atomicMax(max_out, local_max);
    __syncthreads();
    for (int i = threadIdx.x; i < bins && i < static_cast<int>(hist_len); i += kZThreads)
        if (h_small[i]) atomicAdd(&hist[i], static_cast<unsigned long long>(h_small[i]));
}

// The dynamic shared-memory limit is a process-wide attribute of each kernel, so it is set
// once per device to the device's opt-in maximum: lowering it per call would race with
// calls on other host threads (batch lanes) that launch with more.
std::mutex g_attr_mutex;
std::vector<int> g_attr_devices;

void edt_smem_attributes(size_t optin) {
    int dev = 0;
    PMA_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(g_attr_mutex);
    if (std::find(g_attr_devices.begin(), g_attr_devices.end(), dev) != g_attr_devices.end()) return;
    const int bytes = static_cast<int>(optin);
    const auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    PMA_CUDA(cudaFuncSetAttribute(edt_general_x, attr, bytes));
    PMA_CUDA(cudaFuncSetAttribute(edt_general_y, attr, bytes));
    PMA_CUDA(cudaFuncSetAttribute(edt_general_z, attr, bytes));
    PMA_CUDA(cudaFuncSetAttribute(edt_pass_x<1>, attr, bytes));
    PMA_CUDA(cudaFuncSetAttribute(edt_pass_x<4>, attr, bytes));
    PMA_CUDA(cudaFuncSetAttribute(edt_pass_y, attr, bytes));
    PMA_CUDA(cudaFuncSetAttribute(edt_pass_z<128>, attr, bytes));
    PMA_CUDA(cudaFuncSetAttribute(edt_pass_z<512>, attr, bytes));
    g_attr_devices.push_back(dev);
}

// The three passes on stream s. stats: hist_len histogram bins, then the maximum, all set to
// zero first. timed(name): brackets a pass for the timing report. Returns the kernels launched.
template <class Timed>
void edt_passes(const char* who, const uint8_t* solid, pma_dims d, uint32_t* edt2, unsigned long long* hist, size_t hist_len,
                size_t smem_optin, int num_sms, cudaStream_t s, Timed timed) {
    const int SX = d.sx, SY = d.sy, SZ = d.sz;
    auto* d_max = reinterpret_cast<unsigned int*>(hist + hist_len);
    auto need = [&](size_t smem, const char* what) {
        PMA_REQUIRE(smem <= smem_optin, PMA_ERR_ARGUMENT, std::string(who) + ": " + what + " extent too large");
    };
    const int words = (SX + 31) / 32;
    int gx_threads = 256;  // of the general pass X
    while (gx_threads > 32 && static_cast<size_t>(words) * 4 * gx_threads > 96 * 1024) gx_threads >>= 1;
    const size_t gx_smem = static_cast<size_t>(words) * 4 * gx_threads;
    need(gx_smem, "X");
    need(static_cast<size_t>(SY) * 4, "Y");
    need(static_cast<size_t>(SZ) * kTileY * 4 + kHistSmall * 4, "Z");
    const size_t rows = static_cast<size_t>(SX) * SZ, cols = static_cast<size_t>(SY) * SZ;
    const size_t tiles = static_cast<size_t>(SX) * ((SY + kTileY - 1) / kTileY);
    // Distances of pass X are at most 1.5 SX; a walk adds at most the squared line length to the
    // largest input. The columns of pass X take 4 V bytes of shared memory a word and thread.
    const double reach = 1.5 * SX, yl = SY + 16.0, zl = SZ + 16.0;
    const size_t x1 = static_cast<size_t>(words) * 4 * kXThreads;
    const bool fast = reach <= 65535.0 && reach * reach + 2.0 * yl * yl + 2.0 * zl * zl < 4294967295.0 && x1 <= smem_optin;
    if (!fast) {
        PMA_CUDA(cudaMemsetAsync(hist, 0, hist_len * 8 + 16, s));
        timed("edt_pass_x", [&] {
            edt_general_x<<<div_up(cols, gx_threads), gx_threads, gx_smem, s>>>(solid, edt2, SX, SY, SZ, words);
        });
        int warps = 8;
        while (warps > 1 && static_cast<size_t>(warps) * SY * 4 > 96 * 1024) warps >>= 1;
        const size_t blocks = std::min<size_t>((rows + warps - 1) / warps, static_cast<size_t>(num_sms) * 64);
        timed("edt_pass_y", [&] {
            edt_general_y<<<static_cast<unsigned>(blocks), warps * 32, static_cast<size_t>(warps) * SY * 4, s>>>(edt2, SY, rows);
        });
        timed("edt_pass_z", [&] {
            edt_general_z<<<static_cast<unsigned>(tiles), 256, static_cast<size_t>(SZ) * kTileY * 4 + kHistSmall * 4, s>>>(
                edt2, SX, SY, SZ, hist, hist_len, d_max);
        });
        return;
    }
    // Four columns a thread where rows and addresses allow the wider accesses, and the bits fit
    // three blocks an SM (1024 rows: 64 KB).
    const bool four = SY % 4 == 0 && reinterpret_cast<uintptr_t>(solid) % 4 == 0 && reinterpret_cast<uintptr_t>(edt2) % 8 == 0 &&
                      4 * x1 <= smem_optin / 3;
    timed("edt_pass_x", [&] {
        const size_t nclear = hist_len + 2;
        if (four) edt_pass_x<4><<<div_up(cols / 4, kXThreads), kXThreads, 4 * x1, s>>>(solid, edt2, SX, SY, SZ, words, hist, nclear);
        else edt_pass_x<1><<<div_up(cols, kXThreads), kXThreads, x1, s>>>(solid, edt2, SX, SY, SZ, words, hist, nclear);
    });
    timed("edt_pass_y", [&] {
        // below the general pass's 4 SY bytes; 4 (mod 8)
        const size_t row_words = (static_cast<size_t>(SY) / 2 + SY / kOut + 2 + 3) / 8 * 8 + 4;
        int warps = 8;
        while (warps > 1 && warps * (row_words + 32 * kYPad) * 4 > 96 * 1024) warps >>= 1;
        const size_t smem = warps * (row_words + 32 * kYPad) * 4;
        const size_t blocks = std::min<size_t>((rows + warps - 1) / warps, static_cast<size_t>(num_sms) * 64);
        edt_pass_y<<<static_cast<unsigned>(blocks), warps * 32, smem, s>>>(edt2, SY, rows, static_cast<int>(row_words));
    });
    timed("edt_pass_z", [&] {
        // balls inside the image have r^2 <= half^2; hist_len >= kHistSmall covers the rounding
        const long long half = (std::min(SX, std::min(SY, SZ)) - 1) / 2;
        const int bins = SZ > kZShort ? kHistSmall : static_cast<int>((std::min<long long>(kHistSmall, half * half + 1) + 3) / 4 * 4);
        auto smem = [&](int pitch) { return (static_cast<size_t>(SZ) * pitch + bins) * 4; };
        const int pitch = smem(18) <= smem_optin ? 18 : 16;
        const unsigned blocks = static_cast<unsigned>(tiles);
        if (SZ <= kZShort) edt_pass_z<128><<<blocks, 128, smem(pitch), s>>>(edt2, SX, SY, SZ, pitch, bins, hist, hist_len, d_max);
        else edt_pass_z<512><<<blocks, 512, smem(pitch), s>>>(edt2, SX, SY, SZ, pitch, bins, hist, hist_len, d_max);
    });
}

}  // namespace

void edt(pma_ctx* ctx, const uint8_t* solid, pma_dims d, uint32_t* edt2, pma_edt_stats* stats,
         uint64_t* h_hist, size_t hist_cap) {
    KernelTimer kt_stage(ctx, "stage_edt");  // the whole stage, for the untimed remainder
    check_dims(d);
    edt_smem_attributes(ctx->smem_optin);
    PMA_REQUIRE(solid && edt2, PMA_ERR_ARGUMENT, "pma_edt: null device pointer");
    cudaStream_t s = ctx->stream;
    // Non-crossing balls have e <= ((min extent - 1) / 2)^2.
    const int minext = std::min(d.sx, std::min(d.sy, d.sz));
    size_t hist_len = static_cast<size_t>((minext - 1) / 2) * ((minext - 1) / 2) + 1;
    hist_len = std::max<size_t>(hist_len, kHistSmall);
    auto* d_hist = static_cast<unsigned long long*>(ctx->scratch("edt.hist", hist_len * 8 + 16));
    edt_passes("pma_edt", solid, d, edt2, d_hist, hist_len, ctx->smem_optin, ctx->num_sms, s, [&](const char* name, auto launch) {
        KernelTimer kt(ctx, name);
        launch();
        ctx->check_launch(name);
    });
    // the maximum and the first bins come back together; more bins than that by a copy
    const size_t head = h_hist ? std::min<size_t>(std::min(hist_cap, hist_len), 4096) : 0;
    auto* h = static_cast<unsigned long long*>(ctx->host_staging(8 * (head + 1)));
    ReadBack rb;
    rb.add(h, d_hist + hist_len, 8);
    if (head) rb.add(h + 1, d_hist, head * 8);
    read_back(ctx, rb);
    const unsigned int maxv = static_cast<unsigned int>(h[0]);
    if (stats) {
        stats->max_edt2 = maxv;
        stats->pad_ = 0;
        stats->hist_len = static_cast<uint64_t>(maxv) + 1;
    }
    if (h_hist && hist_cap) {
        size_t want = std::min<size_t>(hist_cap, static_cast<size_t>(maxv) + 1);
        size_t have = std::min(want, hist_len);
        std::copy(h + 1, h + 1 + std::min(have, head), h_hist);
        if (have > head) PMA_CUDA(cudaMemcpy(h_hist + head, d_hist + head, (have - head) * 8, cudaMemcpyDeviceToHost));
        for (size_t i = have; i < want; ++i) h_hist[i] = 0;
    }
}

// ---------------------------------------------------------------------------------------
// Allocation-free variant (pma_edt_noalloc)
//
// Some callers cannot let the library allocate device memory: an application whose own
// memory pool already holds the device's memory, or one that must not call cudaMalloc and
// cudaFree while it runs because both can synchronise the whole device and stall its other
// streams (a service answering requests on streams it owns, an interactive viewer stepping
// through volumes). Such callers also hold no pma_ctx, whose scratch cache allocates on
// first use. This variant writes its results into the caller's buffers and keeps its only
// scratch - the histogram bins and the running maximum of pass Z - in a fixed array in the
// module's global memory. Its size bounds the volumes it accepts: a 2^18-bin histogram
// covers balls up to e = 511^2, i.e. volumes whose smallest extent is at most 1024.
// ---------------------------------------------------------------------------------------
namespace {

constexpr size_t kNoAllocHistBins = size_t(1) << 18;
constexpr int kNoAllocMaxDevices = 64;

struct NoAllocDevice {
    unsigned long long* scratch = nullptr;  // address of the static array on that device
    size_t smem_optin = 0;
    int num_sms = 0;
};

std::mutex g_noalloc_mutex;
NoAllocDevice g_noalloc_devices[kNoAllocMaxDevices];

}  // namespace

// Bins [0, kNoAllocHistBins) followed by two words; the maximum sits in the first word
// after the bins in use (hist_len), as in the context-based path.
static __device__ __align__(256) unsigned long long g_edt_noalloc_scratch[kNoAllocHistBins + 2];

// Once per device, with that device current: the scratch address, the shared-memory limit
// and the SM count. Later calls read the cached values.
static NoAllocDevice noalloc_device() {
    int dev = 0;
    PMA_CUDA(cudaGetDevice(&dev));
    PMA_REQUIRE(dev >= 0 && dev < kNoAllocMaxDevices, PMA_ERR_ARGUMENT,
                "pma_edt_noalloc: device ordinal above 63");
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    NoAllocDevice& e = g_noalloc_devices[dev];
    if (!e.scratch) {
        void* p = nullptr;
        const cudaError_t rc = cudaGetSymbolAddress(&p, g_edt_noalloc_scratch);
        PMA_REQUIRE(rc == cudaSuccess && p, PMA_ERR_CUDA,
                    std::string("pma_edt_noalloc: cudaGetSymbolAddress of the scratch array failed: ") +
                        cudaGetErrorString(rc));
        int optin = 0;
        PMA_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
        PMA_CUDA(cudaDeviceGetAttribute(&e.num_sms, cudaDevAttrMultiProcessorCount, dev));
        e.smem_optin = static_cast<size_t>(optin);
        e.scratch = static_cast<unsigned long long*>(p);
    }
    return e;
}

void edt_noalloc(const uint8_t* solid, pma_dims d, uint32_t* edt2, pma_edt_stats* stats,
                 uint64_t* h_hist, size_t hist_cap, cudaStream_t s) {
    check_dims(d);
    PMA_REQUIRE(solid && edt2, PMA_ERR_ARGUMENT, "pma_edt_noalloc: null device pointer");
    const int minext = std::min(d.sx, std::min(d.sy, d.sz));
    size_t hist_len = static_cast<size_t>((minext - 1) / 2) * ((minext - 1) / 2) + 1;
    hist_len = std::max<size_t>(hist_len, kHistSmall);
    PMA_REQUIRE(hist_len <= kNoAllocHistBins, PMA_ERR_LIMIT,
                "pma_edt_noalloc: smallest volume extent " + std::to_string(minext) +
                    " is above 1024, the largest its fixed 2 MiB histogram scratch covers; use pma_edt");
    const NoAllocDevice dev = noalloc_device();
    edt_smem_attributes(dev.smem_optin);

    // The bins in use and the maximum word start at zero on every call.
    unsigned long long* d_hist = dev.scratch;
    auto* d_max = reinterpret_cast<unsigned int*>(d_hist + hist_len);
    edt_passes("pma_edt_noalloc", solid, d, edt2, d_hist, hist_len, dev.smem_optin, dev.num_sms, s, [&](const char*, auto launch) {
        launch();
        PMA_CUDA(cudaGetLastError());
    });
    unsigned int maxv = 0;
    PMA_CUDA(cudaMemcpyAsync(&maxv, d_max, 4, cudaMemcpyDeviceToHost, s));
    PMA_CUDA(cudaStreamSynchronize(s));
    if (stats) {
        stats->max_edt2 = maxv;
        stats->pad_ = 0;
        stats->hist_len = static_cast<uint64_t>(maxv) + 1;
    }
    if (h_hist && hist_cap) {
        const size_t want = std::min<size_t>(hist_cap, static_cast<size_t>(maxv) + 1);
        const size_t have = std::min(want, hist_len);
        PMA_CUDA(cudaMemcpyAsync(h_hist, d_hist, have * 8, cudaMemcpyDeviceToHost, s));
        PMA_CUDA(cudaStreamSynchronize(s));
        for (size_t i = have; i < want; ++i) h_hist[i] = 0;
    }
}

}  // namespace pma
