// Pore seeds, initial pore propagation and empty-pore removal
// (PoreAndThroatComputer.cpp:93-269, BasePoreAndThroatComputer.cpp:37-133,
// EmptyPoresRemover.cpp:31-244).
//
// The reference runs one depth-first search per pore: from the seed it follows u -> v when
// v is a void stencil neighbour with crad(v) <= crad(u). Restated exactly:
//  * Plateaus. Voxels of one connected set of equal crad ("plateau") all reach each other,
//    so the set S of seeds reaching a voxel is constant on its plateau, and
//    S(p) = union of S(q) over plateaus q with an edge into p, plus p's own seed.
//  * Seeds. Maximum balls are visited in std::sort order and a ball starts a pore unless an
//    earlier pore already reached its centre. By induction on that order, a ball is a seed
//    exactly when no ball earlier in the order reaches it (a skipped ball was reached by an
//    earlier seed, which then reaches all it reaches). With m(p) the smallest rank of a ball
//    reaching plateau p, p's smallest-rank ball is a seed iff it beats m of every plateau
//    with an edge into p.
//  * Plateaus are found by a union-find over equal-crad neighbours (from 2^24 voxels:
//    pointer jumping on the initial trees, then unions of the recorded parent pairs).
//  * Both recurrences run plateau by plateau in decreasing crad, one launch per crad level. The ball
//    order is the permutation that std::sort gives the same sequence (z, x, y scan order) under the
//    same comparator (ordered_sort_device), so equal radii tie-break exactly as in the reference.
//  * A voxel's label is its seed's pore id when |S| = 1 and a shared type ("throat") when
//    |S| >= 2. Pore volumes, boundary flags, type volumes and type pore lists are exact.
//    The reference numbers types in its depth-first creation order, which also consumed ids
//    for types deleted later. The types are first numbered by (last pore of the type, first
//    voxel of the type), then renumbered in the reference's order by a host replay of each
//    pore's search order (exact_ids.cpp), unless the context asks for the cheaper numbering.
#include <thrust/iterator/counting_iterator.h>

#include <algorithm>
#include <cstring>
#include <map>
#include <memory>
#include <chrono>
#include <thread>
#include <type_traits>
#include <vector>

#include "devutil.cuh"
#include "ordered_sort.cuh"
#include "ordered_sort.h"
#include "type_rows.cuh"

namespace pma {
namespace {

constexpr uint32_t kNone = 0xFFFFFFFFu;

__global__ void flag_outer(const uint8_t* __restrict__ mask, size_t n, uint8_t* __restrict__ flags) {
    PMA_GRID_STRIDE(v, n) flags[v] = mask[v] == 255;
}

__global__ void gather_u32(const uint32_t* __restrict__ src, const uint32_t* __restrict__ idx,
                           size_t n, uint32_t* __restrict__ out) {
    PMA_GRID_STRIDE(i, n) out[i] = src[idx[i]];
}

__global__ void fill_u32(uint32_t* __restrict__ a, size_t n, uint32_t value) {
    PMA_GRID_STRIDE(i, n) a[i] = value;
}

__global__ void flag_seeds(const uint32_t* __restrict__ seed, size_t np, uint8_t* __restrict__ flags) {
    PMA_GRID_STRIDE(p, np) flags[p] = seed[p] != kNone;
}

// up = [seed ranks (ascending) | their pore ids]
__global__ void scatter_seed_ids(const uint32_t* __restrict__ up, size_t npores, uint32_t* __restrict__ rank2pore,
                                 uint32_t* __restrict__ rank2id) {
    PMA_GRID_STRIDE(k, npores) {
        rank2pore[up[k]] = static_cast<uint32_t>(k);
        rank2id[up[k]] = up[npores + k];
    }
}

__global__ void pack_items(const uint32_t* __restrict__ r2, const uint32_t* __restrict__ idx, size_t n,
                           unsigned long long* __restrict__ items) {
    PMA_GRID_STRIDE(i, n) items[i] = (static_cast<unsigned long long>(r2[i]) << 32) | idx[i];
}

__global__ void scatter_rank(const unsigned long long* __restrict__ items, size_t n, uint32_t* __restrict__ crank) {
    PMA_GRID_STRIDE(r, n) crank[static_cast<uint32_t>(items[r])] = static_cast<uint32_t>(r);
}

__global__ void gather_items(const unsigned long long* __restrict__ items, const uint32_t* __restrict__ ranks, size_t n,
                             unsigned long long* __restrict__ out) {
    PMA_GRID_STRIDE(k, n) out[k] = items[ranks[k]];
}

// --- union-find over equal-crad neighbours (parents always point to smaller indices) ---

__device__ __forceinline__ uint32_t uf_root(uint32_t* parent, uint32_t v) {
    uint32_t cur = parent[v];
    if (cur == v) return v;
    uint32_t prev = v, next;
    while (cur > (next = parent[cur])) {
        parent[prev] = next;  // path halving; racing writes only shorten paths
        prev = cur;
        cur = next;
    }
    return cur;
}

// Start every void voxel under its smallest-index equal-crad neighbour (the backward
// offsets, most negative index first), so that most trees exist before any union runs.
__global__ void uf_init(const uint32_t* __restrict__ crad, Grid g, size_t n, int d3q7,
                        uint32_t* __restrict__ parent) {
    PMA_GRID_STRIDE(v, n) {
        const uint32_t r = crad[v];
        if (!r) {
            parent[v] = kNone;
            continue;
        }
        int x, y, z;
        g.coords(v, x, y, z);
        uint32_t p = static_cast<uint32_t>(v);
        for (int k = 12; k >= 0 && p == v; --k) {  // the 13 forward offsets, negated, largest first
            int dx, dy, dz;
            if (k < 4) {
                dz = 0;
                dx = (k == 0) ? 0 : 1;
                dy = (k == 0) ? 1 : k - 2;
            } else {
                dz = 1;
                dx = (k - 4) / 3 - 1;
                dy = (k - 4) % 3 - 1;
            }
            if (d3q7 && (dx != 0) + (dy != 0) + (dz != 0) > 1) continue;
            const int nx = x - dx, ny = y - dy, nz = z - dz;
            if (!g.inside(nx, ny, nz)) continue;
            const size_t w = g.idx(nx, ny, nz);
            if (crad[w] == r) p = static_cast<uint32_t>(w);
        }
        parent[v] = p;
    }
}

// Pointer jumping on the initial trees: parent[v] moves up to a few ancestors at a time, in
// place (a value read may already have jumped in this pass, which only shortens paths). The
// initial trees of a large plateau are chains of backward neighbours hundreds of voxels long;
// after a few passes almost every voxel points at its tree's root, so that uf_hook finds
// most neighbour pairs already joined without walking. Each pass skips once a pass changed
// nothing (done[k - 1] == 0).
// Measured: 1024^3 spinodal 408 -> 371 ms for jumps and hooks together; on a 96^3 sphere pack
// the passes cost more (0.5 ms) than they save, so they run from 2^24 voxels up.
constexpr int kJumpPasses = 6;
constexpr size_t kJumpMinVoxels = size_t(1) << 24;

__global__ void uf_jump(size_t n, uint32_t* __restrict__ parent, unsigned int* __restrict__ changed, int pass) {
    if (pass > 0 && *reinterpret_cast<volatile unsigned int*>(changed + pass - 1) == 0) return;
    unsigned int any = 0;
    PMA_GRID_STRIDE(v, n) {
        const uint32_t p = parent[v];
        if (p == kNone || p == v) continue;
        uint32_t cur = p, next = parent[cur];
        for (int k = 0; k < 4 && next != cur; ++k) {
            cur = next;
            next = parent[cur];
        }
        if (cur != p) {
            parent[v] = cur;
            any = 1;
        }
    }
    if (__any_sync(0xFFFFFFFFu, any) && (threadIdx.x & 31) == 0) changed[pass] = 1;
}

__global__ void uf_hook(const uint32_t* __restrict__ crad, Grid g, size_t n, int d3q7,
                        uint32_t* __restrict__ parent, unsigned int* __restrict__ err, int union_limit) {
    PMA_GRID_STRIDE(v, n) {
        const uint32_t r = crad[v];
        if (!r) continue;
        int x, y, z;
        g.coords(v, x, y, z);
        // Each unordered pair once: the 13 offsets whose linear index delta
        // dz*SX*SY + dx*SY + dy is positive, i.e. (dz, dx, dy) > 0 lexicographically.
        // rv: a known ancestor of v (its parent after the jumps, then its root after each
        // union), so root walks from v start close to the root.
        uint32_t rv = parent[v];
        for (int k = 0; k < 13; ++k) {
            int dx, dy, dz;
            if (k < 4) {
                dz = 0;
                dx = (k == 0) ? 0 : 1;
                dy = (k == 0) ? 1 : k - 2;
            } else {
                dz = 1;
                dx = (k - 4) / 3 - 1;
                dy = (k - 4) % 3 - 1;
            }
            if (d3q7 && (dx != 0) + (dy != 0) + (dz != 0) > 1) continue;
            const int nx = x + dx, ny = y + dy, nz = z + dz;
            if (!g.inside(nx, ny, nz)) continue;
            const size_t w = g.idx(nx, ny, nz);
            if (crad[w] != r) continue;
            if (parent[w] == rv) continue;  // already joined
            uint32_t a = uf_root(parent, rv);
            uint32_t b = uf_root(parent, static_cast<uint32_t>(w));
            int it = 0;
            while (a != b) {
                if (++it > union_limit) {
                    atomicOr(err, 1u);
                    break;
                }
                if (a < b) {
                    const uint32_t old = atomicCAS(&parent[b], b, a);
                    if (old == b) break;
                    b = old;
                } else {
                    const uint32_t old = atomicCAS(&parent[a], a, b);
                    if (old == a) break;
                    a = old;
                }
            }
            rv = a < b ? a : b;  // the surviving root, an ancestor of v
        }
    }
}

// Pairs of neighbouring voxels' ids, each pair of ids once per tile, as 64-bit keys; count receives how many,
// also those beyond cap (not written). Each unordered pair of voxels is looked at from the voxel of smaller index
// (13 forward offsets, in 5 rows along y). A row is read once, coalesced, by a warp of 32 voxels along y: the
// voxel's neighbours at y - 1 and y + 1 come from the lanes beside it, and a slice's rows serve the next slice.
//
// kUnion: id is the union-find's parent. After the pointer jumps almost every voxel points at its initial tree's
// root, so that a pair of equal crad with different parents is the rare case; uf_union_pairs then unions them, one
// thread a pair, instead of one walk to the roots after the other. The partition and its roots are the same:
// each plateau's root is its smallest voxel index, whatever the order of the unions.
// Else id is the plateau: edges (lower-radius plateau, higher-radius one), where crad differs.
//
// Neighbouring voxels mostly report the same pairs, and plateaus are 3-D blobs. A voxel of the same id as the one
// before it along y leaves out what that one has seen of a row (all but the neighbour at y + 1), and any voxel the
// neighbours of its own that follow an equal one. What is left is queued by warp and put, 32 at a time, into
// a set in shared memory over the tile of 4 (z) x 8 (x) x 32 (y) voxels; the set is written out at the tile's end
// with one atomic. A key that finds no slot in eight probes is written at once: the sort and unique (the unions)
// that follow take copies.
//
// What bounds it: instructions. 512^3 random field: edges 8.25 -> 4.3 ms, pairs and unions 5.8 -> 2.5; one thread
// a voxel with 13 look-ups of its own took 1425 instructions a warp for the edges alone, and an atomic on one
// counter per warp and slice. (Reading a slot before the compare-and-swap: 9.7 ms.)
constexpr int kTileY = 32, kTileX = 8, kTileZ = 4;  // a warp covers a row of the tile, one slice after another
constexpr int kPairThreads = 32 * kTileX;

struct PairRow {  // crad (0: solid or outside) and id at y - 1, y and y + 1 of a lane
    uint32_t c[3], i[3];
};

__device__ __forceinline__ PairRow pair_row(const uint32_t* __restrict__ id, const uint32_t* __restrict__ crad, const Grid& g, int x, int y,
                                            int z) {
    const unsigned lane = threadIdx.x & 31;
    PairRow r;
    r.c[1] = 0;
    r.i[1] = kNone;
    uint32_t ce = 0, ie = kNone;  // past the warp's row, at lanes 0 and 31
    if (x >= 0 && x < g.SX && z < g.SZ) {  // the same for the warp
        const size_t at = g.idx(x, y, z);
        if (y < g.SY) {
            r.c[1] = crad[at];
            r.i[1] = id[at];
        }
        if ((lane == 0 && y > 0) || (lane == 31 && y + 1 < g.SY)) {
            const size_t e = lane == 0 ? at - 1 : at + 1;
            ce = crad[e];
            ie = id[e];
        }
    }
    r.c[0] = __shfl_up_sync(0xFFFFFFFFu, r.c[1], 1);
    r.i[0] = __shfl_up_sync(0xFFFFFFFFu, r.i[1], 1);
    r.c[2] = __shfl_down_sync(0xFFFFFFFFu, r.c[1], 1);
    r.i[2] = __shfl_down_sync(0xFFFFFFFFu, r.i[1], 1);
    if (lane == 0) {
        r.c[0] = ce;
        r.i[0] = ie;
    }
    if (lane == 31) {
        r.c[2] = ce;
        r.i[2] = ie;
    }
    return r;
}

template <bool kUnion>
__global__ void __launch_bounds__(kPairThreads, 5) voxel_pairs(const uint32_t* __restrict__ id, const uint32_t* __restrict__ crad, Grid g,
                                                               int d3q7, int sb, unsigned long long* __restrict__ count,
                                                               unsigned long long* __restrict__ out, unsigned long long cap) {
    constexpr int kTable = kUnion ? 1024 : 2048, kPer = kTable / kPairThreads;
    __shared__ unsigned long long table[kTable], s_queue[kTileX][64], s_base;
    __shared__ unsigned s_sum[kTileX];
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5, lt = (1u << lane) - 1u;
    const unsigned nty = (g.SY + kTileY - 1) / kTileY, ntx = (g.SX + kTileX - 1) / kTileX;
    const size_t ntiles = static_cast<size_t>(nty) * ntx * ((g.SZ + kTileZ - 1) / kTileZ);
    unsigned long long* queue = s_queue[warp];
    auto insert = [&](unsigned long long key) {
        unsigned h = static_cast<unsigned>((key * 0x9E3779B97F4A7C15ull) >> 40) & (kTable - 1);
        for (int probe = 0; probe < 8; ++probe, h = (h + 1) & (kTable - 1)) {
            const unsigned long long prev = atomicCAS(&table[h], ~0ull, key);
            if (prev == ~0ull || prev == key) return;
        }
        const unsigned long long pos = atomicAdd(count, 1ull);
        if (pos < cap) out[pos] = key;
    };
    for (int k = 0; k < kPer; ++k) table[threadIdx.x + k * kPairThreads] = ~0ull;
    __syncthreads();
    for (size_t t = blockIdx.x; t < ntiles; t += gridDim.x) {  // block-uniform
        const int y = static_cast<int>(t % nty) * kTileY + static_cast<int>(lane);
        const size_t rest = t / nty;
        const int x = static_cast<int>(rest % ntx) * kTileX + static_cast<int>(warp), z0 = static_cast<int>(rest / ntx) * kTileZ;
        unsigned head = 0, queued = 0;  // of the warp's queue, a ring of 64
        if (x < g.SX) {
            PairRow here = pair_row(id, crad, g, x, y, z0), next = pair_row(id, crad, g, x + 1, y, z0);
            for (int z = z0; z < min(z0 + kTileZ, g.SZ); ++z) {
                const uint32_t p = here.i[1], r = here.c[1];
                const bool as_before = lane > 0 && here.i[0] == p;
                auto consider = [&](bool see, uint32_t q, uint32_t rq) {
                    const bool pair = see && r != 0 && (kUnion ? rq == r && q != p : rq != 0 && rq != r);
                    const unsigned m = __ballot_sync(0xFFFFFFFFu, pair);
                    if (!m) return;
                    if (pair) {
                        unsigned long long key;
                        if (kUnion) key = (static_cast<unsigned long long>(min(p, q)) << 32) | max(p, q);
                        else key = rq < r ? (static_cast<unsigned long long>(q) << sb) | p : (static_cast<unsigned long long>(p) << sb) | q;
                        queue[(head + queued + __popc(m & lt)) & 63] = key;
                    }
                    queued += __popc(m);
                    if (queued >= 32) {
                        __syncwarp();
                        insert(queue[(head + lane) & 63]);
                        head += 32;
                        queued -= 32;
                        __syncwarp();
                    }
                };
                auto row = [&](const PairRow& w) {
                    if (d3q7) {
                        consider(!(as_before && w.i[1] == w.i[0]), w.i[1], w.c[1]);
                    } else {
                        consider(!as_before, w.i[0], w.c[0]);
                        consider(!as_before && w.i[1] != w.i[0], w.i[1], w.c[1]);
                        consider(w.i[2] != w.i[1], w.i[2], w.c[2]);
                    }
                };
                consider(true, here.i[2], here.c[2]);
                row(next);
                if (!d3q7) row(pair_row(id, crad, g, x - 1, y, z + 1));
                here = pair_row(id, crad, g, x, y, z + 1);
                row(here);
                next = pair_row(id, crad, g, x + 1, y, z + 1);
                if (!d3q7) row(next);
            }
            __syncwarp();
            if (lane < queued) insert(queue[(head + lane) & 63]);
        }
        __syncthreads();
        // the set, emptied for the next tile
        unsigned long long keys[kPer];
        unsigned kept = 0;
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            keys[k] = table[threadIdx.x + k * kPairThreads];
            table[threadIdx.x + k * kPairThreads] = ~0ull;
            kept += keys[k] != ~0ull ? 1u : 0u;
        }
        unsigned incl = kept;
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned t2 = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= static_cast<unsigned>(o)) incl += t2;
        }
        if (lane == 31) s_sum[warp] = incl;
        __syncthreads();
        unsigned before = 0, total = 0;
#pragma unroll
        for (unsigned w = 0; w < kTileX; ++w) {
            before += w < warp ? s_sum[w] : 0u;
            total += s_sum[w];
        }
        if (threadIdx.x == 0 && total) s_base = atomicAdd(count, static_cast<unsigned long long>(total));
        __syncthreads();
        unsigned long long pos = s_base + before + incl - kept;
#pragma unroll
        for (int k = 0; k < kPer; ++k)
            if (keys[k] != ~0ull) {
                if (pos < cap) out[pos] = keys[k];
                ++pos;
            }
    }
}

__global__ void uf_union_pairs(const unsigned long long* __restrict__ pairs, size_t np,
                               uint32_t* __restrict__ parent, unsigned int* __restrict__ err, int union_limit) {
    PMA_GRID_STRIDE(i, np) {
        uint32_t a = uf_root(parent, static_cast<uint32_t>(pairs[i] >> 32));
        uint32_t b = uf_root(parent, static_cast<uint32_t>(pairs[i]));
        int it = 0;
        while (a != b) {
            if (++it > union_limit) {
                atomicOr(err, 1u);
                break;
            }
            if (a < b) {
                const uint32_t old = atomicCAS(&parent[b], b, a);
                if (old == b) break;
                b = old;
            } else {
                const uint32_t old = atomicCAS(&parent[a], a, b);
                if (old == a) break;
                a = old;
            }
        }
    }
}

// Read-only root walk: flattening must not halve paths, or a racing halving store could
// replace another voxel's final root pointer with an intermediate ancestor.
__device__ __forceinline__ uint32_t uf_root_readonly(const uint32_t* parent, uint32_t v) {
    uint32_t cur = v, next;
    while ((next = parent[cur]) != cur) cur = next;
    return cur;
}

__global__ void uf_flatten(size_t n, uint32_t* parent) {
    PMA_GRID_STRIDE(v, n) {
        if (parent[v] != kNone) parent[v] = uf_root_readonly(parent, static_cast<uint32_t>(v));
    }
}

__global__ void flag_roots(const uint32_t* __restrict__ parent, size_t n, uint8_t* __restrict__ flags) {
    PMA_GRID_STRIDE(v, n) flags[v] = parent[v] == v;
}

__global__ void scatter_pid(const uint32_t* __restrict__ roots, size_t np, uint32_t* __restrict__ tmp) {
    PMA_GRID_STRIDE(p, np) tmp[roots[p]] = static_cast<uint32_t>(p);
}

// parent[v] (the root voxel) becomes the dense plateau id.
__global__ void to_pid(const uint32_t* __restrict__ tmp, size_t n, size_t np, uint32_t* __restrict__ parent,
                       unsigned int* __restrict__ err) {
    PMA_GRID_STRIDE(v, n) {
        const uint32_t r = parent[v];
        if (r == kNone) continue;
        const uint32_t p = tmp[r];
        if (p < np) {
            parent[v] = p;
        } else {  // not a root: refuse rather than index past the plateau arrays
            parent[v] = kNone;
            atomicOr(err, 8u);
        }
    }
}

__global__ void plateau_stats(const uint32_t* __restrict__ pid, const uint32_t* __restrict__ crad,
                              const uint32_t* __restrict__ crank, Grid g, size_t n,
                              uint32_t* __restrict__ pcrad, unsigned int* __restrict__ psize,
                              unsigned int* __restrict__ pface, uint32_t* __restrict__ pminrank) {
    // Neighbouring voxels mostly share a plateau: lanes of a warp with the same plateau
    // combine their updates (one atomic per plateau and warp).
    const unsigned lane = threadIdx.x & 31;
    PMA_GRID_STRIDE(v, n) {
        const uint32_t p = pid[v];
        int x, y, z;
        g.coords(v, x, y, z);
        const unsigned face = g.on_face(x, y, z) ? 1u : 0u;
        const uint32_t rk = p == kNone ? kNone : crank[v];
        const unsigned peers = __match_any_sync(__activemask(), p);
        const unsigned any_face = __reduce_or_sync(peers, face);
        const uint32_t min_rank = __reduce_min_sync(peers, rk);
        if (p == kNone || static_cast<int>(lane) != __ffs(peers) - 1) continue;
        pcrad[p] = crad[v];
        atomicAdd(&psize[p], static_cast<unsigned>(__popc(peers)));
        if (any_face) pface[p] = 1;
        if (min_rank != kNone) atomicMin(&pminrank[p], min_rank);
    }
}

// CSR offsets of edges sorted by destination (key >> sb), and the sources (the low sb bits) as
// 32-bit words, the form the level sweep reads.
__global__ void edge_offsets(const unsigned long long* __restrict__ edges, size_t ne, size_t np, int sb,
                             unsigned int* __restrict__ eoff, uint32_t* __restrict__ src) {
    PMA_GRID_STRIDE(i, ne + 1) {
        const uint32_t cur = (i < ne) ? static_cast<uint32_t>(edges[i] >> sb) : static_cast<uint32_t>(np);
        const uint32_t prev = (i == 0) ? 0u : static_cast<uint32_t>(edges[i - 1] >> sb) + 1u;
        for (uint32_t p = prev; p <= cur && p <= np; ++p) eoff[p] = static_cast<unsigned int>(i);
        if (i < ne) src[i] = static_cast<uint32_t>(edges[i] & ((1ull << sb) - 1));
    }
}

__global__ void level_starts(const uint32_t* __restrict__ key, size_t np, uint8_t* __restrict__ flags) {
    PMA_GRID_STRIDE(i, np) flags[i] = i == 0 || key[i] != key[i - 1];
}

__global__ void level_keys(const uint32_t* __restrict__ pcrad, size_t np, uint32_t* __restrict__ key,
                           uint32_t* __restrict__ val) {
    PMA_GRID_STRIDE(p, np) {
        key[p] = 0xFFFFFFFFu - pcrad[p];  // ascending key = descending crad
        val[p] = static_cast<uint32_t>(p);
    }
}

// --- level sweep ---------------------------------------------------------------------------
//
// One step per crad level: S(p) = union of S(q) over the edges q -> p, plus p's own seed. A
// predecessor lies in an earlier level, and most plateaus take over the set of a predecessor
// unchanged, so sets are shared: a plateau whose union equals a predecessor's set points at that
// set, and equal predecessor sets (the same pool position) are read once. What remains is latency
// (the loads edge -> set -> elements, once per level):
//  * level_sweep runs one level with a warp per plateau; unions with many elements or
//    many edges are left to the whole block, which collects them in a hash set in shared memory;
//  * runs of small levels go through one launch of one block, a block barrier between levels;
//  * nothing waits for the host: levels are launched one after another, and only a union too large
//    for a block's hash set stops the sweep (later levels return at once), for the host to merge
//    that level's such sets by expansion and a radix sort and to go on behind it.
// (A form with the sets of a level laid out by a scan, a read-back of the level's sizes and a
// sort for every union beyond 2048 elements took 8 launches and a host round trip a level. The
// sweep before and after, ms: 620 levels of 2000 plateaus 70 -> 7.1, 421 levels of 15 plateaus
// 17 -> 1.2, 125 levels of 37000 plateaus 14.9 -> 3.9.)
constexpr int kSweepWarps = 8;       // warps a block, one level
constexpr int kRunWarps = 16;        // warps of the block that runs small levels
constexpr size_t kRunLevel = 64;     // plateaus of a small level at most
constexpr unsigned kWarpSum = 512;   // elements of a warp's union at most (distinct sets)
constexpr int kWarpCap = 128;        // distinct elements of a warp's union
constexpr int kWarpHash = 256;       // slots (power of two, twice kWarpCap)
constexpr int kBlockBits = 12;       // log2 of the slots of a block's hash set (one less in a run of small
                                     // levels: more warps share the memory); half of them are used
constexpr int kSetHash = 512;        // pool positions of the sets a block has seen (power of two)
constexpr unsigned kSlab = 1024;     // pool elements a warp takes at a time
constexpr unsigned kSlabMax = 256;   // larger sets take their room directly
constexpr size_t kSweepList = 1024;  // plateaus of one block at most (its list of large unions)
constexpr unsigned kHardDegree = 1u << 16;  // edges beyond which a union is spread over the GPU

struct PlateauSets {
    const unsigned int* eoff;
    const uint32_t* edges;            // sources, sorted by destination
    const uint32_t* order;            // plateaus in decreasing crad
    const uint32_t* minrank;
    ulonglong2* set;                  // per plateau: pool position, length << 32 | smallest ball rank reaching it
    uint32_t* seed;                   // rank of the plateau's seed or kNone
    uint32_t* pool;
    unsigned long long pool_cap;
    unsigned long long* pool_n;       // elements taken (may pass pool_cap)
    ulonglong2* slab;                 // per warp of the sweep: next element, elements left
    unsigned nslab;
    unsigned int* err;
    unsigned long long* info;         // [0] level that stopped the sweep, [1] its hard sets, [2] their
                                      // elements, [3] keys the expansion wrote
    uint32_t* hard;                   // plateaus of the hard sets
    unsigned long long* cnt;          // [hard] distinct elements
    unsigned long long* first;        // [hard] first merged key
};

// L2: the writer may be another warp of this launch.
__device__ __forceinline__ ulonglong2 ldcg_set(const ulonglong2* p) {
    ulonglong2 v;
    asm volatile("ld.global.cg.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p));
    return v;
}

__device__ __forceinline__ uint32_t set_len(ulonglong2 s) { return static_cast<uint32_t>(s.y >> 32); }

template <int W>
struct SweepShared {
    uint32_t table[W][kWarpHash];
    uint32_t sorted[W][kWarpCap];
    unsigned int count[W];
    // the block's large unions
    uint32_t list[W == kRunWarps ? kRunLevel : kSweepList];
    unsigned int nlist;
    static constexpr int kBits = W == kRunWarps ? kBlockBits - 1 : kBlockBits;
    static constexpr int kSlots = 1 << kBits, kCap = kSlots / 2;  // distinct elements of a block's union
    uint32_t btable[kSlots];
    uint32_t bsorted[kCap];
    unsigned long long seen[kSetHash];
    unsigned int bcount, bover;
    uint32_t wmin[W];
    unsigned long long wmax[W];
    unsigned long long wsum[W];
    unsigned long long place;
};

// Room for k elements of the pool, by warp (all lanes get it); ~0 when the pool is full.
__device__ __forceinline__ unsigned long long sweep_room(const PlateauSets& st, ulonglong2& slab, bool has_slab,
                                                         unsigned k, unsigned lane) {
    unsigned long long at;
    if (has_slab && k <= kSlabMax) {
        if (slab.y < k) {
            unsigned long long b = 0;
            if (lane == 0) b = atomicAdd(st.pool_n, static_cast<unsigned long long>(kSlab));
            slab.x = __shfl_sync(0xFFFFFFFFu, b, 0);
            slab.y = kSlab;
        }
        at = slab.x;
        slab.x += k;
        slab.y -= k;
    } else {
        at = 0;
        if (lane == 0) at = atomicAdd(st.pool_n, static_cast<unsigned long long>(k));
        at = __shfl_sync(0xFFFFFFFFu, at, 0);
    }
    if (at + k <= st.pool_cap) return at;
    if (lane == 0) atomicOr(st.err, 2u);  // the host redoes the sweep with a larger pool
    return ~0ull;
}

__device__ __forceinline__ uint32_t warp_bitonic(uint32_t v, unsigned lane) {  // ascending over the lanes
    for (int k = 2; k <= 32; k <<= 1)
        for (int j = k >> 1; j > 0; j >>= 1) {
            const uint32_t other = __shfl_xor_sync(0xFFFFFFFFu, v, j);
            v = (((lane & j) == 0) == ((lane & k) == 0)) ? min(v, other) : max(v, other);
        }
    return v;
}

// Element u of the concatenation of the warp's sets (lane l's set starts at excl, elements from
// position off): its owner lane by a search over the lanes, then the load.
template <bool RUN>
__device__ __forceinline__ uint32_t warp_element(const PlateauSets& st, uint32_t u, uint32_t excl, unsigned long long off,
                                                 uint32_t total) {
    int owner = 0;
    for (int step = 16; step >= 1; step >>= 1) {
        const uint32_t e = __shfl_sync(0xFFFFFFFFu, excl, owner + step);
        if (e <= u) owner += step;
    }
    const unsigned long long o = __shfl_sync(0xFFFFFFFFu, off, owner);
    const uint32_t oe = __shfl_sync(0xFFFFFFFFu, excl, owner);
    if (u >= total) return kNone;
    const uint32_t* src = st.pool + o + (u - oe);
    return RUN ? __ldcg(src) : __ldg(src);
}

__device__ __forceinline__ uint32_t warp_exclusive(uint32_t v, unsigned lane, uint32_t& total) {
    uint32_t incl = v;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= static_cast<unsigned>(o)) incl += t;
    }
    total = __shfl_sync(0xFFFFFFFFu, incl, 31);
    return incl - v;
}

// One plateau by one warp; false: left to the block.
template <bool RUN, int W>
__device__ bool sweep_plateau(const PlateauSets& st, SweepShared<W>& sh, uint32_t p, ulonglong2& slab, bool has_slab) {
    const unsigned lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned e0 = __ldg(st.eoff + p), e1 = __ldg(st.eoff + p + 1);
    if (e1 - e0 > 32) return false;
    ulonglong2 s = make_ulonglong2(~0ull, kNone);  // no set
    if (e0 + lane < e1) {
        const uint32_t q = __ldg(st.edges + e0 + lane);
        s = RUN ? ldcg_set(st.set + q) : __ldg(st.set + q);
    }
    const uint32_t own = __ldg(st.minrank + p);
    uint32_t len = set_len(s);
    const uint32_t mp = __reduce_min_sync(0xFFFFFFFFu, static_cast<uint32_t>(s.y));
    const uint32_t seed = own < mp ? own : kNone;
    // one lane per distinct set
    const unsigned peers = __match_any_sync(0xFFFFFFFFu, len ? s.x : ~0ull);
    if (len && static_cast<int>(lane) != __ffs(peers) - 1) len = 0;
    const unsigned have = __ballot_sync(0xFFFFFFFFu, len != 0);
    const uint32_t longest = __reduce_max_sync(0xFFFFFFFFu, len);
    const int of = __ffs(__ballot_sync(0xFFFFFFFFu, len == longest)) - 1;  // a lane holding a longest set
    ulonglong2 out;
    out.x = __shfl_sync(0xFFFFFFFFu, s.x, of);
    uint32_t k = longest;
    if (seed != kNone || (have & (have - 1)) != 0) {
        uint32_t total;
        const uint32_t excl = warp_exclusive(len, lane, total);
        if (total > kWarpSum) return false;
        if (total + (seed != kNone ? 1u : 0u) <= 32) {
            uint32_t v = warp_element<RUN>(st, lane, excl, s.x, total);
            if (seed != kNone && lane == total) v = seed;
            v = warp_bitonic(v, lane);
            const uint32_t prev = __shfl_up_sync(0xFFFFFFFFu, v, 1);
            const bool keep = v != kNone && (lane == 0 || prev != v);
            const unsigned mask = __ballot_sync(0xFFFFFFFFu, keep);
            k = __popc(mask);
            if (k != longest) {
                out.x = sweep_room(st, slab, has_slab, k, lane);
                if (out.x == ~0ull) k = 0;
                else if (keep) st.pool[out.x + __popc(mask & ((1u << lane) - 1u))] = v;
            }
        } else {
            for (int i = lane; i < kWarpHash; i += 32) sh.table[w][i] = kNone;
            if (lane == 0) sh.count[w] = 0;
            __syncwarp();
            auto insert = [&](uint32_t x) {
                unsigned h = (x * 2654435761u) >> (32 - 8);  // kWarpHash = 2^8 slots
                for (int probe = 0; probe < kWarpHash; ++probe, h = (h + 1) & (kWarpHash - 1)) {
                    const uint32_t prev = atomicCAS(&sh.table[w][h], kNone, x);
                    if (prev == x) return true;
                    if (prev == kNone) return atomicAdd(&sh.count[w], 1u) < static_cast<unsigned>(kWarpCap);
                }
                return false;
            };
            bool fits = true;
            for (uint32_t u0 = 0; u0 < total; u0 += 32) {
                const uint32_t x = warp_element<RUN>(st, u0 + lane, excl, s.x, total);
                if (x != kNone) fits = insert(x);
                if (!__all_sync(0xFFFFFFFFu, fits)) return false;  // more distinct elements than a warp sorts
            }
            if (seed != kNone && lane == 0) fits = insert(seed);
            if (!__all_sync(0xFFFFFFFFu, fits)) return false;
            __syncwarp();
            k = sh.count[w];
            __syncwarp();
            if (k != longest || seed != kNone) {  // a new set: sorted, then written
                if (lane == 0) sh.count[w] = 0;
                __syncwarp();
                for (int i = lane; i < kWarpHash; i += 32) {
                    const uint32_t x = sh.table[w][i];
                    if (x != kNone) sh.sorted[w][atomicAdd(&sh.count[w], 1u)] = x;
                }
                __syncwarp();
                out.x = sweep_room(st, slab, has_slab, k, lane);
                const bool room = out.x != ~0ull;
                if (k <= 32) {
                    const uint32_t v = warp_bitonic(lane < k ? sh.sorted[w][lane] : kNone, lane);
                    if (room && lane < k) st.pool[out.x + lane] = v;
                } else {  // each element's rank among the k
                    for (uint32_t i = lane; i < k; i += 32) {
                        const uint32_t x = sh.sorted[w][i];
                        uint32_t below = 0;
                        for (uint32_t t = 0; t < k; ++t) below += sh.sorted[w][t] < x ? 1u : 0u;
                        if (room) st.pool[out.x + below] = x;
                    }
                }
                if (!room) k = 0;
                __syncwarp();
            }
        }
    }
    if (lane == 0) {
        st.seed[p] = seed;
        out.y = (static_cast<unsigned long long>(k) << 32) | min(own, mp);
        st.set[p] = out;
    }
    return true;
}

// One plateau by the whole block (uniform arguments).
template <bool RUN, int W>
__device__ void sweep_block(const PlateauSets& st, SweepShared<W>& sh, uint32_t p, unsigned long long level) {
    const unsigned tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const unsigned e0 = __ldg(st.eoff + p), e1 = __ldg(st.eoff + p + 1);
    constexpr int kSlots = SweepShared<W>::kSlots;
    for (int i = tid; i < kSlots; i += W * 32) sh.btable[i] = kNone;
    for (int i = tid; i < kSetHash; i += W * 32) sh.seen[i] = ~0ull;
    if (tid == 0) sh.bcount = sh.bover = 0;
    __syncthreads();
    auto insert = [&](uint32_t x) {
        unsigned h = (x * 2654435761u) >> (32 - SweepShared<W>::kBits);
        for (int probe = 0; probe < kSlots; ++probe, h = (h + 1) & (kSlots - 1)) {
            uint32_t prev = *reinterpret_cast<volatile uint32_t*>(&sh.btable[h]);
            if (prev == kNone) prev = atomicCAS(&sh.btable[h], kNone, x);
            if (prev == x) return;
            if (prev == kNone) {
                if (atomicAdd(&sh.bcount, 1u) >= static_cast<unsigned>(SweepShared<W>::kCap)) sh.bover = 1;
                return;
            }
        }
        sh.bover = 1;
    };
    const bool spread = e1 - e0 > kHardDegree;  // too many edges for one block: only its seed is found here
    uint32_t mp = kNone;
    unsigned long long longest = 0, sum = 0;  // a longest set: length << 32 | lane's edge; all lengths
    for (unsigned eb = e0 + w * 32; eb < e1; eb += W * 32) {
        ulonglong2 s = make_ulonglong2(~0ull, kNone);
        if (eb + lane < e1) {
            const uint32_t q = __ldg(st.edges + eb + lane);
            s = RUN ? ldcg_set(st.set + q) : __ldg(st.set + q);
        }
        uint32_t len = set_len(s);
        mp = min(mp, static_cast<uint32_t>(s.y));
        sum += len;
        // sizes only; other warps set the flag meanwhile, so the warp decides by a vote
        if (spread || __any_sync(0xFFFFFFFFu, *reinterpret_cast<volatile unsigned int*>(&sh.bover))) continue;
        const unsigned peers = __match_any_sync(0xFFFFFFFFu, len ? s.x : ~0ull);
        if (len && static_cast<int>(lane) != __ffs(peers) - 1) len = 0;
        if (len) {  // sets the block has seen already
            unsigned h = static_cast<unsigned>((s.x * 0x9E3779B97F4A7C15ull) >> 55);  // kSetHash = 2^9 slots
            for (int probe = 0; probe < 4; ++probe, h = (h + 1) & (kSetHash - 1)) {
                const unsigned long long prev = atomicCAS(&sh.seen[h], ~0ull, s.x);
                if (prev == s.x) len = 0;
                if (prev == ~0ull || prev == s.x) break;
            }
            longest = max(longest, (static_cast<unsigned long long>(len) << 32) | (eb + lane - e0));
        }
        uint32_t total;
        const uint32_t excl = warp_exclusive(len, lane, total);
        for (uint32_t u0 = 0; u0 < total; u0 += 32) {
            const uint32_t x = warp_element<RUN>(st, u0 + lane, excl, s.x, total);
            if (x != kNone) insert(x);
            if (__any_sync(0xFFFFFFFFu, *reinterpret_cast<volatile unsigned int*>(&sh.bover))) break;
        }
    }
    mp = __reduce_min_sync(0xFFFFFFFFu, mp);
    for (int o = 16; o > 0; o >>= 1) {
        longest = max(longest, __shfl_xor_sync(0xFFFFFFFFu, longest, o));
        sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
    }
    if (lane == 0) {
        sh.wmin[w] = mp;
        sh.wmax[w] = longest;
        sh.wsum[w] = sum;
    }
    __syncthreads();
    for (int i = 0; i < W; ++i) {
        mp = min(mp, sh.wmin[i]);
        longest = max(longest, sh.wmax[i]);
    }
    const uint32_t own = __ldg(st.minrank + p);
    const uint32_t seed = own < mp ? own : kNone;
    const uint32_t m = min(own, mp);
    if (tid == 0 && seed != kNone) insert(seed);
    __syncthreads();
    if (sh.bover || spread) {  // the host merges it
        if (tid == 0) {
            unsigned long long all = seed != kNone ? 1 : 0;
            for (int i = 0; i < W; ++i) all += sh.wsum[i];
            st.seed[p] = seed;
            st.set[p] = make_ulonglong2(0, m);
            st.hard[atomicAdd(&st.info[1], 1ull)] = p;
            atomicAdd(&st.info[2], all);
            atomicMin(&st.info[0], level);
        }
        __syncthreads();
        return;
    }
    const uint32_t k = sh.bcount;
    __syncthreads();  // all have read the count
    if (k == static_cast<uint32_t>(longest >> 32) && seed == kNone) {  // a predecessor's set
        if (tid == 0) {
            const uint32_t q = __ldg(st.edges + e0 + static_cast<uint32_t>(longest));
            const ulonglong2 s = RUN ? ldcg_set(st.set + q) : __ldg(st.set + q);
            st.seed[p] = seed;
            st.set[p] = make_ulonglong2(s.x, (static_cast<unsigned long long>(k) << 32) | m);
        }
        __syncthreads();
        return;
    }
    if (tid == 0) {
        sh.bcount = 0;
        const unsigned long long at = atomicAdd(st.pool_n, static_cast<unsigned long long>(k));
        const bool fits = at + k <= st.pool_cap;
        if (!fits) atomicOr(st.err, 2u);
        sh.place = fits ? at : ~0ull;
        st.seed[p] = seed;
        st.set[p] = make_ulonglong2(fits ? at : 0ull, (static_cast<unsigned long long>(fits ? k : 0u) << 32) | m);
    }
    __syncthreads();
    for (int i = tid; i < kSlots; i += W * 32) {
        const uint32_t x = sh.btable[i];
        if (x != kNone) sh.bsorted[atomicAdd(&sh.bcount, 1u)] = x;
    }
    __syncthreads();
    const unsigned long long place = sh.place;
    if (place != ~0ull) {  // each element's rank among the k
        for (uint32_t i = tid; i < k; i += W * 32) {
            const uint32_t x = sh.bsorted[i];
            uint32_t below = 0;
            for (uint32_t t = 0; t < k; ++t) below += sh.bsorted[t] < x ? 1u : 0u;
            st.pool[place + below] = x;
        }
    }
    __syncthreads();
}

// Levels l0 .. l1 - 1 (starts: the position in `order` of each level's first plateau): one level
// over the grid, or (RUN) several by one block. Returns at once behind a level that stopped.
template <bool RUN, int W>
__global__ void __launch_bounds__(W * 32) level_sweep(PlateauSets st, const uint32_t* __restrict__ starts, unsigned l0,
                                                      unsigned l1) {
    __shared__ SweepShared<W> sh;
    const unsigned lane = threadIdx.x & 31, w = threadIdx.x >> 5, id = blockIdx.x * W + w;
    const bool has_slab = id < st.nslab;
    ulonglong2 slab = has_slab ? st.slab[id] : make_ulonglong2(0, 0);
    for (unsigned l = l0; l < l1; ++l) {
        if (__ldcg(st.info) < l) break;  // uniform: written by an earlier launch, or before a block barrier
        const uint32_t b = __ldg(starts + l), e = __ldg(starts + l + 1);
        if (threadIdx.x == 0) sh.nlist = 0;
        __syncthreads();
        for (uint32_t i = b + id; i < e; i += gridDim.x * W) {
            const uint32_t p = __ldg(st.order + i);
            if (!sweep_plateau<RUN, W>(st, sh, p, slab, has_slab) && lane == 0) sh.list[atomicAdd(&sh.nlist, 1u)] = p;
            __syncwarp();
        }
        __syncthreads();
        const unsigned n = sh.nlist;
        for (unsigned k = 0; k < n; ++k) sweep_block<RUN, W>(st, sh, sh.list[k], l);
        __syncthreads();
    }
    if (has_slab && lane == 0) st.slab[id] = slab;
}

__global__ void unpack_sets(const ulonglong2* __restrict__ set, size_t np, unsigned long long* __restrict__ soff,
                            uint32_t* __restrict__ slen) {
    PMA_GRID_STRIDE(p, np) {
        const ulonglong2 s = set[p];
        soff[p] = s.x;
        slen[p] = set_len(s);
    }
}

// --- hard sets: unions too large for a block ---
//
// Every element of every predecessor set (and the own seed) becomes a key (hard set << shift |
// rank); sorting and removing duplicates yields each union. Keys are 32-bit whenever ranks and
// set indices fit together, else 64-bit, and the radix sort covers the used bits only.
__global__ void level_hard_degrees(PlateauSets st, unsigned long long* __restrict__ deg) {
    const unsigned long long nh = st.info[1];
    PMA_GRID_STRIDE(b, nh) {
        const uint32_t p = st.hard[b];
        deg[b] = st.eoff[p + 1] - st.eoff[p];
    }
}

// One thread per in-edge of a hard plateau (t over the concatenated edge lists, doff = the
// exclusive scan of the in-degrees): a giant plateau with a million in-edges is spread over
// the whole GPU instead of one block. The in-edges of a block mostly belong to one plateau and
// bring the same seeds many times, so each block keeps only the first copy of a key (shared-
// memory hash set; a key that finds no free slot is emitted anyway, the sort and unique that
// follow are exact). Keys of a warp are placed with one atomic.
constexpr int kMergeTable = 2048;

template <class K>
__global__ void __launch_bounds__(256) level_expand(PlateauSets st,
                                                    const unsigned long long* __restrict__ doff,
                                                    const unsigned long long* __restrict__ deg,
                                                    unsigned long long nhard, K* __restrict__ keys,
                                                    unsigned long long cap, int shift) {
    __shared__ K table[kMergeTable];
    const unsigned lane = threadIdx.x & 31, lt = (1u << lane) - 1u;
    const unsigned long long total = doff[nhard - 1] + deg[nhard - 1];
    const unsigned long long stride = static_cast<unsigned long long>(gridDim.x) * blockDim.x;
    const K empty = ~static_cast<K>(0);
    // block-uniform trip count (the table is cleared between rounds)
    for (unsigned long long tb = blockIdx.x * static_cast<unsigned long long>(blockDim.x); tb < total;
         tb += stride) {
        for (int i = threadIdx.x; i < kMergeTable; i += blockDim.x) table[i] = empty;
        __syncthreads();
        const unsigned long long t = tb + threadIdx.x;
        uint32_t len = 0;
        const uint32_t* src = st.pool;
        K hi = 0;
        if (t < total) {
            unsigned long long lo = 0, up = nhard;  // last b with doff[b] <= t
            while (up - lo > 1) {
                const unsigned long long mid = (lo + up) >> 1;
                if (doff[mid] <= t) lo = mid;
                else up = mid;
            }
            const uint32_t p = st.hard[lo];
            const ulonglong2 set = __ldg(st.set + __ldg(st.edges + st.eoff[p] + (t - doff[lo])));
            len = set_len(set);
            src = st.pool + set.x;
            hi = static_cast<K>(lo) << shift;
        }
        // The warp's 32 sets are expanded together, 32 elements per round: element u of the
        // concatenation belongs to the last lane whose exclusive offset is <= u (a shuffle
        // binary search), so one long set does not hold the warp for its whole length.
        uint32_t incl = len;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t2 = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= static_cast<unsigned>(o)) incl += t2;
        }
        const uint32_t excl = incl - len;
        const uint32_t wtotal = __shfl_sync(0xFFFFFFFFu, incl, 31);
        for (uint32_t u0 = 0; u0 < wtotal; u0 += 32) {
            const uint32_t u = u0 + lane;
            int owner = 0;
            for (int step = 16; step >= 1; step >>= 1) {
                const uint32_t e = __shfl_sync(0xFFFFFFFFu, excl, owner + step);
                if (e <= u) owner += step;
            }
            const uint32_t* osrc = reinterpret_cast<const uint32_t*>(
                __shfl_sync(0xFFFFFFFFu, reinterpret_cast<unsigned long long>(src), owner));
            const K ohi = __shfl_sync(0xFFFFFFFFu, hi, owner);
            const uint32_t oexcl = __shfl_sync(0xFFFFFFFFu, excl, owner);
            K key = 0;
            bool emit = false;
            if (u < wtotal) {
                key = ohi | static_cast<K>(__ldg(osrc + (u - oexcl)));
                emit = true;
                unsigned h = static_cast<unsigned>((static_cast<unsigned long long>(key) * 0x9E3779B97F4A7C15ull) >> 40) &
                             (kMergeTable - 1);
                for (int probe = 0; probe < 8; ++probe, h = (h + 1) & (kMergeTable - 1)) {
                    const K prev = atomicCAS(&table[h], empty, key);
                    if (prev == empty) break;
                    if (prev == key) {
                        emit = false;
                        break;
                    }
                }
            }
            const unsigned m = __ballot_sync(0xFFFFFFFFu, emit);
            if (!m) continue;
            const int leader = __ffs(m) - 1;
            unsigned long long pos = 0;
            if (static_cast<int>(lane) == leader) pos = atomicAdd(&st.info[3], static_cast<unsigned long long>(__popc(m)));
            pos = __shfl_sync(0xFFFFFFFFu, pos, leader) + __popc(m & lt);
            if (emit && pos < cap) keys[pos] = key;
        }
        __syncthreads();
    }
    // own seeds
    for (unsigned long long b = blockIdx.x * static_cast<unsigned long long>(blockDim.x) + threadIdx.x; b < nhard;
         b += stride) {
        const uint32_t p = st.hard[b];
        if (st.seed[p] == kNone) continue;
        const unsigned long long pos = atomicAdd(&st.info[3], 1ull);
        if (pos < cap) keys[pos] = (static_cast<K>(b) << shift) | static_cast<K>(st.seed[p]);
    }
}

// Sizes and first positions of the merged unions (keys sorted, duplicates removed).
template <class K>
__global__ void level_runs(const K* __restrict__ keys, size_t n, PlateauSets st, int shift) {
    PMA_GRID_STRIDE(i, n) {
        const size_t b = static_cast<size_t>(keys[i] >> shift);
        if (i == 0 || static_cast<size_t>(keys[i - 1] >> shift) != b) st.first[b] = i;
        atomicAdd(&st.cnt[b], 1ull);
    }
}

__global__ void level_place_hard(PlateauSets st, size_t nhard) {
    PMA_GRID_STRIDE(b, nhard) {
        const uint32_t p = st.hard[b];
        const unsigned long long k = st.cnt[b], at = atomicAdd(st.pool_n, k);
        const bool fits = at + k <= st.pool_cap;
        if (!fits) atomicOr(st.err, 2u);
        const unsigned long long m = st.set[p].y & 0xFFFFFFFFull;
        st.set[p] = make_ulonglong2(fits ? at : 0ull, ((fits ? k : 0ull) << 32) | m);
    }
}

template <class K>
__global__ void level_copy_hard(const K* __restrict__ keys, size_t n, PlateauSets st, int shift) {
    const K low = (static_cast<K>(1) << shift) - 1;
    PMA_GRID_STRIDE(i, n) {
        const size_t b = static_cast<size_t>(keys[i] >> shift);
        const ulonglong2 s = st.set[st.hard[b]];
        const unsigned long long r = i - st.first[b];  // rank within the set
        if (set_len(s) == 0) continue;  // no room in the pool: the sweep is redone
        if (r >= set_len(s)) {  // keys and set bounds disagree: never write outside the set
            atomicOr(st.err, 32u);
            continue;
        }
        st.pool[s.x + r] = static_cast<uint32_t>(keys[i] & low);
    }
}

__global__ void throat_hashes(const unsigned long long* __restrict__ soff, const uint32_t* __restrict__ slen,
                              const uint32_t* __restrict__ pool, const uint32_t* __restrict__ multi,
                              size_t nm, unsigned long long* __restrict__ h1o,
                              unsigned long long* __restrict__ h2o) {
    PMA_GRID_STRIDE(i, nm) {
        const uint32_t p = multi[i];
        unsigned long long a, b;
        list_hash(pool + soff[p], slen[p], a, b);
        h1o[i] = a;
        h2o[i] = b;
    }
}

__global__ void flag_multi(const uint32_t* __restrict__ slen, size_t np, uint8_t* __restrict__ f) {
    PMA_GRID_STRIDE(p, np) f[p] = slen[p] >= 2;
}

// Group starts among plateaus sorted by (h1, h2); verifies list equality within groups.
__global__ void group_starts(const uint32_t* __restrict__ sorted_p, const unsigned long long* __restrict__ h1,
                             const unsigned long long* __restrict__ h2, size_t nm,
                             const unsigned long long* __restrict__ soff, const uint32_t* __restrict__ slen,
                             const uint32_t* __restrict__ pool, uint32_t* __restrict__ start,
                             unsigned int* __restrict__ err) {
    PMA_GRID_STRIDE(i, nm) {
        bool s = (i == 0) || h1[i] != h1[i - 1] || h2[i] != h2[i - 1];
        // equal first hashes, different second ones: sorted by the first hash alone, such sets
        // may interleave (the host then sorts by both)
        if (i > 0 && h1[i] == h1[i - 1] && h2[i] != h2[i - 1]) atomicOr(err, 64u);
        if (!s) {
            const uint32_t a = sorted_p[i], b = sorted_p[i - 1];
            bool eq = slen[a] == slen[b];
            for (uint32_t k = 0; eq && k < slen[a]; ++k) eq = pool[soff[a] + k] == pool[soff[b] + k];
            if (!eq) atomicOr(err, 4u);  // 128-bit hash collision between different sets
        }
        start[i] = s ? 1u : 0u;
    }
}

struct GroupOut {
    unsigned long long* gvol;       // per group
    unsigned long long* gfirst;     // per group: smallest root voxel index
    uint32_t* grep;                 // per group: representative plateau
};

__global__ void group_reduce(const uint32_t* __restrict__ sorted_p, const uint32_t* __restrict__ gid,
                             size_t nm, const unsigned int* __restrict__ psize,
                             const uint32_t* __restrict__ roots, GroupOut go,
                             uint32_t* __restrict__ plateau_group) {
    PMA_GRID_STRIDE(i, nm) {
        const uint32_t p = sorted_p[i];
        const uint32_t gr = gid[i];
        plateau_group[p] = gr;
        atomicAdd(&go.gvol[gr], static_cast<unsigned long long>(psize[p]));
        atomicMin(&go.gfirst[gr], static_cast<unsigned long long>(roots[p]));
        if (i == 0 || gid[i - 1] != gr) go.grep[gr] = p;
    }
}

struct PoreAcc {
    const uint32_t* rank2pore;       // ball rank -> pore index (kNone if not a seed)
    unsigned long long* pvol;
    unsigned int* pbound;
};

__global__ void pore_accumulate(const unsigned long long* __restrict__ soff, const uint32_t* __restrict__ slen,
                                const uint32_t* __restrict__ pool, const unsigned int* __restrict__ psize,
                                const unsigned int* __restrict__ pface, size_t np, PoreAcc pa) {
    const unsigned lane = threadIdx.x & 31;
    PMA_GRID_STRIDE(p, np) {
        const uint32_t n = slen[p];
        const uint32_t* s = pool + soff[p];
        // plateaus of one pore met by a warp add their sizes with one atomic
        const uint32_t pore = n == 1 ? pa.rank2pore[s[0]] : kNone;
        const unsigned long long size = n == 1 ? psize[p] : 0ull;
        const unsigned peers = __match_any_sync(__activemask(), pore);
        unsigned long long sum = 0;
        for (unsigned m = peers; m; m &= m - 1) sum += __shfl_sync(peers, size, __ffs(m) - 1);
        if (pore != kNone && static_cast<int>(lane) == __ffs(peers) - 1) atomicAdd(&pa.pvol[pore], sum);
        if (pface[p])
            for (uint32_t k = 0; k < n; ++k) pa.pbound[pa.rank2pore[s[k]]] = 1;
    }
}

__global__ void plateau_labels(const unsigned long long* __restrict__ soff, const uint32_t* __restrict__ slen,
                               const uint32_t* __restrict__ pool, const uint32_t* __restrict__ rank2id,
                               const uint32_t* __restrict__ plateau_group,
                               const uint32_t* __restrict__ group_tid, size_t np,
                               uint32_t* __restrict__ plabel) {
    PMA_GRID_STRIDE(p, np) {
        const uint32_t n = slen[p];
        uint32_t lab = 0;
        if (n == 1) lab = rank2id[pool[soff[p]]];
        else if (n >= 2) lab = group_tid[plateau_group[p]];
        plabel[p] = lab;
    }
}

__global__ void voxel_labels(const uint32_t* __restrict__ pid, const uint32_t* __restrict__ plabel,
                             size_t n, uint32_t* __restrict__ labels) {
    PMA_GRID_STRIDE(v, n) {
        const uint32_t p = pid[v];
        labels[v] = (p == kNone) ? 0u : plabel[p];
    }
}

// Old -> new label remap by binary search in sorted old ids.
__global__ void remap_labels(uint32_t* __restrict__ labels, size_t n, const uint32_t* __restrict__ old_ids,
                             const uint32_t* __restrict__ new_ids, uint32_t m) {
    const uint32_t first = m ? old_ids[0] : 0xFFFFFFFFu;  // pore labels are below every type id
    PMA_GRID_STRIDE(v, n) {
        const uint32_t l = labels[v];
        if (l == 0 || l < first || m == 0) continue;
        uint32_t lo = 0, hi = m;
        while (lo < hi) {
            const uint32_t mid = (lo + hi) >> 1;
            if (old_ids[mid] < l) lo = mid + 1;
            else hi = mid;
        }
        if (lo < m && old_ids[lo] == l) labels[v] = new_ids[lo];
    }
}

__global__ void to_group_index(const uint32_t* __restrict__ excl, const uint32_t* start, size_t m,
                               uint32_t* out) {
    PMA_GRID_STRIDE(i, m) out[i] = excl[i] + start[i] - 1u;
}

// A type's pore ids in processing order, [second, first, third, ...] of its seed list in ascending ranks,
// which are ascending ids (BasePoreAndThroatComputer.cpp:338-340, 370-371).
struct SeedLists {
    const uint32_t* grep;
    const unsigned long long* soff;
    const uint32_t* slen;
    const uint32_t* pool;
    const uint32_t* rank2id;
    __device__ __forceinline__ uint32_t length(uint32_t g) const { return slen[grep[g]]; }
    __device__ __forceinline__ uint32_t pore(uint32_t g, uint32_t j) const {
        return rank2id[pool[soff[grep[g]] + (j < 2 ? 1 - j : j)]];
    }
};

// Keys that order the types: (last pore, first voxel) (BasePoreAndThroatComputer.cpp:122-130). Both fit 32
// bits, and the first voxels are distinct. In place of the first voxels.
__global__ void type_keys(SeedLists lists, size_t ng, unsigned long long* __restrict__ first_voxel) {
    PMA_GRID_STRIDE(g, ng) {
        const uint32_t p = lists.grep[g];  // lists of at least two: the last seed is the last pore
        const uint32_t last = lists.rank2id[lists.pool[lists.soff[p] + lists.slen[p] - 1]];
        first_voxel[g] = (static_cast<unsigned long long>(last) << 32) | (first_voxel[g] & 0xFFFFFFFFull);
    }
}

template <class T>
T* buf(pma_ctx* ctx, const char* tag, size_t count) {
    return static_cast<T*>(ctx->scratch(tag, std::max<size_t>(count, 1) * sizeof(T)));
}

}  // namespace

void reference_type_ids(pma_ctx* ctx, pma_table* t, uint32_t* labels, const uint32_t* crad2, pma_dims d,
                        pma_stencil st);

pma_table* pores(pma_ctx* ctx, const uint8_t* mask, const uint32_t* edt2, const uint32_t* crad2,
                 pma_dims d, pma_stencil st, uint32_t* labels) {
    KernelTimer kt_stage(ctx, "stage_pores");  // the whole stage, for the untimed remainder
    check_dims(d);
    PMA_REQUIRE(mask && edt2 && crad2 && labels, PMA_ERR_ARGUMENT, "pma_pores: null device pointer");
    cudaStream_t s = ctx->stream;
    const size_t n = voxels(d);
    const Grid g{d.sx, d.sy, d.sz};
    const int d3q7 = st == PMA_D3Q7 ? 1 : 0;
    const unsigned G = grid_for(ctx, n);
    int64_t* d_count = buf<int64_t>(ctx, "pores.count", 4);
    unsigned int* err = reinterpret_cast<unsigned int*>(d_count + 2);
    PMA_CUDA(cudaMemsetAsync(d_count, 0, 32, s));

    // a8: maximum balls in z, x, y scan order (PoreAndThroatComputer.cpp:93-119) = linear order.
    uint8_t* flags = buf<uint8_t>(ctx, "pores.flags", n);
    flag_outer<<<G, 256, 0, s>>>(mask, n, flags);
    ctx->check_launch("flag_outer");
    uint32_t* balls = buf<uint32_t>(ctx, "pores.balls", n);
    const int64_t nb = select_flagged(ctx, thrust::counting_iterator<uint32_t>(0), flags, balls,
                                      static_cast<int64_t>(n), d_count);
    uint32_t* ball_r2 = buf<uint32_t>(ctx, "pores.ball_r2", nb);
    if (nb) {
        gather_u32<<<grid_for(ctx, nb), 256, 0, s>>>(edt2, balls, nb, ball_r2);
        ctx->check_launch("gather_u32");
    }
    // std::sort with the reference's comparator (PoreAndThroatComputer.cpp:121-122): the items are
    // 8-byte (r2, voxel index) pairs compared on r2 alone. std::sort's moves depend only on
    // comparison results, so the permutation equals the one the reference's 16-byte balls go
    // through, and the sorted items carry each rank's voxel.
    auto* items = buf<unsigned long long>(ctx, "pores.d_items", nb);
    uint32_t* pid = buf<uint32_t>(ctx, "pores.pid", n);      // root voxel, then plateau id
    uint32_t* crank = buf<uint32_t>(ctx, "pores.crank", n);  // both are the sort's scratch first
    if (nb) {
        KernelTimer kt(ctx, "pores_sort");
        auto pack = [&] {
            pack_items<<<grid_for(ctx, nb), 256, 0, s>>>(ball_r2, balls, nb, items);
            ctx->check_launch("pack_items");
        };
        pack();
        if (!ordered_sort_device(ctx, items, nb, pid, crank)) {
            // a range reached std::sort's depth limit (an adversary's order; none is known from a volume):
            // libstdc++'s own routines on the host, on up to 16 threads
            pack();
            std::vector<unsigned long long> h(nb);
            PMA_CUDA(cudaMemcpyAsync(h.data(), items, nb * 8, cudaMemcpyDeviceToHost, s));
            ctx->sync();
            int levels = 0;
            while (levels < 4 && (2u << levels) <= std::thread::hardware_concurrency()) ++levels;
            ordered_sort(
                h.data(), h.data() + nb, [](unsigned long long x, unsigned long long y) { return (x >> 32) > (y >> 32); }, levels);
            PMA_CUDA(cudaMemcpyAsync(items, h.data(), nb * 8, cudaMemcpyHostToDevice, s));
            ctx->sync();
        }
    }

    // Plateaus: connected sets of equal crad under the stencil.
    const unsigned pair_grid = static_cast<unsigned>(std::min<size_t>(
        static_cast<size_t>(div_up(d.sy, kTileY)) * div_up(d.sx, kTileX) * div_up(d.sz, kTileZ), ctx->num_sms * 32ull));
    uf_init<<<G, 256, 0, s>>>(crad2, g, n, d3q7, pid);
    ctx->check_launch("uf_init");
    {
        KernelTimer kt(ctx, "uf_jump");
        if (n >= kJumpMinVoxels) {
            unsigned int* changed =
                reinterpret_cast<unsigned int*>(buf<unsigned long long>(ctx, "pores.jump", kJumpPasses));
            PMA_CUDA(cudaMemsetAsync(changed, 0, kJumpPasses * 4, s));
            for (int pass = 0; pass < kJumpPasses; ++pass) uf_jump<<<G, 256, 0, s>>>(n, pid, changed, pass);
            ctx->count_launch(kJumpPasses - 1);
            ctx->check_launch("uf_jump");
        }
    }
    {
        KernelTimer kt(ctx, "uf_hook");
        if (n >= kJumpMinVoxels) {
            // parent pairs, then their unions (the buffer grows to what a call needed)
            auto* pcount = reinterpret_cast<unsigned long long*>(d_count + 1);  // free until the edges
            unsigned long long pcap = std::max<unsigned long long>(
                std::max<unsigned long long>(n / 64, 1ull << 20), ctx->cached_bytes("pores.uf_pairs") / 8);
            unsigned long long npairs = 0;
            unsigned long long* pairs = nullptr;
            for (int attempt = 0;; ++attempt) {
                pairs = buf<unsigned long long>(ctx, "pores.uf_pairs", pcap);
                PMA_CUDA(cudaMemsetAsync(pcount, 0, 8, s));
                voxel_pairs<true><<<pair_grid, kPairThreads, 0, s>>>(pid, crad2, g, d3q7, 0, pcount, pairs, pcap);
                ctx->check_launch("voxel_pairs");
                PMA_CUDA(cudaMemcpyAsync(&npairs, pcount, 8, cudaMemcpyDeviceToHost, s));
                ctx->sync();
                if (npairs <= pcap) break;
                PMA_REQUIRE(attempt < 3, PMA_ERR_INTERNAL, "pma_pores: plateau pair count did not settle");
                pcap = npairs + npairs / 8 + 1024;
            }
            if (npairs) {
                uf_union_pairs<<<grid_for(ctx, npairs), 256, 0, s>>>(pairs, npairs, pid, err,
                                                                      ctx->limits.union_limit);
                ctx->check_launch("uf_union_pairs");
            }
        } else {
            uf_hook<<<G, 256, 0, s>>>(crad2, g, n, d3q7, pid, err, ctx->limits.union_limit);
        }
    }
    ctx->check_launch("uf_hook");
    auto kt_ids = std::make_unique<KernelTimer>(ctx, "plateau_ids");
    uf_flatten<<<G, 256, 0, s>>>(n, pid);
    ctx->check_launch("uf_flatten");
    flag_roots<<<G, 256, 0, s>>>(pid, n, flags);
    ctx->check_launch("flag_roots");
    uint32_t* roots = buf<uint32_t>(ctx, "pores.roots", n);
    const int64_t np = select_flagged(ctx, thrust::counting_iterator<uint32_t>(0), flags, roots,
                                      static_cast<int64_t>(n), d_count);
    if (np) {
        scatter_pid<<<grid_for(ctx, np), 256, 0, s>>>(roots, np, labels);  // labels as scratch
        ctx->check_launch("scatter_pid");
        to_pid<<<G, 256, 0, s>>>(labels, n, np, pid, err);
        ctx->check_launch("to_pid");
    }
    {
        // the union-find's own bound (bit 1) is read here: the level sweep reuses the word
        unsigned int h_err = 0;
        PMA_CUDA(cudaMemcpyAsync(&h_err, err, 4, cudaMemcpyDeviceToHost, s));
        ctx->sync();
        PMA_REQUIRE(!(h_err & 1u), PMA_ERR_LIMIT, "pma_pores: plateau union-find did not converge");
        PMA_REQUIRE(!(h_err & 8u), PMA_ERR_INTERNAL, "pma_pores: plateau labelling left a non-root parent");
    }
    kt_ids.reset();
    // Edges between plateaus, sorted by destination.
    auto kt_edges = std::make_unique<KernelTimer>(ctx, "plateau_edges");
    int sb = 1;  // bits of a plateau id
    while (sb < 32 && (1ull << sb) < static_cast<unsigned long long>(np)) ++sb;
    auto* ecount = reinterpret_cast<unsigned long long*>(d_count + 1);
    // One pass writes the edges into a buffer of at least n/8 entries, or of what an earlier
    // call needed (the edges kept after the per-block de-duplication are far fewer than the
    // voxels); when they do not fit, the pass is repeated with the size it counted.
    unsigned long long ecap = std::max<unsigned long long>(
        std::max<unsigned long long>(n / 8, 1ull << 20), ctx->cached_bytes("pores.edges_raw") / 8);
    unsigned long long* edges_raw = nullptr;
    unsigned long long ne_kept = 0;
    for (int attempt = 0;; ++attempt) {
        edges_raw = buf<unsigned long long>(ctx, "pores.edges_raw", ecap);
        PMA_CUDA(cudaMemsetAsync(ecount, 0, 8, s));
        {
            KernelTimer kt(ctx, "edges_write");
            voxel_pairs<false><<<pair_grid, kPairThreads, 0, s>>>(pid, crad2, g, d3q7, sb, ecount, edges_raw, ecap);
        }
        ctx->check_launch("voxel_pairs");
        PMA_CUDA(cudaMemcpyAsync(&ne_kept, ecount, 8, cudaMemcpyDeviceToHost, s));
        ctx->sync();
        if (ne_kept <= ecap) break;
        PMA_REQUIRE(attempt < 3, PMA_ERR_INTERNAL, "pma_pores: plateau edge count did not settle");
        ecap = ne_kept + ne_kept / 8 + 1024;
    }
    // Keys are (destination << sb | source): sorting groups the predecessors of each plateau.
    int64_t ne = 0;
    if (ne_kept) {
        auto* edges = buf<unsigned long long>(ctx, "pores.edges", ne_kept);
        sort_keys(ctx, edges_raw, edges, static_cast<int64_t>(ne_kept), 2 * sb);  // used bits only
        ne = unique(ctx, edges, edges_raw, static_cast<int64_t>(ne_kept), d_count);
    }
    ctx->count("pores.plateaus", static_cast<double>(np));
    ctx->count("pores.plateau_edges", static_cast<double>(ne));
    ctx->count("pores.plateau_edges_written", static_cast<double>(ne_kept));
    uint32_t* by_dst = buf<uint32_t>(ctx, "pores.esrc", std::max<int64_t>(ne, 1));
    unsigned int* eoff = buf<unsigned int>(ctx, "pores.eoff", np + 1);
    PMA_CUDA(cudaMemsetAsync(eoff, 0, (np + 1) * 4, s));
    edge_offsets<<<grid_for(ctx, ne + 1), 256, 0, s>>>(edges_raw, ne, np, sb, eoff, by_dst);
    ctx->check_launch("edge_offsets");
    kt_edges.reset();

    auto kt_stats = std::make_unique<KernelTimer>(ctx, "plateau_stats");
    fill_u32<<<G, 256, 0, s>>>(crank, n, kNone);
    ctx->check_launch("fill_u32");
    if (nb) {
        scatter_rank<<<grid_for(ctx, nb), 256, 0, s>>>(items, nb, crank);
        ctx->check_launch("scatter_rank");
    }
    uint32_t* pcrad = buf<uint32_t>(ctx, "pores.pcrad", np);
    unsigned int* psize = buf<unsigned int>(ctx, "pores.psize", np);
    unsigned int* pface = buf<unsigned int>(ctx, "pores.pface", np);
    uint32_t* pminrank = buf<uint32_t>(ctx, "pores.pminrank", np);
    PMA_CUDA(cudaMemsetAsync(psize, 0, std::max<int64_t>(np, 1) * 4, s));
    PMA_CUDA(cudaMemsetAsync(pface, 0, std::max<int64_t>(np, 1) * 4, s));
    fill_u32<<<grid_for(ctx, np), 256, 0, s>>>(pminrank, np, kNone);
    ctx->check_launch("fill_u32");
    plateau_stats<<<G, 256, 0, s>>>(pid, crad2, crank, g, n, pcrad, psize, pface, pminrank);
    ctx->check_launch("plateau_stats");
    kt_stats.reset();

    // Levels: plateaus in decreasing crad.
    uint32_t* lkey = buf<uint32_t>(ctx, "pores.lkey", np);
    uint32_t* lval = buf<uint32_t>(ctx, "pores.lval", np);
    uint32_t* lkey2 = buf<uint32_t>(ctx, "pores.lkey2", np);
    uint32_t* order = buf<uint32_t>(ctx, "pores.order", np);
    std::vector<size_t> level_begin;
    if (np) {
        KernelTimer kt(ctx, "level_order");
        level_keys<<<grid_for(ctx, np), 256, 0, s>>>(pcrad, np, lkey, lval);
        ctx->check_launch("level_keys");
        sort_pairs(ctx, lkey, lkey2, lval, order, np);
        // first position of each level, found on the device (a few hundred of np positions)
        level_starts<<<grid_for(ctx, np), 256, 0, s>>>(lkey2, np, flags);
        ctx->check_launch("level_starts");
        const int64_t nl = select_flagged(ctx, thrust::counting_iterator<uint32_t>(0), flags, lval, np, d_count);
        std::vector<uint32_t> starts(nl);
        if (nl) PMA_CUDA(cudaMemcpyAsync(starts.data(), lval, nl * 4, cudaMemcpyDeviceToHost, s));
        ctx->sync();
        for (int64_t i = 0; i < nl; ++i) level_begin.push_back(static_cast<size_t>(starts[i]));
    }
    level_begin.push_back(static_cast<size_t>(np));

    // Level sweep.
    const size_t nlevels = level_begin.size() - 1;
    PlateauSets ps;
    ps.eoff = eoff;
    ps.edges = by_dst;
    ps.order = order;
    ps.minrank = pminrank;
    ps.set = buf<ulonglong2>(ctx, "pores.set", np);
    ps.seed = buf<uint32_t>(ctx, "pores.seed", np);
    ps.err = err;
    ps.info = buf<unsigned long long>(ctx, "pores.info", 5);
    ps.pool_n = ps.info + 4;
    ps.hard = buf<uint32_t>(ctx, "pores.hard", np);
    ps.nslab = static_cast<unsigned>(ctx->num_sms * 8 * kSweepWarps);
    ps.slab = buf<ulonglong2>(ctx, "pores.slab", ps.nslab);
    // first position of each level (lval holds the level starts found above), and the end
    uint32_t* d_starts = buf<uint32_t>(ctx, "pores.level_starts", nlevels + 1);
    std::vector<uint32_t> h_starts(level_begin.begin(), level_begin.end());
    PMA_CUDA(cudaMemcpyAsync(d_starts, h_starts.data(), h_starts.size() * 4, cudaMemcpyHostToDevice, s));
    auto* h_info = static_cast<unsigned long long*>(ctx->host_staging(64));
    unsigned long long pool_cap = std::max<unsigned long long>(1ull << 22, 16ull * np);
    int rank_bits = 1;  // bits of a ball rank
    while (rank_bits < 32 && (1ull << rank_bits) < static_cast<unsigned long long>(nb)) ++rank_bits;
    // Merges the hard sets of the level that stopped the sweep (h_info: their number and elements).
    auto merge_hard = [&](unsigned long long nhard, unsigned long long total) {
        KernelTimer kt2(ctx, "level_merge");
        ctx->count("pores.hard_sets", static_cast<double>(nhard));
        ctx->count("pores.hard_set_elements_expanded", static_cast<double>(total));
        PMA_REQUIRE(total < (1ull << 40), PMA_ERR_MEMORY, "pma_pores: seed-set union too large");
        int hard_bits = 0;
        while ((1ull << hard_bits) < nhard) ++hard_bits;
        auto* deg = buf<unsigned long long>(ctx, "pores.bdeg", nhard);
        auto* doff = buf<unsigned long long>(ctx, "pores.bdoff", nhard);
        ps.cnt = buf<unsigned long long>(ctx, "pores.cnt", nhard);
        ps.first = buf<unsigned long long>(ctx, "pores.first", nhard);
        PMA_CUDA(cudaMemsetAsync(ps.cnt, 0, nhard * 8, s));
        level_hard_degrees<<<grid_for(ctx, nhard), 256, 0, s>>>(ps, deg);
        ctx->check_launch("level_hard_degrees");
        exclusive_sum(ctx, deg, doff, static_cast<int64_t>(nhard));
        auto merge = [&](auto* k0, auto* k1) {
            using K = std::remove_pointer_t<decltype(k0)>;
            level_expand<K><<<static_cast<unsigned>(ctx->num_sms * 16), 256, 0, s>>>(ps, doff, deg, nhard, k0, total,
                                                                                    rank_bits);
            ctx->check_launch("level_expand");
            ReadBack rb;
            rb.add(h_info, ps.info, 32);
            read_back(ctx, rb);
            const int64_t emitted = static_cast<int64_t>(std::min<unsigned long long>(h_info[3], total));
            sort_keys(ctx, k0, k1, emitted, rank_bits + hard_bits);  // radix passes over the used bits only
            const int64_t merged = unique(ctx, k1, k0, emitted, d_count);
            if (!merged) return;
            level_runs<K><<<grid_for(ctx, merged), 256, 0, s>>>(k0, merged, ps, rank_bits);
            ctx->check_launch("level_runs");
            level_place_hard<<<grid_for(ctx, nhard), 256, 0, s>>>(ps, nhard);
            ctx->check_launch("level_place_hard");
            level_copy_hard<K><<<grid_for(ctx, merged), 256, 0, s>>>(k0, merged, ps, rank_bits);
            ctx->check_launch("level_copy_hard");
        };
        if (rank_bits < 32 && rank_bits + hard_bits <= 32)
            merge(buf<uint32_t>(ctx, "pores.lkeys32", total), buf<uint32_t>(ctx, "pores.lkeys32b", total));
        else
            merge(buf<unsigned long long>(ctx, "pores.lkeys", total), buf<unsigned long long>(ctx, "pores.lkeys2", total));
    };
    constexpr unsigned long long kNoStop = ~0ull;
    constexpr unsigned kWindow = 64;  // launches between looks at the stop
    for (int attempt = 0; attempt < 3; ++attempt) {
        ps.pool = buf<uint32_t>(ctx, "pores.pool", pool_cap);
        ps.pool_cap = pool_cap;
        PMA_CUDA(cudaMemsetAsync(ps.info, 0, 40, s));
        PMA_CUDA(cudaMemsetAsync(ps.info, 0xFF, 8, s));  // no stop
        PMA_CUDA(cudaMemsetAsync(err, 0, 4, s));
        PMA_CUDA(cudaMemsetAsync(ps.slab, 0, ps.nslab * sizeof(ulonglong2), s));
        KernelTimer kt(ctx, "level_sets");
        for (size_t l = 0; l < nlevels;) {
            for (unsigned launches = 0; l < nlevels && launches < kWindow; ++launches) {
                size_t r = l;
                while (r < nlevels && level_begin[r + 1] - level_begin[r] <= kRunLevel) ++r;
                if (r > l) {  // a run of small levels
                    level_sweep<true, kRunWarps><<<1, kRunWarps * 32, 0, s>>>(ps, d_starts, static_cast<unsigned>(l),
                                                                             static_cast<unsigned>(r));
                    l = r;
                } else {
                    const size_t k = level_begin[l + 1] - level_begin[l];
                    const size_t blocks = std::max(std::min((k + kSweepWarps - 1) / kSweepWarps,
                                                            static_cast<size_t>(ctx->num_sms) * 8),
                                                   (k + kSweepList - 1) / kSweepList);
                    level_sweep<false, kSweepWarps><<<static_cast<unsigned>(blocks), kSweepWarps * 32, 0, s>>>(
                        ps, d_starts, static_cast<unsigned>(l), static_cast<unsigned>(l + 1));
                    ++l;
                }
                ctx->count_launch();
            }
            ctx->check_launch("level_sweep");
            ReadBack rb;
            rb.add(h_info, ps.info, 32);
            read_back(ctx, rb);
            if (h_info[0] != kNoStop) {  // go on behind the level that stopped
                l = static_cast<size_t>(h_info[0]) + 1;
                merge_hard(h_info[1], h_info[2]);
                PMA_CUDA(cudaMemsetAsync(ps.info, 0xFF, 8, s));
                PMA_CUDA(cudaMemsetAsync(ps.info + 1, 0, 24, s));
            }
        }
        ctx->count("pores.levels", static_cast<double>(nlevels));
        unsigned int h_err = 0;
        unsigned long long used = 0;
        PMA_CUDA(cudaMemcpyAsync(&h_err, err, 4, cudaMemcpyDeviceToHost, s));
        PMA_CUDA(cudaMemcpyAsync(&used, ps.pool_n, 8, cudaMemcpyDeviceToHost, s));
        ctx->sync();
        ctx->count("pores.pool_elements", static_cast<double>(used));
        PMA_REQUIRE(!(h_err & 32u), PMA_ERR_INTERNAL, "pma_pores: merged seed sets disagree with their bounds");
        if (!(h_err & 2u)) break;
        PMA_REQUIRE(attempt < 2, PMA_ERR_MEMORY, "pma_pores: seed-set pool overflow");
        pool_cap = 4 * used + 1024;
    }
    unsigned long long* soff = buf<unsigned long long>(ctx, "pores.soff", np);
    uint32_t* slen = buf<uint32_t>(ctx, "pores.slen", np);
    if (np) {
        unpack_sets<<<grid_for(ctx, np), 256, 0, s>>>(ps.set, np, soff, slen);
        ctx->check_launch("unpack_sets");
    }

    // Seeds -> pores in rank order.
    KernelTimer kt_tables(ctx, "pores_tables");
    auto kt_seeds = std::make_unique<KernelTimer>(ctx, "tables_seeds");
    // the seeds' ball ranks, compacted on the device (a few thousand of up to 10^8 plateaus)
    std::vector<uint32_t> seed_ranks;
    if (np) {
        flag_seeds<<<grid_for(ctx, np), 256, 0, s>>>(ps.seed, np, flags);
        ctx->check_launch("flag_seeds");
        uint32_t* d_seeds = buf<uint32_t>(ctx, "pores.seed_ranks", np);
        const int64_t ns = select_flagged(ctx, ps.seed, flags, d_seeds, np, d_count);
        seed_ranks.resize(ns);
        if (ns) PMA_CUDA(cudaMemcpyAsync(seed_ranks.data(), d_seeds, ns * 4, cudaMemcpyDeviceToHost, s));
        ctx->sync();
    }
    std::sort(seed_ranks.begin(), seed_ranks.end());
    const size_t npores = seed_ranks.size();
    const std::vector<uint32_t> ids = pore_id_sequence(npores);
    // rank -> pore index and rank -> pore id tables on the device
    const size_t nrank = std::max<int64_t>(nb, 1);
    uint32_t* d_rank2pore = buf<uint32_t>(ctx, "pores.rank2pore", nrank);
    uint32_t* d_rank2id = buf<uint32_t>(ctx, "pores.rank2id", nrank);
    fill_u32<<<grid_for(ctx, nrank), 256, 0, s>>>(d_rank2pore, nrank, kNone);
    ctx->check_launch("fill_u32");
    PMA_CUDA(cudaMemsetAsync(d_rank2id, 0, nrank * 4, s));
    auto* seed_items = buf<unsigned long long>(ctx, "pores.seed_items", npores);
    if (npores) {
        std::vector<uint32_t> up(2 * npores);
        std::copy(seed_ranks.begin(), seed_ranks.end(), up.begin());
        std::copy(ids.begin(), ids.end(), up.begin() + npores);
        uint32_t* d_up = buf<uint32_t>(ctx, "pores.seed_up", up.size());
        PMA_CUDA(cudaMemcpyAsync(d_up, up.data(), up.size() * 4, cudaMemcpyHostToDevice, s));
        scatter_seed_ids<<<grid_for(ctx, npores), 256, 0, s>>>(d_up, npores, d_rank2pore, d_rank2id);
        ctx->check_launch("scatter_seed_ids");
        gather_items<<<grid_for(ctx, npores), 256, 0, s>>>(items, d_up, npores, seed_items);
        ctx->check_launch("gather_items");
    }
    PoreAcc pa;
    pa.rank2pore = d_rank2pore;
    pa.pvol = buf<unsigned long long>(ctx, "pores.pvol", npores);
    pa.pbound = buf<unsigned int>(ctx, "pores.pbound", npores);
    PMA_CUDA(cudaMemsetAsync(pa.pvol, 0, std::max<size_t>(npores, 1) * 8, s));
    PMA_CUDA(cudaMemsetAsync(pa.pbound, 0, std::max<size_t>(npores, 1) * 4, s));
    if (np) {
        pore_accumulate<<<grid_for(ctx, np), 256, 0, s>>>(soff, slen, ps.pool, psize, pface, np, pa);
        ctx->check_launch("pore_accumulate");
    }

    kt_seeds.reset();
    // Throats: plateaus with two or more seeds, grouped by equal seed sets.
    auto kt_groups = std::make_unique<KernelTimer>(ctx, "tables_groups");
    if (np) {
        flag_multi<<<grid_for(ctx, np), 256, 0, s>>>(slen, np, flags);
        ctx->check_launch("flag_multi");
    }
    uint32_t* multi = buf<uint32_t>(ctx, "pores.multi", np);
    const int64_t nm = np ? select_flagged(ctx, thrust::counting_iterator<uint32_t>(0), flags, multi,
                                           np, d_count)
                          : 0;
    uint32_t* plateau_group = buf<uint32_t>(ctx, "pores.pgroup", np);
    pma_table* t = new pma_table;
    int64_t ngroups = 0;
    GroupOut go{};
    if (nm) {
        auto* h1 = buf<unsigned long long>(ctx, "pores.h1", nm);
        auto* h2 = buf<unsigned long long>(ctx, "pores.h2", nm);
        auto* ktmp = buf<unsigned long long>(ctx, "pores.ktmp", nm);
        uint32_t* v1 = buf<uint32_t>(ctx, "pores.v1", nm);
        uint32_t* v2 = buf<uint32_t>(ctx, "pores.v2", nm);
        // Group plateaus with equal seed sets: a radix sort by the first hash puts equal sets
        // side by side unless two different sets share it (about n^2 / 2^65 likely), which
        // group_starts flags; then stable sorts by the second hash and then the first put
        // equal (h1, h2) pairs side by side.
        uint32_t* gstart = buf<uint32_t>(ctx, "pores.gstart", nm);
        uint32_t* gid = buf<uint32_t>(ctx, "pores.gid", nm);
        throat_hashes<<<grid_for(ctx, nm), 256, 0, s>>>(soff, slen, ps.pool, multi, nm, h1, h2);
        ctx->check_launch("throat_hashes");
        sort_pairs(ctx, h1, ktmp, multi, v2, nm);
        throat_hashes<<<grid_for(ctx, nm), 256, 0, s>>>(soff, slen, ps.pool, v2, nm, h1, h2);
        ctx->check_launch("throat_hashes");
        group_starts<<<grid_for(ctx, nm), 256, 0, s>>>(v2, h1, h2, nm, soff, slen, ps.pool, gstart, err);
        ctx->check_launch("group_starts");
        {
            unsigned int h_err0 = 0;
            PMA_CUDA(cudaMemcpyAsync(&h_err0, err, 4, cudaMemcpyDeviceToHost, s));
            ctx->sync();
            if (h_err0 & 64u) {
                PMA_CUDA(cudaMemsetAsync(err, 0, 4, s));
                throat_hashes<<<grid_for(ctx, nm), 256, 0, s>>>(soff, slen, ps.pool, multi, nm, h1, h2);
                ctx->check_launch("throat_hashes");
                sort_pairs(ctx, h2, ktmp, multi, v1, nm);
                throat_hashes<<<grid_for(ctx, nm), 256, 0, s>>>(soff, slen, ps.pool, v1, nm, h1, h2);
                ctx->check_launch("throat_hashes");
                sort_pairs(ctx, h1, ktmp, v1, v2, nm);
                throat_hashes<<<grid_for(ctx, nm), 256, 0, s>>>(soff, slen, ps.pool, v2, nm, h1, h2);
                ctx->check_launch("throat_hashes");
                group_starts<<<grid_for(ctx, nm), 256, 0, s>>>(v2, h1, h2, nm, soff, slen, ps.pool, gstart, err);
                ctx->check_launch("group_starts");
            }
        }
        exclusive_sum(ctx, gstart, gid, nm);
        uint32_t last_off = 0, last_start = 0;
        PMA_CUDA(cudaMemcpyAsync(&last_off, gid + nm - 1, 4, cudaMemcpyDeviceToHost, s));
        PMA_CUDA(cudaMemcpyAsync(&last_start, gstart + nm - 1, 4, cudaMemcpyDeviceToHost, s));
        ctx->sync();
        ngroups = static_cast<int64_t>(last_off) + last_start;
        to_group_index<<<grid_for(ctx, nm), 256, 0, s>>>(gid, gstart, nm, gstart);
        ctx->check_launch("to_group_index");
        go.gvol = buf<unsigned long long>(ctx, "pores.gvol", ngroups);
        go.gfirst = buf<unsigned long long>(ctx, "pores.gfirst", ngroups);
        go.grep = buf<uint32_t>(ctx, "pores.grep", ngroups);
        PMA_CUDA(cudaMemsetAsync(go.gvol, 0, ngroups * 8, s));
        PMA_CUDA(cudaMemsetAsync(go.gfirst, 0xFF, ngroups * 8, s));
        group_reduce<<<grid_for(ctx, nm), 256, 0, s>>>(v2, gstart, nm, psize, roots, go, plateau_group);
        ctx->check_launch("group_reduce");
        unsigned int h_err = 0;
        PMA_CUDA(cudaMemcpyAsync(&h_err, err, 4, cudaMemcpyDeviceToHost, s));
        ctx->sync();
        PMA_REQUIRE(!(h_err & 4u), PMA_ERR_INTERNAL, "pma_pores: seed-set hash collision");
    }
    kt_groups.reset();
    auto kt_types = std::make_unique<KernelTimer>(ctx, "tables_ids");
    uint32_t* group_tid = buf<uint32_t>(ctx, "pores.gtid", ngroups);
    if (ngroups) {
        const SeedLists lists{go.grep, soff, slen, ps.pool, d_rank2id};
        type_keys<<<grid_for(ctx, ngroups), 256, 0, s>>>(lists, ngroups, go.gfirst);
        ctx->check_launch("type_keys");
        type_rows(ctx, go.gfirst, ngroups, lists, go.gvol, group_tid, t);
    }

    kt_types.reset();
    auto kt_labels = std::make_unique<KernelTimer>(ctx, "tables_labels");
    // Labels.
    uint32_t* plabel = buf<uint32_t>(ctx, "pores.plabel", np);
    if (np) {
        plateau_labels<<<grid_for(ctx, np), 256, 0, s>>>(soff, slen, ps.pool, d_rank2id, plateau_group,
                                                         group_tid, np, plabel);
        ctx->check_launch("plateau_labels");
    }
    voxel_labels<<<G, 256, 0, s>>>(pid, plabel, n, labels);
    ctx->check_launch("voxel_labels");

    kt_labels.reset();
    KernelTimer kt_rows(ctx, "tables_rows");
    // The pores' rows, in id order.
    std::vector<unsigned long long> pvol(npores);
    std::vector<unsigned int> pbound(npores);
    std::vector<unsigned long long> h_items(npores);
    if (npores) {
        PMA_CUDA(cudaMemcpyAsync(h_items.data(), seed_items, npores * 8, cudaMemcpyDeviceToHost, s));
        PMA_CUDA(cudaMemcpyAsync(pvol.data(), pa.pvol, npores * 8, cudaMemcpyDeviceToHost, s));
        PMA_CUDA(cudaMemcpyAsync(pbound.data(), pa.pbound, npores * 4, cudaMemcpyDeviceToHost, s));
    }
    ctx->sync();
    for (size_t k = 0; k < npores; ++k) {
        int x, y, z;
        g.coords(static_cast<uint32_t>(h_items[k]), x, y, z);
        pma_pore p;
        std::memset(&p, 0, sizeof(p));
        p.id = ids[k];
        p.seed_x = x;
        p.seed_y = y;
        p.seed_z = z;
        p.seed_r2 = static_cast<uint32_t>(h_items[k] >> 32);
        p.is_boundary = pbound[k] ? 1 : 0;
        p.volume = pvol[k];
        t->pores.push_back(p);
    }
    if (ctx->reference_throat_ids && ngroups) {
        KernelTimer kt_exact(ctx, "exact_type_ids");
        reference_type_ids(ctx, t, labels, crad2, d, st);
    }
    return t;
}

// Renumbers the shared types of the initial propagation in the reference's creation order
// (exact_ids.cpp) and relabels their voxels.
void reference_type_ids(pma_ctx* ctx, pma_table* t, uint32_t* labels, const uint32_t* crad2, pma_dims d,
                        pma_stencil st) {
    cudaStream_t s = ctx->stream;
    const size_t n = voxels(d);
    const size_t ng = t->throats.size();
    std::vector<uint32_t> h_labels(n), h_crad(n);
    PMA_CUDA(cudaMemcpyAsync(h_labels.data(), labels, n * 4, cudaMemcpyDeviceToHost, s));
    PMA_CUDA(cudaMemcpyAsync(h_crad.data(), crad2, n * 4, cudaMemcpyDeviceToHost, s));
    ctx->sync();
    std::vector<std::vector<uint32_t>> lists(ng);
    std::vector<uint32_t> fast(ng);
    for (size_t g = 0; g < ng; ++g) {
        const pma_throat& th = t->throats[g];
        lists[g].assign(t->pool.begin() + th.pool_offset, t->pool.begin() + th.pool_offset + th.n_pores);
        std::sort(lists[g].begin(), lists[g].end());
        fast[g] = th.id;
    }
    const std::vector<uint32_t> exact =
        replay_type_ids(h_crad.data(), h_labels.data(), d, st == PMA_D3Q7, t->pores, lists, fast);
    // voxels: old id -> new id (old ids ascending, as the rows are)
    std::vector<uint32_t> old_ids(ng), new_ids(ng);
    for (size_t g = 0; g < ng; ++g) {
        old_ids[g] = fast[g];
        new_ids[g] = exact[g];
    }
    PMA_REQUIRE(std::is_sorted(old_ids.begin(), old_ids.end()), PMA_ERR_INTERNAL, "pma_pores: type rows out of order");
    uint32_t* d_old = buf<uint32_t>(ctx, "pores.exact_old", ng);
    uint32_t* d_new = buf<uint32_t>(ctx, "pores.exact_new", ng);
    PMA_CUDA(cudaMemcpyAsync(d_old, old_ids.data(), ng * 4, cudaMemcpyHostToDevice, s));
    PMA_CUDA(cudaMemcpyAsync(d_new, new_ids.data(), ng * 4, cudaMemcpyHostToDevice, s));
    remap_labels<<<grid_for(ctx, n), 256, 0, s>>>(labels, n, d_old, d_new, static_cast<uint32_t>(ng));
    ctx->check_launch("remap_labels");
    // rows in ascending (new) id order
    std::vector<size_t> order(ng);
    for (size_t g = 0; g < ng; ++g) order[g] = g;
    std::sort(order.begin(), order.end(), [&](size_t a, size_t b) { return exact[a] < exact[b]; });
    std::vector<pma_throat> rows;
    std::vector<uint32_t> pool;
    rows.reserve(ng);
    pool.reserve(t->pool.size());
    for (size_t k = 0; k < ng; ++k) {
        pma_throat th = t->throats[order[k]];
        const uint64_t off = th.pool_offset;
        th.id = exact[order[k]];
        th.pool_offset = pool.size();
        pool.insert(pool.end(), t->pool.begin() + off, t->pool.begin() + off + th.n_pores);
        rows.push_back(th);
    }
    t->throats.swap(rows);
    t->pool.swap(pool);
    ctx->sync();
}

// a11: EmptyPoresRemover.cpp:31-244 on the host table, then one relabel launch.
void remove_empty_pores(pma_ctx* ctx, pma_table* t, uint32_t* labels, pma_dims d) {
    KernelTimer kt_stage(ctx, "stage_removal");
    check_dims(d);
    PMA_REQUIRE(labels, PMA_ERR_ARGUMENT, "pma_remove_empty_pores: null labels");
    auto kt_host = std::make_unique<KernelTimer>(ctx, "removal_tables");
    auto mark = std::chrono::steady_clock::now();
    auto phase = [&](const char* name) {  // host time of each part, with the timing report
        const auto now = std::chrono::steady_clock::now();
        ctx->count(name, std::chrono::duration<double, std::milli>(now - mark).count());
        mark = now;
    };
    // EPR.cpp:193-244: drop zero-volume pores and remove them from the type lists.
    std::vector<uint32_t> empty;
    std::vector<pma_pore> kept;
    for (const pma_pore& p : t->pores) {
        if (p.volume == 0) empty.push_back(p.id);
        else kept.push_back(p);
    }
    std::sort(empty.begin(), empty.end());
    // empty pores by id (pore ids are below every type id and dense enough for a flag array)
    uint32_t max_pore = 0;
    for (const pma_pore& p : t->pores) max_pore = std::max(max_pore, p.id);
    std::vector<uint8_t> is_empty(static_cast<size_t>(max_pore) + 1, 0);
    for (uint32_t id : empty) is_empty[id] = 1;
    // Types in ascending id order with sorted, filtered pore lists (flat arrays).
    const size_t nt = t->throats.size();
    std::vector<uint32_t> by_id(nt);
    for (size_t i = 0; i < nt; ++i) by_id[i] = static_cast<uint32_t>(i);
    auto id_less = [&](uint32_t a, uint32_t b) { return t->throats[a].id < t->throats[b].id; };
    if (!std::is_sorted(by_id.begin(), by_id.end(), id_less)) std::sort(by_id.begin(), by_id.end(), id_less);
    // One pass, on host threads when there are many types: each list filtered and sorted in the place
    // that its whole length would take, and hashed.
    std::vector<size_t> loff(nt + 1, 0);
    for (size_t k = 0; k < nt; ++k) loff[k + 1] = loff[k] + t->throats[by_id[k]].n_pores;
    std::vector<uint32_t> lists(loff[nt]), len(nt);
    std::vector<unsigned long long> lhash(nt);
    auto filter = [&](size_t lo, size_t hi) {
        for (size_t k = lo; k < hi; ++k) {
            const pma_throat& th = t->throats[by_id[k]];
            const uint32_t* from = t->pool.data() + th.pool_offset;
            uint32_t* list = lists.data() + loff[k];
            uint32_t m = 0;
            for (uint32_t i = 0; i < th.n_pores; ++i) {
                const uint32_t pid = from[i];
                if (pid > max_pore || !is_empty[pid]) list[m++] = pid;
            }
            if (m > 1 && !std::is_sorted(list, list + m)) std::sort(list, list + m);
            unsigned long long h = 1469598103934665603ull ^ m;
            for (uint32_t i = 0; i < m; ++i) h = (h ^ list[i]) * 1099511628211ull;
            len[k] = m;
            lhash[k] = h;
        }
    };
    const unsigned nth = nt >= (1u << 15) ? std::max(1u, std::min(8u, std::thread::hardware_concurrency())) : 1u;
    {
        std::vector<std::thread> ts;
        for (unsigned i = 1; i < nth; ++i) {
            try {
                ts.emplace_back(filter, nt * i / nth, nt * (i + 1) / nth);
            } catch (const std::system_error&) {
                filter(nt * i / nth, nt * (i + 1) / nth);  // no thread to be had: in line
            }
        }
        filter(0, nt / nth);
        for (auto& th : ts) th.join();
    }
    phase("removal.filter_ms");
    ctx->count("removal.types", static_cast<double>(nt));
    std::vector<char> alive(nt, 1);
    std::vector<std::pair<uint32_t, uint32_t>> remap;  // (old id, new id)
    // EPR.cpp:167-191: types with fewer than two pores.
    for (size_t k = 0; k < nt; ++k)
        if (len[k] < 2) {
            if (len[k] == 1) remap.emplace_back(t->throats[by_id[k]].id, lists[loff[k]]);
            alive[k] = 0;
        }
    // EPR.cpp:126-165: merge types with equal pore lists into the largest id. A hash table holds the first
    // type of each list; equal hashes are settled by comparing the lists. (Sorting the hashes of 82
    // thousand types took 4.2 ms; the whole removal took 8.1 ms before this form and the one-pass filter, 3.0 after.)
    size_t slots = 16;
    while (slots < 2 * nt) slots *= 2;
    std::vector<uint32_t> first(slots, kNone), like(nt, kNone), keep(nt, 0);  // like: the first type of k's list
    bool merged = false;
    for (size_t k = 0; k < nt; ++k) {
        if (!alive[k]) continue;
        const uint32_t* list = lists.data() + loff[k];
        for (size_t h = static_cast<size_t>((lhash[k] * 0x9E3779B97F4A7C15ull) >> 32) & (slots - 1);; h = (h + 1) & (slots - 1)) {
            const uint32_t f = first[h];
            if (f == kNone) first[h] = like[k] = static_cast<uint32_t>(k);
            else if (lhash[f] == lhash[k] && len[f] == len[k] && std::equal(list, list + len[k], lists.data() + loff[f])) like[k] = f;
            else continue;
            break;
        }
        merged |= like[k] != k;
        keep[like[k]] = std::max(keep[like[k]], t->throats[by_id[k]].id);
    }
    for (size_t k = 0; k < nt && merged; ++k) {
        if (!alive[k]) continue;
        const uint32_t id = t->throats[by_id[k]].id;
        if (id != keep[like[k]]) {
            alive[k] = 0;
            remap.emplace_back(id, keep[like[k]]);
        }
    }
    phase("removal.merge_ms");
    std::vector<pma_throat> throats;
    std::vector<uint32_t> pool;
    throats.reserve(nt);
    pool.reserve(lists.size());
    for (size_t k = 0; k < nt; ++k) {
        if (!alive[k]) continue;
        pma_throat th;
        th.id = t->throats[by_id[k]].id;
        th.volume = t->throats[by_id[k]].volume;
        th.n_pores = len[k];
        th.pool_offset = pool.size();
        pool.insert(pool.end(), lists.begin() + loff[k], lists.begin() + loff[k] + len[k]);
        throats.push_back(th);
    }
    t->pores.swap(kept);
    t->throats.swap(throats);
    t->pool.swap(pool);
    std::sort(remap.begin(), remap.end());
    phase("removal.rows_ms");
    kt_host.reset();
    if (remap.empty()) return;  // EPR.cpp:54-57
    std::vector<uint32_t> o, nw;
    for (auto& kv : remap) {
        o.push_back(kv.first);
        nw.push_back(kv.second);
    }  // ascending old ids: remap_labels searches them
    cudaStream_t s = ctx->stream;
    uint32_t* d_old = buf<uint32_t>(ctx, "remove.old", o.size());
    uint32_t* d_new = buf<uint32_t>(ctx, "remove.new", nw.size());
    PMA_CUDA(cudaMemcpyAsync(d_old, o.data(), o.size() * 4, cudaMemcpyHostToDevice, s));
    PMA_CUDA(cudaMemcpyAsync(d_new, nw.data(), nw.size() * 4, cudaMemcpyHostToDevice, s));
    const size_t n = voxels(d);
    remap_labels<<<grid_for(ctx, n), 256, 0, s>>>(labels, n, d_old, d_new, static_cast<uint32_t>(o.size()));
    ctx->check_launch("remap_labels");
    ctx->sync();
}

}  // namespace pma
