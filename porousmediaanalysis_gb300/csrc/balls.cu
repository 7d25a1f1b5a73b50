// Containing-ball radii, winning centres and the maximum-ball mask
// (ContainingBallsAssigner.cpp:101-250).
//
// Single-thread semantics of the reference: centres are visited in x, y, z order and a
// voxel takes a new centre only on a strictly larger squared radius, so each void voxel
// ends with the largest r^2 covering it and, among those, the lexicographically smallest
// (x, y, z) centre. Both orders fit one 64-bit key,
//     key = (r^2 << 32) | (0xFFFFFFFF - ((x * SY + y) * SZ + z)),
// and the winner of a voxel is the covering centre of largest key.
//
// Work reduction: a centre whose discrete ball lies inside the ball of one of its 26
// neighbours can never win a voxel (the neighbour covers the same voxels with a strictly
// larger radius), so it is dropped. Containment B(c, R) in B(c + e, R') holds iff
// R' >= M_k(R) = max over lattice v with |v|^2 <= R of |v + e|^2, k = |e|^2; M_k is computed
// exactly for R < kExactTable and replaced above it by the continuous sufficient condition
// (sqrt(R) + sqrt(k))^2 <= R'.
//
// Gather: the volume is cut into 8^3 tiles, in groups of 2 x 2 x 2; every kept centre is listed in each
// group its ball reaches, and from there in each of the group's tiles that it reaches, unless its
// key is below the tile's floor (the largest key found of a ball covering the whole tile, which every
// voxel of the tile is covered by). One CTA per tile orders its list by radius in shared memory, and
// each warp of voxels takes, per voxel, the largest key among the entries whose ball covers it: the
// reference's winner. A warp only tests entries that reach the box of its voxels that may still gain
// and stops where the radius order shows that no later entry can, so the work is close to the
// winners' ranks in the list rather than the ball volumes a scatter would touch.
//
// What bounds it: instructions and barriers in the gather, a chunk after the other; atomics and scattered
// stores in the fill. Atomics go at 60 G/s, whatever they add: one for each entry of a tile (1.1 G in
// a 704 x 768 x 811 spinodal) took 18 ms in the count and again in the fill; the groups' lists have a
// quarter of the entries, and the split reads them in order. That spinodal, ms: kept centres 13 -> 2.9 (bricks),
// floors and counts 23 -> 4.6 (groups; a quarter of the centres for the floors, 9 -> 2.5), fill 19 -> 7.0
// and split 7.3, gather 117 -> 38 (least key by 32-bit reductions and 2 x 4 x 4 boxes 82, centres by
// descending radius 73, the box of the lanes still open 44, lists in the order of the radii 41, four CTAs
// an SM 38); stage 170 -> 65. A gather that filters its group's list itself took 68 ms, one that keeps the
// lists' own order 45, lists in chunks of 1024 44.
#include <thrust/iterator/counting_iterator.h>

#include <vector>

#include "devutil.cuh"
#include "group_runs.h"

namespace pma {
namespace {

constexpr uint32_t kExactTable = 1u << 16;
constexpr int kTile = 8;          // tile edge
constexpr int kTileVox = 512;     // voxels (and threads) per tile
constexpr int kGroup = 2;         // tiles along the edge of a group, which shares one list
constexpr int kListCap = 2048;    // entries ordered in shared memory at a time; longer lists go in chunks

__device__ __forceinline__ uint32_t isqrt_u32(uint32_t n) {
    uint32_t r = static_cast<uint32_t>(sqrtf(static_cast<float>(n)));
    while (r * r > n) --r;
    while ((r + 1) * (r + 1) <= n) ++r;
    return r;
}

// M_k(R) for k = 1, 2, 3, one thread per R.
__global__ void balls_containment_table(uint32_t* __restrict__ m1, uint32_t* __restrict__ m2,
                                        uint32_t* __restrict__ m3, uint32_t nR) {
    const uint32_t R = blockIdx.x * blockDim.x + threadIdx.x;
    if (R >= nR) return;
    uint32_t b1 = 0, b2 = 0, b3 = 0;
    const uint32_t amax = isqrt_u32(R);
    for (uint32_t a = 0; a <= amax; ++a) {
        const uint32_t ra = R - a * a;
        const uint32_t bmax = isqrt_u32(ra);
        for (uint32_t b = 0; b <= bmax; ++b) {
            const uint32_t c = isqrt_u32(ra - b * b);
            const uint32_t a1 = (a + 1) * (a + 1), bb = b * b, b1s = (b + 1) * (b + 1);
            const uint32_t cc = c * c, c1 = (c + 1) * (c + 1);
            const uint32_t v1 = a1 + bb + cc, v2 = a1 + b1s + cc, v3 = a1 + b1s + c1;
            b1 = v1 > b1 ? v1 : b1;
            b2 = v2 > b2 ? v2 : b2;
            b3 = v3 > b3 ? v3 : b3;
        }
    }
    m1[R] = b1;
    m2[R] = b2;
    m3[R] = b3;
}

// B(c, R) lies inside the ball of a neighbour at squared distance k whose r^2 is Rn: Rn >= M_k(R), or the
// continuous bound where the table ends. Both grow with Rn: the largest Rn of each k decides.
__device__ __forceinline__ bool contained(uint32_t R, uint32_t Rn, int k, const uint32_t* __restrict__ mtab, uint32_t ntab) {
    if (Rn <= R) return false;
    if (R < ntab) return Rn >= __ldg(mtab + (k - 1) * ntab + R);
    // (sqrt(R) + sqrt(k))^2 <= Rn  <=>  t >= 0 and t^2 >= 4kR, t = Rn - R - k
    const long long t = static_cast<long long>(Rn) - R - k;
    return t >= 0 && static_cast<unsigned long long>(t) * t >= 4ull * static_cast<unsigned long long>(k) * R;
}

// Kept centres (flag 1). A block takes a brick of 32 x 8 x 8 voxels (y, x, z) with its halo in shared
// memory; a thread walks the eight slices of its (x, y), and of each slice takes its own value,
// the largest of the four neighbours at distance 1 and the largest of the four diagonal ones:
// three slices together give the largest neighbour at each distance. (Reading up to 26
// neighbours and table entries a voxel through L1 took 12.4 ms on 704 x 768 x 811 voxels, this 2.9.)
constexpr int kBrickY = 32, kBrickX = 8, kBrickZ = 8;
constexpr int kHaloY = kBrickY + 2, kHaloX = kBrickX + 2, kHaloZ = kBrickZ + 2;

__global__ void __launch_bounds__(32 * kBrickX) balls_candidate_flags(const uint32_t* __restrict__ edt2, Grid g, int BY, int BX,
                                                                      const uint32_t* __restrict__ mtab, uint32_t ntab,
                                                                      uint32_t nR, uint8_t* __restrict__ flags,
                                                                      unsigned int* __restrict__ err) {
    constexpr int kRows = kHaloX * kHaloZ;
    __shared__ uint32_t tile[kRows * kHaloY];
    const int lane = threadIdx.x & 31, row = threadIdx.x >> 5;
    const unsigned rest = blockIdx.x / static_cast<unsigned>(BY);
    const int y0 = static_cast<int>(blockIdx.x - rest * static_cast<unsigned>(BY)) * kBrickY;
    const int z0 = static_cast<int>(rest / static_cast<unsigned>(BX)) * kBrickZ;
    const int x0 = static_cast<int>(rest % static_cast<unsigned>(BX)) * kBrickX;
    auto value = [&](int x, int y, int z) { return g.inside(x, y, z) ? __ldg(edt2 + g.idx(x, y, z)) : 0u; };
#pragma unroll
    for (int q = 0; q < (kRows + kBrickX - 1) / kBrickX; ++q) {
        const int r = q * kBrickX + row;
        if (r < kRows) tile[r * kHaloY + 1 + lane] = value(x0 - 1 + r % kHaloX, y0 + lane, z0 - 1 + r / kHaloX);
    }
    if (threadIdx.x < 2 * kRows) {
        const int r = threadIdx.x >> 1, side = threadIdx.x & 1;
        tile[r * kHaloY + side * (kHaloY - 1)] = value(x0 - 1 + r % kHaloX, side ? y0 + kBrickY : y0 - 1, z0 - 1 + r / kHaloX);
    }
    __syncthreads();
    const uint32_t* col = tile + row * kHaloY + lane;  // (x - 1, y - 1) of slice z - 1
    constexpr int kSlice = kHaloX * kHaloY;
    const int x = x0 + row, y = y0 + lane;
    const bool in = x < g.SX && y < g.SY;
    uint32_t c0 = 0, f0 = 0, d0 = 0, c1 = 0, f1 = 0, d1 = 0;
#pragma unroll
    for (int p = 0; p < kHaloZ; ++p) {
        const uint32_t* q = col + p * kSlice;
        const uint32_t c2 = q[kHaloY + 1];
        const uint32_t f2 = max(max(q[kHaloY], q[kHaloY + 2]), max(q[1], q[2 * kHaloY + 1]));
        const uint32_t d2 = max(max(q[0], q[2]), max(q[2 * kHaloY], q[2 * kHaloY + 2]));
        const int z = z0 + p - 2;  // the slice between c0 and c2
        if (p >= 2 && in && z < g.SZ) {
            const uint32_t R = c1;
            uint8_t f = 0;
            if (R >= nR) {  // max_edt2 below the data: refuse rather than index past the table
                atomicOr(err, 1u);
            } else if (R != 0) {
                f = !contained(R, max(max(c0, c2), f1), 1, mtab, ntab) && !contained(R, max(max(f0, f2), d1), 2, mtab, ntab) &&
                    !contained(R, max(d0, d2), 3, mtab, ntab);
            }
            flags[g.idx(x, y, z)] = f;
        }
        c0 = c1;
        f0 = f1;
        d0 = d1;
        c1 = c2;
        f1 = f2;
        d1 = d2;
    }
}

struct Tiles {
    int TX, TY, TZ;  // tiles (or groups of them) per axis
    __device__ __forceinline__ size_t id(int tx, int ty, int tz) const {
        return (static_cast<size_t>(tz) * TX + tx) * TY + ty;
    }
};

// Visits the groups whose box is within sqrt(R) of centre (x, y, z), restricted to group
// z-range [tz0, tz1).
template <class F>
__device__ __forceinline__ void for_each_group(Grid g, Tiles t, int x, int y, int z, uint32_t R,
                                               int tz0, int tz1, F f) {
    constexpr int kEdge = kTile * kGroup;
    const int r = static_cast<int>(isqrt_u32(R));
    const int ax = max(x - r, 0) / kEdge, bx = min(x + r, g.SX - 1) / kEdge;
    const int ay = max(y - r, 0) / kEdge, by = min(y + r, g.SY - 1) / kEdge;
    const int az = max(max(z - r, 0) / kEdge, tz0), bz = min(min(z + r, g.SZ - 1) / kEdge, tz1 - 1);
    for (int tz = az; tz <= bz; ++tz) {
        const int lz = tz * kEdge, hz = min(lz + kEdge - 1, g.SZ - 1);
        const int dz = z < lz ? lz - z : (z > hz ? z - hz : 0);
        for (int tx = ax; tx <= bx; ++tx) {
            const int lx = tx * kEdge, hx = min(lx + kEdge - 1, g.SX - 1);
            const int dx = x < lx ? lx - x : (x > hx ? x - hx : 0);
            const int dxz = dx * dx + dz * dz;
            if (static_cast<uint32_t>(dxz) > R) continue;
            for (int ty = ay; ty <= by; ++ty) {
                const int ly = ty * kEdge, hy = min(ly + kEdge - 1, g.SY - 1);
                const int dy = y < ly ? ly - y : (y > hy ? y - hy : 0);
                if (static_cast<uint32_t>(dxz + dy * dy) > R) continue;
                f(t.id(tx, ty, tz));
            }
        }
    }
}

__device__ __forceinline__ unsigned long long ball_key(Grid g, int x, int y, int z, uint32_t R) {
    const uint32_t lex = (static_cast<uint32_t>(x) * g.SY + y) * static_cast<uint32_t>(g.SZ) + z;
    return (static_cast<unsigned long long>(R) << 32) | (0xFFFFFFFFu - lex);
}

// Squared radii of the kept centres, counted down from the largest (a sort key, descending r^2).
__global__ void balls_radii(const uint32_t* __restrict__ edt2, const uint32_t* __restrict__ cand, size_t nc, uint32_t max_edt2,
                            uint32_t* __restrict__ down) {
    PMA_GRID_STRIDE(i, nc) down[i] = max_edt2 - edt2[cand[i]];
}

// Floor of a tile: the largest key among balls covering the whole tile (those found here: balls
// of r^2 below kFloorR2 cover no whole tile except clipped ones, and are left out). Every voxel of the
// tile is covered by that ball, so its winner's key is at least the floor, and list entries
// below it can be left out.
constexpr uint32_t kFloorR2 = 37;  // half the diagonal between a tile's corner voxels: 3 * 3.5^2 = 36.75

__global__ void balls_tile_floor(const uint32_t* __restrict__ cand, const uint32_t* __restrict__ down, uint32_t max_edt2,
                                 size_t nc, size_t step, Grid g, Tiles t, unsigned long long* __restrict__ floor) {
    PMA_GRID_STRIDE(k, (nc + step - 1) / step) {
        const size_t i = k * step;
        const uint32_t R = max_edt2 - down[i];
        if (R < kFloorR2) continue;
        int x, y, z;
        g.coords(cand[i], x, y, z);
        const int r = static_cast<int>(isqrt_u32(R));
        const unsigned long long key = ball_key(g, x, y, z, R);
        // per axis: tiles whose far voxel is within r
        const int ax = (max(x - r, 0) + kTile - 1) / kTile, bx = min(x + r, g.SX - 1) == g.SX - 1 ? t.TX - 1 : (x + r + 1) / kTile - 1;
        const int ay = (max(y - r, 0) + kTile - 1) / kTile, by = min(y + r, g.SY - 1) == g.SY - 1 ? t.TY - 1 : (y + r + 1) / kTile - 1;
        const int az = (max(z - r, 0) + kTile - 1) / kTile, bz = min(z + r, g.SZ - 1) == g.SZ - 1 ? t.TZ - 1 : (z + r + 1) / kTile - 1;
        for (int tz = az; tz <= bz; ++tz) {
            const int fz = max(abs(z - tz * kTile), abs(min(tz * kTile + kTile, g.SZ) - 1 - z));
            for (int tx = ax; tx <= bx; ++tx) {
                const int fx = max(abs(x - tx * kTile), abs(min(tx * kTile + kTile, g.SX) - 1 - x));
                const uint32_t fxz = static_cast<uint32_t>(fx * fx + fz * fz);
                if (fxz > R) continue;
                for (int ty = ay; ty <= by; ++ty) {
                    const int fy = max(abs(y - ty * kTile), abs(min(ty * kTile + kTile, g.SY) - 1 - y));
                    if (fxz + static_cast<uint32_t>(fy * fy) > R) continue;
                    const size_t tid = t.id(tx, ty, tz);
                    // most lose to one recorded before: a plain read (possibly old: floors only grow) first
                    if (key > *reinterpret_cast<volatile unsigned long long*>(floor + tid)) atomicMax(&floor[tid], key);
                }
            }
        }
    }
}

// Floor of a group: the least of its tiles' floors, what every voxel of the group's winner's key is at least.
__global__ void balls_group_floor(const unsigned long long* __restrict__ floor, Tiles t, Tiles gt, size_t ngroups,
                                  unsigned long long* __restrict__ gfloor) {
    PMA_GRID_STRIDE(i, ngroups) {
        const int gy = static_cast<int>(i % gt.TY);
        const size_t rest = i / gt.TY;
        const int gx = static_cast<int>(rest % gt.TX), gz = static_cast<int>(rest / gt.TX);
        unsigned long long least = ~0ull;
        for (int tz = gz * kGroup; tz < min(gz * kGroup + kGroup, t.TZ); ++tz)
            for (int tx = gx * kGroup; tx < min(gx * kGroup + kGroup, t.TX); ++tx)
                for (int ty = gy * kGroup; ty < min(gy * kGroup + kGroup, t.TY); ++ty) least = min(least, floor[t.id(tx, ty, tz)]);
        gfloor[i] = least;
    }
}

// Adds one to *counter and returns what it held. Where the lanes' centres are neighbours (kNear) most
// of them are at the same counter, and one lane adds for all.
template <bool kNear>
__device__ __forceinline__ unsigned int add_one(unsigned int* counter, size_t id) {
    if (!kNear) return atomicAdd(counter, 1u);
    const unsigned lane = threadIdx.x & 31, peers = __match_any_sync(__activemask(), static_cast<unsigned int>(id));
    const int leader = __ffs(peers) - 1;
    unsigned int at = 0;
    if (static_cast<int>(lane) == leader) at = atomicAdd(counter, __popc(peers));
    return __shfl_sync(peers, at, leader) + __popc(peers & ((1u << lane) - 1u));
}

template <bool kNear>
struct CountGroup {
    const unsigned long long* gfloor;
    unsigned int* gcount;
    unsigned long long key;
    __device__ void operator()(size_t id) const {
        if (key >= __ldg(gfloor + id)) add_one<kNear>(&gcount[id], id);
    }
};

template <bool kNear>
struct FillGroup {
    const unsigned long long* gfloor;
    const unsigned long long* goff;
    unsigned long long base;
    size_t g0, g1;  // the groups being filled
    unsigned int* gcursor;
    unsigned long long* groups;
    unsigned long long key;
    __device__ void operator()(size_t id) const {
        if (id < g0 || id >= g1 || key < __ldg(gfloor + id)) return;
        const unsigned int at = add_one<kNear>(&gcursor[id], id);
        groups[goff[id] - base + at] = key;
    }
};

template <bool kNear>
__global__ void balls_group_count(const uint32_t* __restrict__ cand, const uint32_t* __restrict__ down, uint32_t max_edt2,
                                  size_t nc, Grid g, Tiles gt, const unsigned long long* __restrict__ gfloor,
                                  unsigned int* __restrict__ gcount) {
    PMA_GRID_STRIDE(i, nc) {
        int x, y, z;
        g.coords(cand[i], x, y, z);
        const uint32_t R = max_edt2 - down[i];
        for_each_group(g, gt, x, y, z, R, 0, gt.TZ, CountGroup<kNear>{gfloor, gcount, ball_key(g, x, y, z, R)});
    }
}

template <bool kNear>
__global__ void balls_group_fill(const uint32_t* __restrict__ cand, const uint32_t* __restrict__ down, uint32_t max_edt2,
                                 size_t nc, Grid g, Tiles gt, size_t g0, size_t g1,
                                 const unsigned long long* __restrict__ gfloor,
                                 const unsigned long long* __restrict__ goff, unsigned long long base,
                                 unsigned int* __restrict__ gcursor, unsigned long long* __restrict__ groups) {
    const size_t per_z = static_cast<size_t>(gt.TX) * gt.TY;
    const int gz0 = static_cast<int>(g0 / per_z), gz1 = static_cast<int>((g1 - 1) / per_z) + 1;
    PMA_GRID_STRIDE(i, nc) {
        int x, y, z;
        g.coords(cand[i], x, y, z);
        const uint32_t R = max_edt2 - down[i];
        for_each_group(g, gt, x, y, z, R, gz0, gz1,
                       FillGroup<kNear>{gfloor, goff, base, g0, g1, gcursor, groups, ball_key(g, x, y, z, R)});
    }
}

__device__ __forceinline__ int4 decode_key(unsigned long long key, Grid g, FastDiv fsz) {
    const uint32_t lex = 0xFFFFFFFFu - static_cast<uint32_t>(key);
    const uint32_t xy = fsz.div(lex), x = g.fy.div(xy);
    return make_int4(static_cast<int>(x), static_cast<int>(xy - x * static_cast<uint32_t>(g.SY)),
                     static_cast<int>(lex - xy * static_cast<uint32_t>(g.SZ)), static_cast<int>(key >> 32));
}

// 32-bit arithmetic while every offset is below 2^15 (the squared sum then fits), 64-bit
// otherwise (only balls of radius >= 2^15, e.g. the virtual-solid distances of a long empty
// volume).
__device__ __forceinline__ bool covers(int4 c, int vx, int vy, int vz) {
    const unsigned dx = static_cast<unsigned>(abs(vx - c.x)), dy = static_cast<unsigned>(abs(vy - c.y));
    const unsigned dz = static_cast<unsigned>(abs(vz - c.z));
    if ((dx | dy | dz) < (1u << 15)) return dx * dx + dy * dy + dz * dz <= static_cast<uint32_t>(c.w);
    const unsigned long long d2 = static_cast<unsigned long long>(dx) * dx +
                                  static_cast<unsigned long long>(dy) * dy + static_cast<unsigned long long>(dz) * dz;
    return d2 <= static_cast<uint32_t>(c.w);
}

__device__ __forceinline__ unsigned long long pos_key(int4 c, Grid g) {
    const uint32_t lex = (static_cast<uint32_t>(c.x) * g.SY + static_cast<uint32_t>(c.y)) * static_cast<uint32_t>(g.SZ) +
                         static_cast<uint32_t>(c.z);
    return (static_cast<unsigned long long>(static_cast<uint32_t>(c.w)) << 32) | (0xFFFFFFFFu - lex);
}

// Lanes of a warp's box lie at y + 4 x + 16 z: the y (x) values present in a lane mask, as 4 bits.
__device__ __forceinline__ unsigned int fold_y(unsigned int m) {
    m |= m >> 16;
    m |= m >> 8;
    m |= m >> 4;
    return m & 15u;
}
__device__ __forceinline__ unsigned int fold_x(unsigned int m) {
    m |= m >> 16;
    return ((m & 0xFu) ? 1u : 0u) | ((m & 0xF0u) ? 2u : 0u) | ((m & 0xF00u) ? 4u : 0u) | ((m & 0xF000u) ? 8u : 0u);
}

constexpr int kSub = kGroup * kGroup * kGroup;  // tiles of a group

// Tile `sub` of a group, which may lie outside the volume.
__device__ __forceinline__ void tile_of(Tiles gt, size_t group, int sub, int& tx, int& ty, int& tz) {
    const size_t rest = group / gt.TY;
    ty = static_cast<int>(group % gt.TY) * kGroup + sub % kGroup;
    tx = static_cast<int>(rest % gt.TX) * kGroup + sub / kGroup % kGroup;
    tz = static_cast<int>(rest / gt.TX) * kGroup + sub / (kGroup * kGroup);
}

// Where a tile's list starts: each tile of a group has room for the whole group's list.
__device__ __forceinline__ unsigned long long tile_list(unsigned long long group_at, unsigned int group_count, int sub) {
    return group_at * kSub + static_cast<unsigned long long>(group_count) * sub;
}

// Splits each group's list into its tiles' lists: the entries that reach the tile and are not below
// its floor. One CTA per group; an entry is decoded once and tested against the eight tiles, a
// warp takes its places in all eight lists with one atomic instruction in shared memory.
constexpr int kSplitThreads = 256;

__global__ void __launch_bounds__(kSplitThreads) balls_split(Grid g, FastDiv fsz, Tiles t, Tiles gt, size_t g0,
                                                             const unsigned long long* __restrict__ floor,
                                                             const unsigned int* __restrict__ gcount,
                                                             const unsigned long long* __restrict__ goff, unsigned long long base,
                                                             unsigned long long tile_base,
                                                             const unsigned long long* __restrict__ groups,
                                                             unsigned long long* __restrict__ entries,
                                                             unsigned int* __restrict__ tcount) {
    static_assert(kGroup == 2, "two tiles an axis");
    __shared__ unsigned int s_n[kSub];
    __shared__ unsigned long long s_floor[kSub];
    const size_t group = g0 + blockIdx.x;
    const unsigned lane = threadIdx.x & 31;
    int tx, ty, tz;
    if (threadIdx.x < kSub) {
        tile_of(gt, group, threadIdx.x, tx, ty, tz);
        s_n[threadIdx.x] = 0;
        s_floor[threadIdx.x] = ty < t.TY && tx < t.TX && tz < t.TZ ? floor[t.id(tx, ty, tz)] : ~0ull;  // no tile: nothing
    }
    tile_of(gt, group, 0, tx, ty, tz);
    __syncthreads();
    const unsigned int L = gcount[group];
    const unsigned long long* list = groups + (goff[group] - base);
    unsigned long long* out = entries + tile_list(goff[group] - tile_base, L, 0);
    // voxels a ball must reach along an axis, from the tile's first to its last
    auto reach = [](int c, int tile, int size) {
        const int lo = tile * kTile, hi = min(lo + kTile, size) - 1;
        return max(max(lo - c, c - hi), 0);
    };
    for (unsigned int i0 = 0; i0 < L; i0 += kSplitThreads) {
        const unsigned int i = i0 + threadIdx.x;
        const unsigned long long key = i < L ? list[i] : 0ull;
        unsigned int to = 0;  // tiles that take the entry
        if (i < L) {
            const int4 c = decode_key(key, g, fsz);
            int dx[kGroup], dy[kGroup], dz[kGroup];
#pragma unroll
            for (int k = 0; k < kGroup; ++k) {
                dx[k] = reach(c.x, tx + k, g.SX);
                dy[k] = reach(c.y, ty + k, g.SY);
                dz[k] = reach(c.z, tz + k, g.SZ);
            }
#pragma unroll
            for (int sub = 0; sub < kSub; ++sub)
                if (key >= s_floor[sub] && covers(make_int4(dx[sub / 2 % 2], dy[sub % 2], dz[sub / 4], c.w), 0, 0, 0)) to |= 1u << sub;
        }
        unsigned int mine = 0, n = 0;  // the lanes that go to tile `lane`
#pragma unroll
        for (int sub = 0; sub < kSub; ++sub) {
            const unsigned int m = __ballot_sync(0xFFFFFFFFu, (to >> sub) & 1u);
            if (lane == static_cast<unsigned>(sub)) mine = m;
        }
        if (lane < kSub && mine) n = atomicAdd(&s_n[lane], __popc(mine));
#pragma unroll
        for (int sub = 0; sub < kSub; ++sub) {
            const unsigned int m = __shfl_sync(0xFFFFFFFFu, mine, sub), from = __shfl_sync(0xFFFFFFFFu, n, sub);
            if ((to >> sub) & 1u) out[static_cast<unsigned long long>(L) * sub + from + __popc(m & ((1u << lane) - 1u))] = key;
        }
    }
    __syncthreads();
    if (threadIdx.x < kSub) tcount[static_cast<size_t>(blockIdx.x) * kSub + threadIdx.x] = s_n[threadIdx.x];
}

// One CTA per tile of the groups from g0 on: winner key of each voxel.
//
// The tile's list is taken in chunks of up to kListCap entries. Each chunk is decoded into
// shared memory ordered by radius, largest first (a counting sort on r^2 when the chunk's r^2
// span fits kSortBins, else left in list order). A warp covers a 2 x 4 x 4 box of voxels and
// keeps, per lane, the largest covering key so far (best). It reads the chunk 32 entries at a
// time: an entry can matter only if its ball reaches the box of the lanes whose best is not above
// the radii still to come; the lanes test every such entry against their own voxel.
// In a chunk sorted by radius the warp stops once no lane is left whose best has an r^2 of at most
// the next entry's (every later entry's key is smaller). The result is the largest covering key over
// the whole list, i.e. the covering centre of largest key.
constexpr int kSortBins = 2048;

__global__ void __launch_bounds__(kTileVox, 4) balls_tile_gather(
    const uint32_t* __restrict__ edt2, Grid g, FastDiv fsz, Tiles t, Tiles gt, size_t g0,
    const unsigned int* __restrict__ tcount, const unsigned int* __restrict__ gcount,
    const unsigned long long* __restrict__ goff, unsigned long long tile_base, const unsigned long long* __restrict__ entries,
    unsigned long long* __restrict__ keys, unsigned int* __restrict__ err) {
    __shared__ int4 s_pos[kListCap];
    __shared__ unsigned int s_bin[kSortBins];
    __shared__ unsigned int s_rmin, s_rmax, s_wsum[kTileVox / 32];
    const size_t group = g0 + blockIdx.x / kSub;
    int tx, ty, tz;
    tile_of(gt, group, blockIdx.x % kSub, tx, ty, tz);
    if (ty >= t.TY || tx >= t.TX || tz >= t.TZ) return;
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // a warp covers a box of 2 x 4 x 4 voxels (z, x, y)
    const int by0 = ty * kTile + (warp & 1) * 4, bx0 = tx * kTile + ((warp >> 1) & 1) * 4, bz0 = tz * kTile + (warp >> 2) * 2;
    const int vy = by0 + (lane & 3), vx = bx0 + ((lane >> 2) & 3), vz = bz0 + (lane >> 4);
    const bool inside = vx < g.SX && vy < g.SY && vz < g.SZ;
    const size_t v = inside ? g.idx(vx, vy, vz) : 0;
    const bool void_voxel = inside && edt2[v] != 0;
    const unsigned int L = tcount[blockIdx.x];
    const unsigned long long* list = entries + tile_list(goff[group] - tile_base, gcount[group], blockIdx.x % kSub);
    unsigned long long best = void_voxel ? 0ull : ~0ull;
    for (unsigned int c0 = 0; c0 < L; c0 += kListCap) {
        const unsigned int m = min(static_cast<unsigned int>(kListCap), L - c0);
        // radius span of the chunk; the entries stay in registers
        constexpr int kPer = kListCap / kTileVox;
        unsigned long long k[kPer];
        if (threadIdx.x == 0) {
            s_rmin = 0xFFFFFFFFu;
            s_rmax = 0;
        }
        for (int i = threadIdx.x; i < kSortBins; i += blockDim.x) s_bin[i] = 0;
        __syncthreads();
        unsigned int rmin = 0xFFFFFFFFu, rmax = 0;
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
            const unsigned int i = threadIdx.x + q * kTileVox;
            k[q] = i < m ? list[c0 + i] : 0ull;
            if (i < m) {
                rmin = min(rmin, static_cast<unsigned int>(k[q] >> 32));
                rmax = max(rmax, static_cast<unsigned int>(k[q] >> 32));
            }
        }
        rmin = __reduce_min_sync(0xFFFFFFFFu, rmin);
        rmax = __reduce_max_sync(0xFFFFFFFFu, rmax);
        if (lane == 0) {
            atomicMin(&s_rmin, rmin);
            atomicMax(&s_rmax, rmax);
        }
        __syncthreads();
        const unsigned int r_hi = s_rmax;
        if (!__syncthreads_or(static_cast<uint32_t>(best >> 32) <= r_hi)) continue;  // no voxel of the block can gain
        const bool sorted = r_hi - s_rmin < static_cast<unsigned int>(kSortBins);
        unsigned int rank[kPer];
        if (sorted) {  // counting sort, descending r^2: bin = r_hi - r^2
            // equal radii are common: lanes with the same bin take their ranks with one atomic
#pragma unroll
            for (int q = 0; q < kPer; ++q) {
                const unsigned int i = threadIdx.x + q * kTileVox;
                const unsigned int bin = i < m ? r_hi - static_cast<unsigned int>(k[q] >> 32) : 0xFFFFFFFFu;
                const unsigned int peers = __match_any_sync(0xFFFFFFFFu, bin);
                const int leader = __ffs(peers) - 1;
                unsigned int at = 0;
                if (bin != 0xFFFFFFFFu && static_cast<int>(lane) == leader) at = atomicAdd(&s_bin[bin], __popc(peers));
                at = __shfl_sync(0xFFFFFFFFu, at, leader);
                rank[q] = at + __popc(peers & ((1u << lane) - 1u));
            }
            __syncthreads();
            // exclusive scan of the bins, four per thread
            unsigned int b4[kSortBins / kTileVox], sum = 0;
#pragma unroll
            for (int q = 0; q < kSortBins / kTileVox; ++q) {
                b4[q] = s_bin[threadIdx.x * (kSortBins / kTileVox) + q];
                sum += b4[q];
            }
            unsigned int incl = sum;
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned int t2 = __shfl_up_sync(0xFFFFFFFFu, incl, o);
                if (lane >= static_cast<unsigned>(o)) incl += t2;
            }
            if (lane == 31) s_wsum[warp] = incl;
            __syncthreads();
            if (warp == 0) {
                unsigned int w = lane < kTileVox / 32 ? s_wsum[lane] : 0u;
                for (int o = 1; o < 32; o <<= 1) {
                    const unsigned int t2 = __shfl_up_sync(0xFFFFFFFFu, w, o);
                    if (lane >= static_cast<unsigned>(o)) w += t2;
                }
                if (lane < kTileVox / 32) s_wsum[lane] = w;
            }
            __syncthreads();
            unsigned int run = (warp ? s_wsum[warp - 1] : 0u) + incl - sum;
#pragma unroll
            for (int q = 0; q < kSortBins / kTileVox; ++q) {
                s_bin[threadIdx.x * (kSortBins / kTileVox) + q] = run;
                run += b4[q];
            }
            __syncthreads();
        }
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
            const unsigned int i = threadIdx.x + q * kTileVox;
            if (i < m) {
                const unsigned int at = sorted ? s_bin[r_hi - static_cast<unsigned int>(k[q] >> 32)] + rank[q] : i;
                s_pos[at] = decode_key(k[q], g, fsz);
            }
        }
        __syncthreads();
        // the warp's pass over the chunk; open: lanes whose best may still be beaten, in the box
        // [lo, hi] of which a ball has to reach
        unsigned int open = 0;
        int lox = 0, loy = 0, loz = 0, hix = 0, hiy = 0, hiz = 0;
        for (unsigned int e0 = 0; e0 < m; e0 += 32) {
            const uint32_t most = sorted ? static_cast<uint32_t>(s_pos[e0].w) : r_hi;  // r^2 from here on
            const unsigned int now = __ballot_sync(0xFFFFFFFFu, static_cast<uint32_t>(best >> 32) <= most);
            if (!now) break;
            if (now != open) {
                open = now;
                const unsigned int y4 = fold_y(now), x4 = fold_x(now);
                loy = by0 + __ffs(y4) - 1;
                hiy = by0 + 31 - __clz(y4);
                lox = bx0 + __ffs(x4) - 1;
                hix = bx0 + 31 - __clz(x4);
                loz = bz0 + ((now & 0xFFFFu) ? 0 : 1);
                hiz = bz0 + ((now >> 16) ? 1 : 0);
            }
            bool cand = false;
            if (e0 + lane < m) {
                const int4 c = s_pos[e0 + lane];
                const int dx = max(max(lox - c.x, c.x - hix), 0), dy = max(max(loy - c.y, c.y - hiy), 0),
                          dz = max(max(loz - c.z, c.z - hiz), 0);
                cand = covers(make_int4(dx, dy, dz, c.w), 0, 0, 0);
            }
            unsigned int mask = __ballot_sync(0xFFFFFFFFu, cand);
            while (mask) {
                const int b = __ffs(mask) - 1;
                mask &= mask - 1;
                const int4 c = s_pos[e0 + b];
                if (covers(c, vx, vy, vz)) {
                    const unsigned long long kc = pos_key(c, g);
                    if (kc > best) best = kc;  // never where best is ~0: solid or outside
                }
            }
        }
        if (c0 + kListCap < L) __syncthreads();  // before the next chunk replaces s_pos
    }
    if (inside) {
        if (void_voxel && best == 0) atomicOr(err, 2u);  // no kept ball covers a void voxel
        keys[v] = void_voxel ? best : ~0ull;
    }
}

__global__ void balls_unpack(const unsigned long long* __restrict__ keys, Grid g, size_t n,
                             uint32_t* __restrict__ crad2, uint32_t* __restrict__ cxo,
                             uint32_t* __restrict__ cyo, uint32_t* __restrict__ czo,
                             uint8_t* __restrict__ mask) {
    const uint32_t syz = static_cast<uint32_t>(g.SY) * g.SZ;
    PMA_GRID_STRIDE(v, n) {
        const unsigned long long k = keys[v];
        if (k == ~0ull || k == 0) {
            crad2[v] = 0;
            cxo[v] = 0xFFFFFFFFu;
            cyo[v] = 0xFFFFFFFFu;
            czo[v] = 0xFFFFFFFFu;
            mask[v] = 0;
        } else {
            const uint32_t lex = 0xFFFFFFFFu - static_cast<uint32_t>(k);
            crad2[v] = static_cast<uint32_t>(k >> 32);
            cxo[v] = lex / syz;
            const uint32_t rem = lex % syz;
            cyo[v] = rem / g.SZ;
            czo[v] = rem % g.SZ;
            mask[v] = 127;
        }
    }
}

// Marks winning centres (OUTER = 255) from the packed keys.
__global__ void balls_mark(const unsigned long long* __restrict__ keys, Grid g, size_t n,
                           uint8_t* __restrict__ mask) {
    const uint32_t syz = static_cast<uint32_t>(g.SY) * g.SZ;
    const uint32_t limit = static_cast<uint32_t>(n);
    PMA_GRID_STRIDE(v, n) {
        const unsigned long long k = keys[v];
        if (k == ~0ull || k == 0) continue;
        const uint32_t lex = 0xFFFFFFFFu - static_cast<uint32_t>(k);
        if (lex >= limit) continue;
        const uint32_t x = lex / syz, rem = lex % syz;
        mask[g.idx(static_cast<int>(x), static_cast<int>(rem / g.SZ), static_cast<int>(rem % g.SZ))] = 255;
    }
}

__global__ void count_value(const uint8_t* __restrict__ a, size_t n, uint8_t value,
                            unsigned long long* __restrict__ out) {
    unsigned long long c = 0;
    PMA_GRID_STRIDE(v, n) c += (a[v] == value);
    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xFFFFFFFFu, c, o);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(out, c);
}

template <class T>
T* buf(pma_ctx* ctx, const char* tag, size_t count) {
    return static_cast<T*>(ctx->scratch(tag, std::max<size_t>(count, 1) * sizeof(T)));
}

// Group counts as 64-bit values, with a zero past the end (the scan then gives the total).
__global__ void widen_counts(const unsigned int* __restrict__ c, size_t n, unsigned long long* __restrict__ out) {
    PMA_GRID_STRIDE(i, n + 1) out[i] = i < n ? c[i] : 0ull;
}

// Offsets of the first group of each z-slab (and the total at tz).
__global__ void slab_offsets(const unsigned long long* __restrict__ toff, size_t per_z, int tz,
                             unsigned long long* __restrict__ zoff) {
    const int z = blockIdx.x * blockDim.x + threadIdx.x;
    if (z <= tz) zoff[z] = toff[static_cast<size_t>(z) * per_z];
}

}  // namespace

void containing_balls(pma_ctx* ctx, const uint32_t* edt2, pma_dims d, uint32_t max_edt2,
                      uint32_t* crad2, uint32_t* cx, uint32_t* cy, uint32_t* cz, uint8_t* mask,
                      uint64_t* count) {
    KernelTimer kt_stage(ctx, "stage_balls");  // the whole stage, for the untimed remainder
    check_dims(d);
    PMA_REQUIRE(edt2 && crad2 && cx && cy && cz && mask, PMA_ERR_ARGUMENT,
                "pma_containing_balls: null device pointer");
    cudaStream_t s = ctx->stream;
    const size_t n = voxels(d);
    const Grid g{d.sx, d.sy, d.sz};
    const uint32_t nR = max_edt2 + 1;
    const uint32_t ntab = std::min<uint32_t>(nR, kExactTable);
    const unsigned G = grid_for(ctx, n);

    auto* keys = buf<unsigned long long>(ctx, "balls.keys", n);
    auto* mtab = buf<uint32_t>(ctx, "balls.mtab", 3ull * ntab);
    auto* misc = buf<unsigned long long>(ctx, "balls.misc", 4);  // [0] count, [1] err, [2] select
    auto* err = reinterpret_cast<unsigned int*>(misc + 1);
    PMA_CUDA(cudaMemsetAsync(misc, 0, 32, s));

    // Kept centres.
    balls_containment_table<<<div_up(ntab, 128), 128, 0, s>>>(mtab, mtab + ntab, mtab + 2 * ntab, ntab);
    ctx->check_launch("balls_containment_table");
    uint8_t* flags = buf<uint8_t>(ctx, "balls.flags", n);
    uint32_t* cand = buf<uint32_t>(ctx, "balls.cand", n);
    int64_t nc = 0;
    {
        KernelTimer kt(ctx, "balls_candidates");
        const unsigned BY = div_up(d.sy, kBrickY), BX = div_up(d.sx, kBrickX), BZ = div_up(d.sz, kBrickZ);
        balls_candidate_flags<<<BY * BX * BZ, 32 * kBrickX, 0, s>>>(edt2, g, static_cast<int>(BY), static_cast<int>(BX), mtab,
                                                                   ntab, nR, flags, err);
        ctx->check_launch("balls_candidate_flags");
        nc = select_flagged(ctx, thrust::counting_iterator<uint32_t>(0), flags, cand,
                            static_cast<int64_t>(n), reinterpret_cast<int64_t*>(misc + 2));
    }
    unsigned int h_err = 0;
    PMA_CUDA(cudaMemcpyAsync(&h_err, err, 4, cudaMemcpyDeviceToHost, s));
    ctx->sync();
    PMA_REQUIRE(!(h_err & 1u), PMA_ERR_ARGUMENT,
                "pma_containing_balls: max_edt2 is smaller than the largest squared distance");

    // Large volumes take the kept centres by descending radius: the lanes of a warp then visit equally
    // many tiles, floors rise early, and the tile lists come out nearly ordered, so that a gather's
    // later chunks hold smaller balls and are mostly skipped. Below kSortCentres the sort's launches cost
    // more than it saves.
    constexpr int64_t kSortCentres = 1 << 18;
    // of centres in that order every fourth serves for the floors, which are near those of all
    constexpr size_t kFloorStep = 4;
    const bool sorted = nc >= kSortCentres;
    uint32_t* down = buf<uint32_t>(ctx, "balls.down", nc);
    if (nc) {
        balls_radii<<<grid_for(ctx, nc), 256, 0, s>>>(edt2, cand, nc, max_edt2, down);
        ctx->check_launch("balls_radii");
        if (sorted) {
            KernelTimer kt(ctx, "balls_sort");
            int bits = 1;
            while (bits < 32 && (max_edt2 >> bits) != 0) ++bits;
            uint32_t* down2 = buf<uint32_t>(ctx, "balls.down2", nc);
            uint32_t* cand2 = buf<uint32_t>(ctx, "balls.cand2", nc);
            sort_pairs(ctx, down, down2, cand, cand2, nc, bits);
            down = down2;
            cand = cand2;
        }
    }
    // Lists: counts, 64-bit offsets, then fill, split and gather by runs of groups whose entries fit the
    // memory budget. One centre a thread and no strides: the lists keep the order of the centres roughly.
    Tiles t{(d.sx + kTile - 1) / kTile, (d.sy + kTile - 1) / kTile, (d.sz + kTile - 1) / kTile};
    const size_t ntiles = static_cast<size_t>(t.TX) * t.TY * t.TZ;
    const Tiles gt{(t.TX + kGroup - 1) / kGroup, (t.TY + kGroup - 1) / kGroup, (t.TZ + kGroup - 1) / kGroup};
    const size_t per_z = static_cast<size_t>(gt.TX) * gt.TY;
    const size_t ngroups = per_z * gt.TZ;
    // Few groups: dozens of the threads in flight are at one counter. Fill of a 128^3 union (512 groups) 0.26 ms
    // without add_one's grouping, 0.11 with it; of 32 thousand groups (512^3) 0.84 and 0.99.
    const bool near = ngroups < 8192;
    unsigned int* gcount = buf<unsigned int>(ctx, "balls.gcount", ngroups);
    unsigned int* gcursor = buf<unsigned int>(ctx, "balls.gcursor", ngroups);
    auto* goff = buf<unsigned long long>(ctx, "balls.goff", ngroups + 1);
    auto* floor = buf<unsigned long long>(ctx, "balls.floor", ntiles);
    auto* gfloor = buf<unsigned long long>(ctx, "balls.gfloor", ngroups);
    PMA_CUDA(cudaMemsetAsync(gcount, 0, ngroups * 4, s));
    PMA_CUDA(cudaMemsetAsync(gcursor, 0, ngroups * 4, s));
    PMA_CUDA(cudaMemsetAsync(floor, 0, ntiles * 8, s));
    if (nc) {
        KernelTimer kt(ctx, "balls_tile_count");
        const size_t step = sorted ? kFloorStep : 1;
        balls_tile_floor<<<div_up((nc + step - 1) / step, 256), 256, 0, s>>>(cand, down, max_edt2, nc, step, g, t, floor);
        ctx->check_launch("balls_tile_floor");
        balls_group_floor<<<grid_for(ctx, ngroups), 256, 0, s>>>(floor, t, gt, ngroups, gfloor);
        ctx->check_launch("balls_group_floor");
        (near ? balls_group_count<true> : balls_group_count<false>)<<<div_up(nc, 256), 256, 0, s>>>(cand, down, max_edt2, nc, g, gt, gfloor, gcount);
        ctx->check_launch("balls_group_count");
    }
    // 64-bit list offsets by a device scan; the host reads back the offsets at the layers of groups (and
    // those within a layer that does not fit), which choose the runs that fit the memory budget
    auto* tc64 = buf<unsigned long long>(ctx, "balls.tc64", ngroups + 1);
    widen_counts<<<grid_for(ctx, ngroups + 1), 256, 0, s>>>(gcount, ngroups, tc64);
    ctx->check_launch("widen_counts");
    exclusive_sum(ctx, tc64, goff, static_cast<int64_t>(ngroups + 1));
    auto* zoff = buf<unsigned long long>(ctx, "balls.zoff", gt.TZ + 1);
    slab_offsets<<<div_up(gt.TZ + 1, 256), 256, 0, s>>>(goff, per_z, gt.TZ, zoff);
    ctx->check_launch("slab_offsets");
    std::vector<unsigned long long> hz(gt.TZ + 1);
    PMA_CUDA(cudaMemcpyAsync(hz.data(), zoff, (gt.TZ + 1) * 8ull, cudaMemcpyDeviceToHost, s));
    ctx->sync();
    std::vector<unsigned long long> layer;  // offsets of layer layer_z's groups and of the next one's first
    size_t layer_z = ~size_t(0);
    auto layer_at = [&](size_t z) -> const unsigned long long* {
        if (layer_z != z) {
            layer.resize(per_z + 1);
            PMA_CUDA(cudaMemcpyAsync(layer.data(), goff + z * per_z, (per_z + 1) * 8, cudaMemcpyDeviceToHost, s));
            ctx->sync();
            layer_z = z;
        }
        return layer.data();
    };
    auto offset_of = [&](size_t group) {
        const size_t z = group / per_z;
        return group == z * per_z ? hz[z] : layer_at(z)[group - z * per_z];
    };
    size_t free_b = 0, total_b = 0;
    PMA_CUDA(cudaMemGetInfo(&free_b, &total_b));
    // Group lists by runs of groups that fit the memory budget, and of these the tiles' lists (with room for
    // every entry of the group in each of its tiles) by runs that fit theirs: whole layers of groups, or a
    // part of one where a layer alone takes more (wide and thin volumes; at least one group).
    const unsigned long long budget = std::max<unsigned long long>(1ull << 20, std::min<unsigned long long>(free_b / 6, 32ull << 30) / 8);
    // 16 bytes a voxel: with the groups' lists what lists of the tiles alone would take, four to seven slabs. At least
    // 512 MB: runs too short to fill the GPU last as long as their longest lists. With 64 MB a volume with few
    // large pores, whose lists are long, went layer by layer: random field of sigma 14, 160^3 36.9 ms, 256^3 31.8;
    // with 256 MB 13.8 and 32.0, with 512 MB 9.0 and 18.8 (tiles' own lists, without groups, 11.6 and 23.6).
    const unsigned long long tile_bytes = std::min<unsigned long long>({free_b / 6, 8ull << 30, std::max<unsigned long long>(512ull << 20, 16ull * n)});
    const unsigned long long tile_budget = std::max<unsigned long long>(1ull << 17, tile_bytes / (8 * kSub));
    const FastDiv fsz(static_cast<uint32_t>(d.sz));
    struct Run {  // groups [g0, g1), entries [e0, e1)
        size_t g0, g1;
        unsigned long long e0, e1;
    };
    auto runs = [&](size_t g0, size_t end, unsigned long long most, unsigned long long& longest) {
        std::vector<Run> v;
        for (size_t g1; g0 < end; g0 = g1) {
            g1 = group_run_end(hz.data(), per_z, g0, end, most, layer_at);
            v.push_back({g0, g1, offset_of(g0), offset_of(g1)});
            longest = std::max(longest, v.back().e1 - v.back().e0);
        }
        return v;
    };
    unsigned long long fill_room = 0, split_room = 0;
    const std::vector<Run> fills = runs(0, ngroups, budget, fill_room);
    std::vector<std::vector<Run>> splits;
    for (const Run& f : fills) splits.push_back(runs(f.g0, f.g1, tile_budget, split_room));
    size_t most_groups = 0;
    for (const auto& v : splits)
        for (const Run& r : v) most_groups = std::max(most_groups, r.g1 - r.g0);
    auto* groups = buf<unsigned long long>(ctx, "balls.groups", fill_room);
    auto* entries = buf<unsigned long long>(ctx, "balls.entries", split_room * kSub);
    auto* tcount = buf<unsigned int>(ctx, "balls.tcount", most_groups * kSub);
    for (size_t k = 0; k < fills.size(); ++k) {
        const Run& f = fills[k];
        if (nc) {
            KernelTimer kt(ctx, "balls_tile_fill");
            (near ? balls_group_fill<true> : balls_group_fill<false>)<<<div_up(nc, 256), 256, 0, s>>>(
                cand, down, max_edt2, nc, g, gt, f.g0, f.g1, gfloor, goff, f.e0, gcursor, groups);
            ctx->check_launch("balls_group_fill");
        }
        for (const Run& r : splits[k]) {
            const unsigned run = static_cast<unsigned>(r.g1 - r.g0);
            ctx->count("balls.runs", static_cast<double>(r.e1 - r.e0));
            {
                KernelTimer kt(ctx, "balls_split");
                balls_split<<<run, kSplitThreads, 0, s>>>(g, fsz, t, gt, r.g0, floor, gcount, goff, f.e0, r.e0, groups, entries, tcount);
                ctx->check_launch("balls_split");
            }
            KernelTimer kt(ctx, "balls_tile_gather");
            balls_tile_gather<<<run * kSub, kTileVox, 0, s>>>(edt2, g, fsz, t, gt, r.g0, tcount, gcount, goff, r.e0, entries, keys, err);
            ctx->check_launch("balls_tile_gather");
        }
    }
    balls_unpack<<<G, 256, 0, s>>>(keys, g, n, crad2, cx, cy, cz, mask);
    ctx->check_launch("balls_unpack");
    balls_mark<<<G, 256, 0, s>>>(keys, g, n, mask);
    ctx->check_launch("balls_mark");
    PMA_CUDA(cudaMemsetAsync(misc, 0, 8, s));
    count_value<<<G, 256, 0, s>>>(mask, n, 255, misc);
    ctx->check_launch("count_value");
    unsigned long long c = 0;
    PMA_CUDA(cudaMemcpyAsync(&c, misc, 8, cudaMemcpyDeviceToHost, s));
    PMA_CUDA(cudaMemcpyAsync(&h_err, err, 4, cudaMemcpyDeviceToHost, s));
    ctx->sync();
    PMA_REQUIRE(!(h_err & 2u), PMA_ERR_INTERNAL, "pma_containing_balls: uncovered void voxel");
    if (count) *count = c;
}

}  // namespace pma
