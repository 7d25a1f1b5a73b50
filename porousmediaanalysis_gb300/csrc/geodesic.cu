// Geodesic (shortest-path) distances, cavity ids and cavity restarts
// (ShortestPathComputer.cpp:39-511).
//
// The reference settles voxels with Dijkstra over an indexed heap (HeapUtilities.h).
// Every settled distance equals min over void neighbours u of fl(d(u) + w(u, v)); this
// system has one greatest fixed point below the initial values and any monotone
// relaxation that runs until nothing improves reaches it, so the parallel form below is
// bit-identical in float32 (and in float64 against the float64 restatement).
//
// Steps: all step weights w are >= 1 (1, sqrt 2, sqrt 3, or 1 for D3Q7) and in round-to-nearest
// fl(d + w) >= floor(d) + 1, so the predecessor of a voxel of distance in [k, k + 1) has a
// distance below k. Step k therefore settles exactly the unreached voxels whose minimum over
// their neighbours is below k + 1, and their values are final. Each voxel pulls its own value:
// it is written once, by one thread, with no atomics (pushing from the settled voxels instead
// took an atomic minimum and a mark from each of up to nine neighbours that reach a voxel).
// A neighbour settled in the same step may be seen or not: it has distance >= k and
// gives at least k + 1, which settles nothing in step k.
//
// The volume is cut into bricks of 32 x 8 x 8 voxels (y, x, z). A step loads each brick of its
// list with a one-voxel halo into shared memory and evaluates its unreached voxels. A brick
// goes on the next step's list when it still holds unreached voxels that could be settled, or
// when a neighbouring brick settled a voxel next to one of its unreached voxels.
#include "devutil.cuh"

#include <cfloat>
#include <cmath>
#include <cstring>

namespace pma {
namespace {

template <class T> struct Bits;
template <> struct Bits<float> {
    typedef unsigned int U;
    static __device__ __forceinline__ U to(float f) { return __float_as_uint(f); }
    static __device__ __forceinline__ float from(U u) { return __uint_as_float(u); }
    static __device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
    static __host__ __device__ float unknown() { return FLT_MAX; }
    static __device__ __forceinline__ U infinity() { return 0x7F800000u; }
    // Values in shared memory: solid (-1) becomes infinity. Distances are far below the bound used here.
    static __device__ __forceinline__ U to_tile(U u) { return static_cast<int>(u) < 0 ? infinity() : u; }
    static __device__ __forceinline__ bool is_settled(U u) { return u < 0x7F000000u; }
    static __device__ __forceinline__ bool is_unreached(U u) { return u == 0x7F7FFFFFu; }
};
template <> struct Bits<double> {
    typedef unsigned long long U;
    static __device__ __forceinline__ U to(double f) { return static_cast<U>(__double_as_longlong(f)); }
    static __device__ __forceinline__ double from(U u) { return __longlong_as_double(static_cast<long long>(u)); }
    static __device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
    static __host__ __device__ double unknown() { return DBL_MAX; }
    static __device__ __forceinline__ U infinity() { return 0x7FF0000000000000ull; }
    // (the high words alone decide)
    static __device__ __forceinline__ U to_tile(U u) { return static_cast<int>(u >> 32) < 0 ? infinity() : u; }
    static __device__ __forceinline__ bool is_settled(U u) { return static_cast<uint32_t>(u >> 32) < 0x7FE00000u; }
    static __device__ __forceinline__ bool is_unreached(U u) { return static_cast<uint32_t>(u >> 32) == 0x7FEFFFFFu; }
};

struct Geo {
    int SX, SY, SZ;
    __device__ __forceinline__ size_t idx(int x, int y, int z) const {
        return (static_cast<size_t>(z) * SX + x) * SY + y;
    }
};

constexpr int kBrickY = 32, kBrickX = 8, kBrickZ = 8;
constexpr int kHaloY = kBrickY + 2, kHaloX = kBrickX + 2, kHaloZ = kBrickZ + 2;
constexpr int kBrickThreads = 32 * kBrickX;
constexpr int kRing = 4;  // lists in use at once: step k appends to those of k + 1

struct Bricks {
    int BY, BX, BZ;          // bricks per axis
    uint32_t n;              // in all
    uint32_t* list;          // kRing lists of n bricks: step k reads list k & 3
    unsigned int* count;     // [kRing]
    uint32_t* mark;          // per brick: the last step (of all cavities) it was listed for
    unsigned long long* settled;  // voxels settled in this cavity
    unsigned int* walls;          // bit 2i: plane axis i at 0, bit 2i+1: at size-1
};

// Lists a brick for step k (epoch0: steps before this cavity's step 0).
__device__ __forceinline__ void geo_list(const Bricks& b, uint32_t brick, int k, uint32_t epoch0) {
    if (atomicExch(&b.mark[brick], epoch0 + static_cast<uint32_t>(k)) == epoch0 + static_cast<uint32_t>(k)) return;
    const unsigned at = atomicAdd(&b.count[k & (kRing - 1)], 1u);
    if (at < b.n) b.list[static_cast<size_t>(k & (kRing - 1)) * b.n + at] = brick;
}

__device__ __forceinline__ unsigned geo_walls(const Geo& g, int x, int y, int z) {
    unsigned w = 0;
    if (x == 0) w |= 1u;
    if (x == g.SX - 1 && g.SX > 1) w |= 2u;
    if (y == 0) w |= 4u;
    if (y == g.SY - 1 && g.SY > 1) w |= 8u;
    if (z == 0) w |= 16u;
    if (z == g.SZ - 1 && g.SZ > 1) w |= 32u;
    return w;
}

template <class T>
__global__ void geo_init(const uint8_t* __restrict__ solid, size_t n, T* __restrict__ dist,
                         uint32_t* __restrict__ cavity) {
    for (size_t v = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; v < n;
         v += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const bool s = solid[v] != 0;  // SPC.cpp:354-372
        dist[v] = s ? static_cast<T>(-1) : Bits<T>::unknown();
        cavity[v] = s ? 0u : 0xFFFFFFFFu;
    }
}

// The start voxel, settled in step 0; the bricks around it go on the list of step 1.
template <class T>
__global__ void geo_start(Geo g, Bricks b, T* dist, uint32_t* cavity, int x, int y, int z, uint32_t cavity_id, uint32_t epoch0) {
    const int dy = static_cast<int>(threadIdx.x) % 3 - 1, dx = static_cast<int>(threadIdx.x) / 3 % 3 - 1,
              dz = static_cast<int>(threadIdx.x) / 9 - 1;
    if (threadIdx.x == 0) {
        const size_t v = g.idx(x, y, z);
        dist[v] = static_cast<T>(0);
        cavity[v] = cavity_id;
        *b.settled = 1;
        *b.walls = geo_walls(g, x, y, z);
    }
    const int ny = y + dy, nx = x + dx, nz = z + dz;
    if (threadIdx.x < 27 && ny >= 0 && ny < g.SY && nx >= 0 && nx < g.SX && nz >= 0 && nz < g.SZ)
        geo_list(b, static_cast<uint32_t>((nz / kBrickZ * b.BX + nx / kBrickX) * b.BY + ny / kBrickY), 1, epoch0);
}

// A row of three mask words, one bit to either side (26 neighbours) or the bits themselves.
__device__ __forceinline__ unsigned long long geo_spread(unsigned long long m) { return m | m << 1 | m >> 1; }

// Neighbours of the set bits of the halo's rows (34-bit masks, [slice][row]) in row (x, z).
template <bool D3Q7, class F>
__device__ __forceinline__ unsigned long long geo_dilate(F mask, int x, int z) {
    unsigned long long m = 0;
    if (D3Q7) {
        const unsigned long long own = mask(x, z);
        return own << 1 | own >> 1 | mask(x - 1, z) | mask(x + 1, z) | mask(x, z - 1) | mask(x, z + 1);
    }
#pragma unroll
    for (int dz = -1; dz <= 1; ++dz)
#pragma unroll
        for (int dx = -1; dx <= 1; ++dx) m |= mask(x + dx, z + dz);
    return geo_spread(m);
}

// Step k, one block per listed brick. The brick's values and its halo's go to shared memory, with
// one bit mask per row of settled and of unreached voxels; the unreached neighbours of settled
// voxels (a tenth of the brick's) are listed from the masks and evaluated, one thread each; the masks of
// what was settled then say which bricks are listed for the next step. Distances are compared as
// unsigned integers (their bits order as the values do): solid reads as infinity, unreached as
// the largest finite value. The least neighbour per step weight is found first and only three
// sums are formed (rounding is monotone).
// What bounds it: the block's barriers and the bricks' loads (27 KB of a float64 brick with its halo, once
// for each of the about 25 steps that the front takes through a brick: 330 B a voxel). A mid-front step at
// 512^3: 30 and 25 % of the cycles between two instructions, issue slots 49 % and DRAM 42 % busy.
// Five blocks an SM (48 registers, the loads of a whole brick in flight); six spill (1024^3 spinodal,
// float64: 121 against 157 ms). Before and after, ms: that volume 253 -> 121 (a step of 14000
// bricks 130 us, 2.9 TB/s of brick loads); 301 x 257 x 411 field, float32, D3Q7 10.2 -> 6.6.
template <class T, bool D3Q7>
__global__ void __launch_bounds__(kBrickThreads, 5)
    geo_step(Geo g, T w1, T w2, T w3, T* __restrict__ dist, uint32_t* __restrict__ cavity, Bricks b, int k, uint32_t cavity_id,
             uint32_t epoch0) {
    typedef typename Bits<T>::U U;
    constexpr int kRows = kHaloX * kHaloZ, kOwnRows = kBrickX * kBrickZ;
    __shared__ U tile[kRows * kHaloY];
    __shared__ uint32_t settled[kRows], unreached[kRows];
    __shared__ uint16_t todo[kOwnRows * kBrickY];                    // candidates: row * 32 + voxel
    __shared__ uint32_t now[kOwnRows];                               // settled in this step
    __shared__ uint8_t edge[2][kRows];                               // halo columns: bit 0 settled, bit 1 unreached
    __shared__ unsigned s_todo, s_next;                              // s_next: bricks to list (bit 13: this one)
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned n = min(b.count[k & (kRing - 1)], b.n);
    const uint32_t* list = b.list + static_cast<size_t>(k & (kRing - 1)) * b.n;
    if (blockIdx.x == 0 && tid == 0) b.count[(k - 1) & (kRing - 1)] = 0;  // read by the step before, written by the one after next
    const U kSolid = Bits<T>::infinity();
    const T end = static_cast<T>(k) + static_cast<T>(1);
    unsigned long long my_settled = 0;
    unsigned my_walls = 0;
    uint32_t brick = blockIdx.x < n ? list[blockIdx.x] : 0u;
    for (unsigned i = blockIdx.x; i < n; i += gridDim.x) {
        const uint32_t rest = brick / static_cast<uint32_t>(b.BY);
        const int by = static_cast<int>(brick - rest * static_cast<uint32_t>(b.BY));
        const int bz = static_cast<int>(rest / static_cast<uint32_t>(b.BX)), bx = static_cast<int>(rest) - bz * b.BX;
        const int y0 = by * kBrickY, x0 = bx * kBrickX, z0 = bz * kBrickZ;
        if (i + gridDim.x < n) brick = list[i + gridDim.x];
        // Rows of the halo's slices, a warp a row: warp w takes row w of each slice (pointers advance by
        // a plane), then its share of rows 8 and 9. Lane q keeps the masks of the warp's q-th row.
        {
            const int y = y0 + lane;
            const size_t plane = static_cast<size_t>(g.SX) * g.SY;
            uint32_t ms = 0, mu = 0;
            auto put = [&](int q, int r, U u) {
                u = Bits<T>::to_tile(u);
                tile[r * kHaloY + 1 + lane] = u;
                const unsigned bs = __ballot_sync(0xFFFFFFFFu, Bits<T>::is_settled(u)),
                               bu = __ballot_sync(0xFFFFFFFFu, Bits<T>::is_unreached(u));
                if (lane == q) {
                    ms = bs;
                    mu = bu;
                }
            };
            constexpr int kRest = 2 * kHaloZ, kMore = (kRest + 7) / 8;  // rows 8 and 9 of each slice
            // every load first
            U u[kHaloZ], more[kMore], e = kSolid;
            {
                const int x = x0 - 1 + warp;
                const bool in = x >= 0 && x < g.SX && y < g.SY;
                const T* p = dist + (static_cast<long long>(z0 - 1) * g.SX + x) * g.SY + y;
#pragma unroll
                for (int q = 0; q < kHaloZ; ++q, p += plane)
                    u[q] = in && static_cast<unsigned>(z0 - 1 + q) < static_cast<unsigned>(g.SZ) ? Bits<T>::to(*p) : kSolid;
            }
#pragma unroll
            for (int q = 0; q < kMore; ++q) {
                const int i2 = q * 8 + warp, x = x0 - 1 + kBrickX + (i2 & 1), z = z0 - 1 + (i2 >> 1);
                more[q] = kSolid;
                if (i2 < kRest && x < g.SX && static_cast<unsigned>(z) < static_cast<unsigned>(g.SZ) && y < g.SY)
                    more[q] = Bits<T>::to(dist[g.idx(x, y, z)]);
            }
            const int er = tid >> 1, side = tid & 1;  // the halo's columns
            if (tid < 2 * kRows) {
                const int x = x0 - 1 + er % kHaloX, z = z0 - 1 + er / kHaloX, ye = side ? y0 + kBrickY : y0 - 1;
                if (static_cast<unsigned>(x) < static_cast<unsigned>(g.SX) && static_cast<unsigned>(z) < static_cast<unsigned>(g.SZ) &&
                    static_cast<unsigned>(ye) < static_cast<unsigned>(g.SY))
                    e = Bits<T>::to(dist[g.idx(x, ye, z)]);
            }
#pragma unroll
            for (int q = 0; q < kHaloZ; ++q) put(q, q * kHaloX + warp, u[q]);
#pragma unroll
            for (int q = 0; q < kMore; ++q)
                if (q * 8 + warp < kRest) put(kHaloZ + q, ((q * 8 + warp) >> 1) * kHaloX + kBrickX + (warp & 1), more[q]);
            if (tid < 2 * kRows) {
                e = Bits<T>::to_tile(e);
                tile[er * kHaloY + side * (kHaloY - 1)] = e;
                edge[side][er] = (Bits<T>::is_settled(e) ? 1 : 0) | (Bits<T>::is_unreached(e) ? 2 : 0);
            }
            const int own = lane < kHaloZ ? lane * kHaloX + warp : (lane - kHaloZ) * 8 + warp < kRest && lane < kHaloZ + 3
                                ? (((lane - kHaloZ) * 8 + warp) >> 1) * kHaloX + kBrickX + (warp & 1) : -1;
            if (own >= 0) {
                settled[own] = ms;
                unreached[own] = mu;
            }
            if (tid < kOwnRows) now[tid] = 0;
            if (tid == 0) s_todo = s_next = 0;
        }
        __syncthreads();
        // a row's mask with the halo's columns: bits 0 and 33
        auto settled_row = [&](int x, int z) {
            const int r = z * kHaloX + x;
            return static_cast<unsigned long long>(settled[r]) << 1 | (edge[0][r] & 1u) | static_cast<unsigned long long>(edge[1][r] & 1u) << 33;
        };
        if (tid < kOwnRows) {
            const int x = tid % kBrickX + 1, z = tid / kBrickX + 1;
            uint32_t c = static_cast<uint32_t>(geo_dilate<D3Q7>(settled_row, x, z) >> 1) & unreached[z * kHaloX + x];
            uint32_t at = c ? atomicAdd(&s_todo, static_cast<unsigned>(__popc(c))) : 0u;
            for (; c; c &= c - 1) todo[at++] = static_cast<uint16_t>(tid * 32 + __ffs(c) - 1);
        }
        __syncthreads();
        const unsigned m = s_todo;
        for (unsigned c = tid; c < m; c += kBrickThreads) {
            const int own = todo[c], ly = own & 31, r = own >> 5, lx = r % kBrickX, lz = r / kBrickX;
            const U* q = tile + ((lz + 1) * kHaloX + lx + 1) * kHaloY + ly + 1;
            constexpr int DX = kHaloY, DZ = kHaloX * kHaloY;
            U face = min(min(min(q[-1], q[1]), min(q[-DX], q[DX])), min(q[-DZ], q[DZ]));
            T t = Bits<T>::add(Bits<T>::from(face), D3Q7 ? static_cast<T>(1) : w1);
            if (!D3Q7) {
                U e = min(min(q[-DX - 1], q[-DX + 1]), min(q[DX - 1], q[DX + 1]));
                e = min(e, min(min(q[-DZ - 1], q[-DZ + 1]), min(q[-DZ - DX], q[-DZ + DX])));
                e = min(e, min(min(q[DZ - 1], q[DZ + 1]), min(q[DZ - DX], q[DZ + DX])));
                U d = min(min(q[-DZ - DX - 1], q[-DZ - DX + 1]), min(q[-DZ + DX - 1], q[-DZ + DX + 1]));
                d = min(d, min(min(q[DZ - DX - 1], q[DZ - DX + 1]), min(q[DZ + DX - 1], q[DZ + DX + 1])));
                const T t2 = Bits<T>::add(Bits<T>::from(e), w2), t3 = Bits<T>::add(Bits<T>::from(d), w3);
                t = t2 < t ? t2 : t;
                t = t3 < t ? t3 : t;
            }
            if (t < end) {
                const int y = y0 + ly, x = x0 + lx, z = z0 + lz;
                const size_t v = g.idx(x, y, z);
                dist[v] = t;
                cavity[v] = cavity_id;
                ++my_settled;
                my_walls |= geo_walls(g, x, y, z);
                atomicOr(&now[r], 1u << ly);
            } else {
                s_next = 1u << 13;  // a later step's: nothing else is in s_next yet
            }
        }
        __syncthreads();
        if (tid < kRows) {  // unreached neighbours of what was settled, row by row of the halo
            const int px = tid % kHaloX, pz = tid / kHaloX;
            auto mask = [&](int mx, int mz) {
                return mx >= 1 && mx <= kBrickX && mz >= 1 && mz <= kBrickZ
                           ? static_cast<unsigned long long>(now[(mz - 1) * kBrickX + mx - 1]) << 1
                           : 0ull;
            };
            const unsigned long long open = static_cast<unsigned long long>(unreached[tid]) << 1 | (edge[0][tid] >> 1) |
                                            static_cast<unsigned long long>(edge[1][tid] >> 1) << 33;
            const unsigned long long hit = geo_dilate<D3Q7>(mask, px, pz) & open & ~mask(px, pz);
            const int sz = pz == 0 ? 0 : (pz == kHaloZ - 1 ? 2 : 1), sx = px == 0 ? 0 : (px == kHaloX - 1 ? 2 : 1);
            unsigned next = 0;
            if (hit & 1ull) next |= 1u;
            if (hit & 0x1FFFFFFFEull) next |= 2u;
            if (hit >> 33) next |= 4u;
            if (next) atomicOr(&s_next, next << (sz * 9 + sx * 3));
        }
        __syncthreads();
        if (tid < 27 && ((s_next >> tid) & 1u)) {
            const int nz = bz + tid / 9 - 1, nx = bx + tid / 3 % 3 - 1, ny = by + tid % 3 - 1;
            if (nz >= 0 && nz < b.BZ && nx >= 0 && nx < b.BX && ny >= 0 && ny < b.BY)
                geo_list(b, static_cast<uint32_t>((nz * b.BX + nx) * b.BY + ny), k + 1, epoch0);
        }
        // no barrier: what the next brick's loads overwrite was read before the last one, and s_next is read
        // by the warp whose first thread clears it, behind votes of the whole warp (put's): every lane has
        // branched on its bit by then
    }
    for (int o = 16; o > 0; o >>= 1) my_settled += __shfl_xor_sync(0xFFFFFFFFu, my_settled, o);
    my_walls = __reduce_or_sync(0xFFFFFFFFu, my_walls);
    if (lane == 0) {
        if (my_settled) atomicAdd(b.settled, my_settled);
        if (my_walls) atomicOr(b.walls, my_walls);
    }
}

// Start-voxel search on box shells h0 .. h0+nh-1 around the centre, in the reference's
// visiting order (SPC.cpp:460-511). Writes the smallest (shell, order) key of a void,
// unreached voxel.
template <class T>
__global__ void geo_shell_search(const uint8_t* __restrict__ solid, const T* __restrict__ dist,
                                 Geo g, int cx, int cy, int cz, int h0, int nh,
                                 unsigned long long* __restrict__ best) {
    const int s[3] = {g.SX, g.SY, g.SZ};
    const int c[3] = {cx, cy, cz};
    const int h = h0 + blockIdx.y;
    if (blockIdx.y >= nh) return;
    // segment sizes in order (k, f)
    unsigned long long off = 0;
    unsigned long long t = blockIdx.x * static_cast<unsigned long long>(blockDim.x) + threadIdx.x;
    for (int k = 0; k < 3; ++k) {
        const int a = (k == 0) ? 1 : 0, b = (k == 2) ? 1 : 2;
        const int a0 = max(c[a] - h, 0), a1 = min(c[a] + h, s[a] - 1);
        const int b0 = max(c[b] - h, 0), b1 = min(c[b] + h, s[b] - 1);
        const int f0 = max(c[k] - h, 0), f1 = min(c[k] + h, s[k] - 1);
        const int nf = (f0 == f1) ? 1 : 2;
        const unsigned long long na = a1 - a0 + 1, nb = b1 - b0 + 1;
        const unsigned long long seg = static_cast<unsigned long long>(nf) * na * nb;
        for (unsigned long long i = t; i < seg; i += gridDim.x * static_cast<unsigned long long>(blockDim.x)) {
            const int f = static_cast<int>(i / (na * nb));
            const unsigned long long r = i % (na * nb);
            int p[3];
            p[a] = a0 + static_cast<int>(r / nb);
            p[b] = b0 + static_cast<int>(r % nb);
            p[k] = f == 0 ? f0 : f1;
            const size_t v = g.idx(p[0], p[1], p[2]);
            if (solid[v] == 0 && dist[v] == Bits<T>::unknown())
                atomicMin(best, (static_cast<unsigned long long>(blockIdx.y) << 40) | (off + i));
        }
        off += seg;
    }
}

}  // namespace

template <class T>
std::vector<pma_cavity> geodesic(pma_ctx* ctx, const uint8_t* solid, pma_dims d, pma_stencil st, T* dist,
                                 uint32_t* cavity) {
    KernelTimer kt_stage(ctx, "stage_geodesic");  // the whole stage, for the untimed remainder
    check_dims(d);
    PMA_REQUIRE(solid && dist && cavity, PMA_ERR_ARGUMENT, "pma_geodesic: null device pointer");
    cudaStream_t s = ctx->stream;
    const size_t n = voxels(d);
    const Geo g{d.sx, d.sy, d.sz};
    const int d3q7 = st == PMA_D3Q7 ? 1 : 0;
    const T w1 = std::sqrt(static_cast<T>(1)), w2 = std::sqrt(static_cast<T>(2)),
            w3 = std::sqrt(static_cast<T>(3));  // SPC.cpp:31-36
    const unsigned grid = static_cast<unsigned>(std::min<size_t>(div_up(n, 256), ctx->num_sms * 16ull));

    Bricks br;
    br.BY = (d.sy + kBrickY - 1) / kBrickY;
    br.BX = (d.sx + kBrickX - 1) / kBrickX;
    br.BZ = (d.sz + kBrickZ - 1) / kBrickZ;
    const size_t nbricks = static_cast<size_t>(br.BY) * br.BX * br.BZ;
    br.n = static_cast<uint32_t>(nbricks);
    br.list = static_cast<uint32_t*>(ctx->scratch("geo.list", kRing * nbricks * 4));
    br.mark = static_cast<uint32_t*>(ctx->scratch("geo.mark", nbricks * 4));
    auto* misc = static_cast<unsigned long long*>(ctx->scratch("geo.misc", 64));
    br.count = reinterpret_cast<unsigned int*>(misc);          // 4 x u32 = misc[0..1]
    br.walls = reinterpret_cast<unsigned int*>(misc + 3);      // misc[3] low
    br.settled = misc + 4;
    unsigned long long* best = misc + 5;
    PMA_CUDA(cudaMemsetAsync(br.mark, 0, nbricks * 4, s));
    uint32_t epoch0 = 0;  // steps of the cavities before this one: marks of different cavities differ

    geo_init<T><<<grid, 256, 0, s>>>(solid, n, dist, cavity);
    ctx->check_launch("geo_init");

    // SPC.cpp:443-458: centre = round(size * 0.5) clipped to size - 1.
    int sz3[3] = {d.sx, d.sy, d.sz}, c[3];
    for (int i = 0; i < 3; ++i) c[i] = std::min(static_cast<int>(sz3[i] * 0.5 + 0.5), sz3[i] - 1);
    int maxh = 0;
    for (int i = 0; i < 3; ++i) maxh = std::max(maxh, std::max(sz3[i] - 1 - c[i], c[i]));
    int walls_total = 0;
    for (int i = 0; i < 3; ++i) walls_total += (sz3[i] == 1) ? 1 : 2;
    const size_t center_idx = (static_cast<size_t>(c[2]) * d.sx + c[0]) * d.sy + c[1];

    auto* h = static_cast<unsigned long long*>(ctx->host_staging(64));
    int half = 0;
    uint32_t cavity_id = 0;
    std::vector<pma_cavity> rows;
    const int max_steps_per_sync = 32;
    const uint64_t bucket_limit = ctx->limits.geodesic_buckets ? ctx->limits.geodesic_buckets : 2ull * n + 64;
    const unsigned step_grid = static_cast<unsigned>(std::min<size_t>(nbricks, ctx->num_sms * 5ull));  // all resident
    while (true) {  // SPC.cpp:94-140
        ++half;
        // SelectStartingPosition (SPC.cpp:396-426)
        bool found = false;
        int start[3] = {0, 0, 0};
        {
            uint8_t sv = 1;
            T dv = 0;
            PMA_CUDA(cudaMemcpyAsync(&sv, solid + center_idx, 1, cudaMemcpyDeviceToHost, s));
            PMA_CUDA(cudaMemcpyAsync(&dv, dist + center_idx, sizeof(T), cudaMemcpyDeviceToHost, s));
            ctx->sync();
            if (sv == 0 && dv == Bits<T>::unknown()) {
                found = true;
                for (int i = 0; i < 3; ++i) start[i] = c[i];
            }
        }
        while (!found && half < maxh) {
            const int nh = std::min(16, maxh - half);
            PMA_CUDA(cudaMemsetAsync(best, 0xFF, 8, s));
            unsigned long long face = 2ull * std::max(d.sx, std::max(d.sy, d.sz)) *
                                      std::max(d.sx, std::max(d.sy, d.sz));
            unsigned gx = static_cast<unsigned>(std::min<unsigned long long>((face + 255) / 256, 4096));
            geo_shell_search<T><<<dim3(gx, nh), 256, 0, s>>>(solid, dist, g, c[0], c[1], c[2], half, nh, best);
            ctx->check_launch("geo_shell_search");
            PMA_CUDA(cudaMemcpyAsync(h, best, 8, cudaMemcpyDeviceToHost, s));
            ctx->sync();
            const unsigned long long b = h[0];
            if (b == ~0ull) {
                half += nh;
                continue;
            }
            half += static_cast<int>(b >> 40);
            unsigned long long flat = b & ((1ull << 40) - 1);
            // decode in the same segment order as the kernel
            for (int k = 0; k < 3 && !found; ++k) {
                const int a = (k == 0) ? 1 : 0, bb = (k == 2) ? 1 : 2;
                const int a0 = std::max(c[a] - half, 0), a1 = std::min(c[a] + half, sz3[a] - 1);
                const int b0 = std::max(c[bb] - half, 0), b1 = std::min(c[bb] + half, sz3[bb] - 1);
                const int f0 = std::max(c[k] - half, 0), f1 = std::min(c[k] + half, sz3[k] - 1);
                const int nf = (f0 == f1) ? 1 : 2;
                const unsigned long long na = a1 - a0 + 1, nb = b1 - b0 + 1, seg = nf * na * nb;
                if (flat < seg) {
                    const int fi = static_cast<int>(flat / (na * nb));
                    const unsigned long long r = flat % (na * nb);
                    start[a] = a0 + static_cast<int>(r / nb);
                    start[bb] = b0 + static_cast<int>(r % nb);
                    start[k] = fi == 0 ? f0 : f1;
                    found = true;
                } else {
                    flat -= seg;
                }
            }
            PMA_REQUIRE(found, PMA_ERR_INTERNAL, "geodesic: shell search decode failed");
        }
        if (!found) break;

        cavity_id += 127;
        PMA_CUDA(cudaMemsetAsync(misc, 0, 5 * 8, s));  // counts, walls, settled
        geo_start<T><<<1, 32, 0, s>>>(g, br, dist, cavity, start[0], start[1], start[2], cavity_id, epoch0);
        ctx->check_launch("geo_start");
        int k = 1;
        while (true) {
            KernelTimer kt(ctx, "geo_bucket");
            // up to the next multiple of max_steps_per_sync: the bucket limit is looked at there (step 0 was geo_start's)
            const int from = k, to = (k / max_steps_per_sync + 1) * max_steps_per_sync;
            for (; k < to; ++k) {
                if (d3q7) geo_step<T, true><<<step_grid, kBrickThreads, 0, s>>>(g, w1, w2, w3, dist, cavity, br, k, cavity_id, epoch0);
                else geo_step<T, false><<<step_grid, kBrickThreads, 0, s>>>(g, w1, w2, w3, dist, cavity, br, k, cavity_id, epoch0);
            }
            ctx->count_launch(to - from - 1);
            ctx->check_launch("geo_step");
            ReadBack rb;
            rb.add(h, misc, 5 * 8);
            read_back(ctx, rb);
            // the list of step k holds all pending work
            if (reinterpret_cast<const unsigned*>(h)[k & (kRing - 1)] == 0) break;
            // Distances are below 2 per voxel step, so no step can exceed 2n.
            PMA_REQUIRE(static_cast<uint64_t>(k) <= bucket_limit, PMA_ERR_LIMIT,
                        "geodesic: bucket sweep did not terminate");
        }
        epoch0 += static_cast<uint32_t>(k) + 1;
        ctx->count("geo.buckets", k);
        const unsigned walls_bits = static_cast<unsigned>(h[3]);
        const unsigned long long settled = h[4];
        const int reached = __builtin_popcount(walls_bits);
        {  // SPC.cpp:143-164: one row per cavity, however many there are
            pma_cavity o;
            std::memset(&o, 0, sizeof(o));
            o.id = cavity_id;
            o.seed_x = start[0];
            o.seed_y = start[1];
            o.seed_z = start[2];
            o.reached_walls = reached;
            o.reaches_all_walls = reached == walls_total ? 1 : 0;
            o.void_count = settled;
            const int dx = start[0] - c[0], dy = start[1] - c[1], dz = start[2] - c[2];
            o.distance_to_center = static_cast<float>(std::sqrt(static_cast<double>(dx * dx + dy * dy + dz * dz)));
            rows.push_back(o);
        }
        if (reached == walls_total) break;
    }
    return rows;
}

template std::vector<pma_cavity> geodesic<float>(pma_ctx*, const uint8_t*, pma_dims, pma_stencil, float*,
                                                 uint32_t*);
template std::vector<pma_cavity> geodesic<double>(pma_ctx*, const uint8_t*, pma_dims, pma_stencil, double*,
                                                  uint32_t*);

}  // namespace pma
