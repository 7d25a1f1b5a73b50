// Watershed pore and throat labelling (WatershedComputer.cpp:30-219), bit-exact.
//
// The reference floods from all seeds with one FIFO queue per depth (containing radius
// squared), deepest first. A popped node of pore P visits its stencil neighbours in loop
// order; a void neighbour w with crad(w) <= depth is "touched": the first touch claims w
// for P and queues it at depth crad(w); later touches by other pores only extend w's
// shared type ([second, first, third, ...], BasePoreAndThroatComputer.cpp:37-110) and do
// not queue it. Queued nodes keep propagating their claimer's pore.
//
// Parallel replay. Within one depth the FIFO runs generation by generation: generation 0 is
// the queue content when the depth starts (seeds in pore-id order, then nodes queued while
// deeper levels ran, in queue order); generation k+1 is what generation k queues at the same
// depth, in push order. Every touch gets the time (generation, node position * 27 +
// neighbour index), which orders touches exactly as the sequential loop does. Per generation:
//   claim    - the smallest-time touch of each unclaimed voxel wins (atomicMin on time);
//   resolve  - the winner records the claim; a voxel of the same depth joins the next
//              generation, a shallower one is appended, time-stamped, to its depth's bucket,
//              which is sorted by time when that depth starts; in the same pass, touches by
//              pores other than the voxel's owner record, per voxel and pore, their first
//              touch time (extensions).
// Frontier sizes stay on the device; the next generation is compacted in event order (see
// ws_generations; ws_small runs the small generations).
//
// Voxel state: one 64-bit word per voxel holds the claim state, which is the untouched mark,
// the smallest touch of the running generation (kTouched | event), or the claimer (pore
// index + 1). Claimed < touched < untouched numerically, so the claim phase's atomicMin keeps
// the smallest touch and never undoes a claim; a touched voxel is always claimed by the
// generation's resolve phase, so no touch outlives its generation. When the containing radii
// fit 16 bits (radius below 256 voxels) they ride in the word's low bits: a touch then costs one
// random load, and its atomic hits the same sector.
//
// Shared types: a voxel's key is its claimer plus its extending pores in time order; every
// prefix of length >= 2 was created at the time of its last extension. All prefixes are
// hashed, grouped with radix sorts and ranked by creation time on the device, which
// reproduces the reference's id sequence (UINT32_MAX - 1, - 2, ...) exactly, including
// types whose volume later dropped to zero. A voxel's extending pores are kept in a chain of
// fixed-size records, so a key may hold as many pores as the stencil lets touch one voxel
// (the reference keys types by an unbounded pore-id vector,
// BasePoreAndThroatComputer.cpp:112-133).
#include <cooperative_groups.h>
#include <thrust/iterator/counting_iterator.h>

#include <algorithm>
#include <cstring>
#include <memory>
#include <mutex>
#include <vector>

#include "devutil.cuh"
#include "type_rows.cuh"

namespace pma {
namespace {

constexpr uint32_t kNone = 0xFFFFFFFFu;
constexpr int kSlots = 6;         // extending pores per record; a voxel chains more records
constexpr int kMaxExt = 26;       // extending pores of one voxel at most (26 neighbours touch it)
constexpr int kMaxHops = (kMaxExt + kSlots - 1) / kSlots;  // records in one voxel's chain
constexpr int kKeyMax = kMaxExt + 1;  // longest key: the claimer and every extending pore
constexpr int kGensPerLaunch = 64;  // generations per cooperative launch (host checks between)
constexpr unsigned long long kMaxGen = 1ull << 23;              // generations per call
constexpr unsigned long long kSeqMask = (1ull << 40) - 1;       // touch time within a generation
constexpr unsigned long long kUntouched = (1ull << 48) - 1;     // claim states (48-bit field)
constexpr unsigned long long kTouched = 1ull << 46;
constexpr uint32_t kRecBusy = 0xFFFFFFFFu;  // ext[w] while its record is being allocated

struct WsState {
    Grid g;
    int d3q7;
    const uint32_t* crad;
    unsigned long long* state;    // per voxel: claim state, << 16 | radius when packed
    int packed;                   // 1: radii below 2^16 are held in the state words
    uint32_t* ext;                // shared-voxel record + 1, 0 = none
    uint32_t* ext_pore;           // [records][kSlots]
    unsigned long long* ext_time;
    uint32_t* ext_next;           // [records]: the voxel's next record + 1, 0 = none
    unsigned int* ext_count;
    uint32_t ext_cap;
    ulonglong2* log;              // extending touches not recorded yet: (time, pore << 32 | voxel);
                                  // ~0 in entries that were reserved and not used
    unsigned long long* log_n;    // entries reserved (may pass log_cap)
    uint32_t log_cap;
    unsigned int* pbound;         // per pore
    unsigned int* err;
    int spin_limit;               // polls of one wait on another block before giving up
    unsigned long long* gen_hist; // NULL, or per log2 of the frontier size: [c] generations,
                                  // [64 + c] ns in claim phases, [128 + c] ns in resolve phases
    int time_shift;               // bucket entry time = (generation << time_shift) | event
    uint32_t* touched;            // a bit per event: its claim phase touched an unclaimed voxel
    uint32_t* won;                // a bit per event: it gives a node of the next generation
    unsigned long long* bpos;        // per depth: where its bucket's next entry goes
    unsigned long long* ent_time;
    unsigned long long* ent_val;
};

__host__ __device__ __forceinline__ unsigned long long ws_word(int packed, unsigned long long st, uint32_t r) {
    return packed ? (st << 16) | r : st;
}

// Claim state of a state word: the claimer (pore index + 1) or 0.
__device__ __forceinline__ uint32_t ws_claimer(int packed, unsigned long long word) {
    const unsigned long long st = packed ? word >> 16 : word;
    return st < kTouched ? static_cast<uint32_t>(st) : 0u;
}

__global__ void ws_init(size_t n, const uint32_t* __restrict__ crad, int packed,
                        unsigned long long* __restrict__ state, uint32_t* __restrict__ ext) {
    PMA_GRID_STRIDE(v, n) {
        state[v] = ws_word(packed, kUntouched, packed ? crad[v] : 0u);
        ext[v] = 0;
    }
}

__global__ void ws_seed(const uint32_t* __restrict__ seed_voxel, size_t np, const uint32_t* __restrict__ crad,
                        int packed, unsigned long long* __restrict__ state) {
    PMA_GRID_STRIDE(k, np) {
        const uint32_t v = seed_voxel[k];
        state[v] = ws_word(packed, k + 1, packed ? crad[v] : 0u);
    }
}

__global__ void ws_seed_entries(const unsigned long long* __restrict__ a, size_t np,
                                unsigned long long* __restrict__ ent_time,
                                unsigned long long* __restrict__ ent_val) {
    PMA_GRID_STRIDE(k, np) {
        ent_time[a[k]] = a[np + k];
        ent_val[a[k]] = a[2 * np + k];
    }
}

// A frontier node: its voxel and its pore index, with kFace set when the voxel lies on a face of
// the volume (the other nodes' neighbours are all inside: no coordinates to work out).
constexpr uint32_t kFace = 0x80000000u;

__device__ __forceinline__ uint32_t ws_node(const Grid& g, uint32_t v, uint32_t pore) {
    int x, y, z;
    g.coords(v, x, y, z);
    return g.on_face(x, y, z) ? pore | kFace : pore;
}

// Voxel count per containing radius. Few distinct radii take most voxels, so counts gather
// in a shared-memory copy of the bins first when they fit (nb <= kHistShared).
constexpr uint32_t kHistShared = 8192;

__global__ void ws_histograms(const uint32_t* __restrict__ crad, size_t n, uint32_t nb,
                              unsigned int* __restrict__ hist) {
    __shared__ unsigned int local[kHistShared];
    const bool shared = nb <= kHistShared;
    if (shared)
        for (uint32_t i = threadIdx.x; i < nb; i += blockDim.x) local[i] = 0;
    __syncthreads();
    PMA_GRID_STRIDE(v, n) {
        const uint32_t r = crad[v];
        if (!r) continue;
        if (shared) atomicAdd(&local[r], 1u);
        else atomicAdd(&hist[r], 1u);
    }
    __syncthreads();
    if (shared)
        for (uint32_t i = threadIdx.x; i < nb; i += blockDim.x)
            if (local[i]) atomicAdd(&hist[i], local[i]);
}

// The record a link (ext[w] or a record's next field) points to, allocated by the one touch
// that moves the link from 0 to kRecBusy; touches that meet kRecBusy wait (a few
// instructions) for the record number. Returns 0 when the records ran out (err bit 1: the
// flood is redone with more) or the wait gave up (err bit 8).
__device__ __forceinline__ uint32_t ws_follow(uint32_t* link, const WsState& s) {
    uint32_t rec = *reinterpret_cast<volatile uint32_t*>(link);
    if (rec == 0) {
        rec = atomicCAS(link, 0u, kRecBusy);
        if (rec == 0) {
            // the warp's allocating lanes take their record numbers with one atomic (a single
            // counter for every new shared voxel of the flood would serialise them)
            const unsigned peers = __activemask();
            const int leader = __ffs(peers) - 1;
            const unsigned lane = threadIdx.x & 31;
            unsigned first = 0;
            if (static_cast<int>(lane) == leader) first = atomicAdd(s.ext_count, static_cast<unsigned>(__popc(peers)));
            first = __shfl_sync(peers, first, leader);
            const uint32_t fresh = first + __popc(peers & ((1u << lane) - 1u)) + 1;
            if (fresh > s.ext_cap) {  // out of records: flag a redo with more
                atomicExch(link, 0u);
                atomicOr(s.err, 1u);
                return 0;
            }
            atomicExch(link, fresh);
            return fresh;
        }
    }
    for (int spins = 0; rec == kRecBusy; ++spins) {
        if (spins > s.spin_limit) {
            atomicOr(s.err, 8u);
            return 0;
        }
        rec = atomicAdd(link, 0u);
    }
    if (rec == 0) atomicOr(s.err, 1u);  // the allocating touch ran out of records
    return rec;
}

// A touch that waits for a record number that nothing writes: the wait runs out after spin_limit polls
// and sets bit 8, the path of a stalled allocation.
__global__ void ws_wait_selftest(WsState s, uint32_t* link) {
    if (threadIdx.x != 0) return;
    *reinterpret_cast<volatile uint32_t*>(link) = kRecBusy;
    ws_follow(link, s);
}

// Records that `pore` touched shared voxel w at time t (its first touch per pore is kept).
// Out of line: it is the rare path of the touch kernel. Slots fill in order along the
// voxel's record chain, so two touches by one pore meet at the same slot.
__device__ __noinline__ void ws_extend(const WsState& s, size_t w, uint32_t pore, unsigned long long t) {
    uint32_t* link = s.ext + w;
    uint32_t rec = 0;
#pragma unroll 1
    for (int hop = 0; hop < kMaxHops; ++hop) {
        rec = ws_follow(link, s);
        if (!rec) break;
#pragma unroll 1
        for (int k = 0; k < kSlots; ++k) {
            const size_t slot = static_cast<size_t>(rec - 1) * kSlots + k;
            const uint32_t cur = atomicCAS(&s.ext_pore[slot], kNone, pore);
            if (cur == kNone || cur == pore) {
                atomicMin(&s.ext_time[slot], t);
                return;
            }
        }
        link = s.ext_next + (rec - 1);
    }
    if (rec) atomicOr(s.err, 2u);  // more extending pores than neighbours: cannot happen
}

// The flood itself only notes extending touches in a log, and ws_record_extensions records them
// later, one thread per entry: a record takes up to six dependent atomics, which would lengthen
// every generation by their latency (a touch of the flood waits for one), and claims never
// depend on extensions. A touch that finds the log full records itself in line. (640 x 600 x 672
// spinodal: generations of 2^13 nodes 23.8 -> 17 us, of 2^16 87 -> 70; stage 361 -> 315 ms.)
// Out of line, like ws_extend: the generation loops run once through a long way of code per
// generation, and inlined copies of the rare paths cost them instruction cache misses.
__device__ __noinline__ void ws_note(const WsState& s, uint32_t w, uint32_t pore, unsigned long long t) {
    const unsigned peers = __activemask();
    const int leader = __ffs(peers) - 1;
    const unsigned lane = threadIdx.x & 31;
    unsigned long long first = 0;
    if (static_cast<int>(lane) == leader) first = atomicAdd(s.log_n, static_cast<unsigned long long>(__popc(peers)));
    first = __shfl_sync(peers, first, leader);
    const unsigned long long pos = first + __popc(peers & ((1u << lane) - 1u));
    if (pos < s.log_cap) s.log[pos] = make_ulonglong2(t, (static_cast<unsigned long long>(pore) << 32) | w);
    else ws_extend(s, w, pore, t);
}

__global__ void ws_record_extensions(WsState s, uint32_t begin, uint32_t end) {
    PMA_GRID_STRIDE(k, end - begin) {
        const ulonglong2 e = s.log[begin + k];
        if (e.y != ~0ull) ws_extend(s, static_cast<uint32_t>(e.y), static_cast<uint32_t>(e.y >> 32), e.x);
    }
}

// Appends a claim (entry time, pore << 32 | voxel of radius r, below the running depth) to its
// depth's bucket. Lanes appending to the same depth take their slots with one atomic: a generation's claims of
// shallower voxels mostly go to a few depths, and one counter per depth would serialise them.
__device__ __forceinline__ void ws_append_entry(const WsState& s, unsigned lanes, uint32_t r, unsigned long long time,
                                                unsigned long long val) {
    const unsigned lane = threadIdx.x & 31;
    const unsigned peers = __match_any_sync(lanes, r);
    const int leader = __ffs(peers) - 1;
    unsigned long long first = 0;
    if (static_cast<int>(lane) == leader) first = atomicAdd(&s.bpos[r], static_cast<unsigned long long>(__popc(peers)));
    first = __shfl_sync(peers, first, leader);
    const unsigned long long at = first + __popc(peers & ((1u << lane) - 1u));
    s.ent_time[at] = time;
    s.ent_val[at] = val;
}

__device__ __forceinline__ unsigned long long ws_clock() {  // ns
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Touch events of a generation's nodes, one per node i and stencil position j: seq = i * 27 + j. The
// claim phase lets the smallest touch time of each unclaimed voxel win (atomicMin on its state
// word) and sets the event's bit in `touched`. A touch of a voxel claimed in an earlier
// generation is final there already: it is an extension when the toucher is not the owner (claims
// never change, and extensions keep each pore's smallest time, so the order of recording does
// not matter). The resolve phase takes the touched events only: the winner records its claim, every
// other touch by a pore other than the winner's is an extension.
//
// A warp takes strips of events, kStrip a lane (one in generations that the grid covers at once): the
// strip's nodes and touch bits are read one strip ahead, a lane's state words are loaded
// together, and extensions and claims of shallower voxels gather in lists of the warp, which go to the log and
// the buckets about a hundred at a time. No block barrier comes between strips. All generations of a launch run in
// one kernel, so data written by other blocks earlier in the launch is read with __ldcg (L2, not a possibly
// stale L1 line); only the radii, which never change, go through the read-only path.
// What bounds a generation: below 2^14 nodes the three grid barriers (about 2 us each with 608 blocks)
// and the chain of dependent loads between them, above it instructions and the latency of
// the scattered state words (40 % of the issue slots, L2 at 11 %). Generations of 2^13 / 2^17 / 2^20 nodes, us:
// one event a thread with a node load, a state load and an answered atomic one after the other
// 17 / 147 / 780, now 18 / 94 / 580; stage of a 640 x 600 x 672 spinodal 315 -> 288 ms, of a 512^3
// field 146 -> 123 ms. (Chunks of 1024 events a block with a block barrier each: the same within 2 %.)
constexpr int kGenThreads = 256;
constexpr int kGenWarps = kGenThreads / 32;
constexpr int kStrip = 2;             // events a lane of a strip
constexpr unsigned kGenList = 128;    // entries of a warp's lists

struct WsGenShared {
    uint32_t delta[27];                 // index step of a stencil position
    unsigned int count[kGenWarps], base[kGenWarps];
    ulonglong2 ext[kGenWarps][kGenList];                                            // as in the log
    unsigned long long up_time[kGenWarps][kGenList], up_val[kGenWarps][kGenList];  // as in a bucket
    uint32_t up_r[kGenWarps][kGenList];
};

struct WsLists {  // lengths of the warp's lists
    unsigned ext, up;
};

__device__ __noinline__ void ws_flush_ext(const WsState& s, WsGenShared& sh, unsigned n) {
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned long long base = 0;
    if (lane == 0) base = atomicAdd(s.log_n, static_cast<unsigned long long>(n));
    base = __shfl_sync(0xFFFFFFFFu, base, 0);
    __syncwarp();
    for (unsigned i = lane; i < n; i += 32) {
        const ulonglong2 e = sh.ext[warp][i];
        if (base + i < s.log_cap) s.log[base + i] = e;
        else ws_extend(s, static_cast<uint32_t>(e.y), static_cast<uint32_t>(e.y >> 32), e.x);  // log full
    }
    __syncwarp();
}

__device__ __noinline__ void ws_flush_up(const WsState& s, WsGenShared& sh, unsigned n) {
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncwarp();
    for (unsigned i0 = 0; i0 < n; i0 += 32) {
        const unsigned lanes = n - i0 >= 32 ? 0xFFFFFFFFu : (1u << (n - i0)) - 1u;
        if (lane < n - i0) ws_append_entry(s, lanes, sh.up_r[warp][i0 + lane], sh.up_time[warp][i0 + lane], sh.up_val[warp][i0 + lane]);
    }
    __syncwarp();
}

// All 32 lanes call; ext = this lane has an extending touch.
__device__ __forceinline__ void ws_list_ext(const WsState& s, WsGenShared& sh, WsLists& l, bool ext, uint32_t w, uint32_t pore,
                                            unsigned long long t) {
    const unsigned m = __ballot_sync(0xFFFFFFFFu, ext);
    if (!m) return;
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (l.ext > kGenList - 32) {
        ws_flush_ext(s, sh, l.ext);
        l.ext = 0;
    }
    if (ext) sh.ext[warp][l.ext + __popc(m & ((1u << lane) - 1u))] = make_ulonglong2(t, (static_cast<unsigned long long>(pore) << 32) | w);
    l.ext += __popc(m);
}

__device__ __forceinline__ void ws_list_up(const WsState& s, WsGenShared& sh, WsLists& l, bool up, uint32_t w, uint32_t pore,
                                           uint32_t r, unsigned long long time) {
    const unsigned m = __ballot_sync(0xFFFFFFFFu, up);
    if (!m) return;
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (l.up > kGenList - 32) {
        ws_flush_up(s, sh, l.up);
        l.up = 0;
    }
    if (up) {
        const unsigned at = l.up + __popc(m & ((1u << lane) - 1u));
        sh.up_time[warp][at] = time;
        sh.up_val[warp][at] = (static_cast<unsigned long long>(pore) << 32) | w;
        sh.up_r[warp][at] = r;
    }
    l.up += __popc(m);
}

// A strip of PER * 32 events: its first event, that event's node and how many events of that node come before.
struct WsStrip {
    unsigned long long e0, first;
    uint32_t skip, n;  // n: events of the strip
};

template <int PER>
__device__ __forceinline__ WsStrip ws_strip(unsigned long long c, unsigned long long nev) {
    WsStrip k;
    k.e0 = c * (PER * 32);
    k.first = k.e0 / 27;
    k.skip = static_cast<uint32_t>(k.e0 - k.first * 27);
    k.n = static_cast<uint32_t>(min(nev - k.e0, static_cast<unsigned long long>(PER * 32)));
    return k;
}

// Lane i: the strip's i-th node (at most four with kStrip 2); lane k: the touch bits of the strip's k-th 32 events.
static_assert((26 + kStrip * 32 + 26) / 27 <= 32, "a lane per node of a strip");
struct WsAhead {
    uint32_t v, p, touched;
};

template <int PER>
__device__ __forceinline__ WsAhead ws_fetch(const WsState& s, const WsStrip& k, const uint32_t* gv, const uint32_t* gp, bool touched) {
    const unsigned lane = threadIdx.x & 31;
    WsAhead a{0, 0, 0};
    if (lane < (k.skip + k.n + 26) / 27) {
        a.v = __ldcg(gv + k.first + lane);
        a.p = __ldcg(gp + k.first + lane);
    }
    if (touched && lane < PER) a.touched = __ldcg(s.touched + (k.e0 >> 5) + lane);
    return a;
}

template <int PER>
__device__ __forceinline__ void ws_claim_strip(const WsState& s, WsGenShared& sh, WsLists& l, const WsStrip& ck, const WsAhead& a,
                                               uint32_t depth, unsigned long long gen) {
    const unsigned lane = threadIdx.x & 31;
    unsigned long long word[PER];
    uint32_t w[PER], pore[PER], rad[PER];
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        const uint32_t e = k * 32 + lane, i = (ck.skip + e) / 27;
        const int j = static_cast<int>(ck.skip + e - i * 27);
        const uint32_t v = __shfl_sync(0xFFFFFFFFu, a.v, i), node = __shfl_sync(0xFFFFFFFFu, a.p, i);
        bool live = e < ck.n && j != 13;
        int dx, dy, dz;
        if (s.d3q7) live = live && stencil_offset(j, 1, dx, dy, dz);
        pore[k] = node & ~kFace;
        w[k] = v + sh.delta[j];
        if (live && (node & kFace)) {
            int x, y, z;
            s.g.coords(v, x, y, z);
            stencil_offset(j, 0, dx, dy, dz);
            if (!s.g.inside(x + dx, y + dy, z + dz)) {  // WC.cpp:140-144
                s.pbound[pore[k]] = 1;
                live = false;
            }
        }
        word[k] = 0;  // radius 0
        rad[k] = 0;
        if (live) {
            word[k] = __ldcg(s.state + w[k]);
            if (!s.packed) rad[k] = __ldg(s.crad + w[k]);
        }
    }
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        const unsigned long long seq = ck.e0 + k * 32 + lane;
        const uint32_t r = s.packed ? static_cast<uint32_t>(word[k] & 0xFFFFu) : rad[k];
        const unsigned long long st = s.packed ? word[k] >> 16 : word[k];
        const bool in = r != 0 && r <= depth, open = in && st >= kTouched;  // WC.cpp:152-156
        if (open) atomicMin(&s.state[w[k]], ws_word(s.packed, kTouched | seq, r));
        const unsigned m = __ballot_sync(0xFFFFFFFFu, open);
        if (lane == 0) s.touched[(ck.e0 >> 5) + k] = m;
        ws_list_ext(s, sh, l, in && !open && st - 1 != pore[k], w[k], pore[k], (gen << 40) | seq);
    }
}

// Returns the strip's claims of this depth.
template <int PER>
__device__ __forceinline__ unsigned ws_resolve_strip(const WsState& s, WsGenShared& sh, WsLists& l, const WsStrip& ck, const WsAhead& a,
                                                     const uint32_t* gp, uint32_t depth, unsigned long long gen) {
    const unsigned lane = threadIdx.x & 31;
    unsigned count = 0;
    unsigned long long word[PER];
    uint32_t w[PER], pore[PER], rad[PER], owner[PER], hits = 0;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        const uint32_t e = k * 32 + lane, i = (ck.skip + e) / 27;
        hits |= (__shfl_sync(0xFFFFFFFFu, a.touched, k) >> lane & 1u) << k;
        pore[k] = __shfl_sync(0xFFFFFFFFu, a.p, i) & ~kFace;
        w[k] = __shfl_sync(0xFFFFFFFFu, a.v, i) + sh.delta[ck.skip + e - i * 27];
        word[k] = 0;
        rad[k] = 0;
        if ((hits >> k) & 1u) {
            word[k] = __ldcg(s.state + w[k]);
            if (!s.packed) rad[k] = __ldg(s.crad + w[k]);
        }
    }
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        const unsigned long long seq = ck.e0 + k * 32 + lane;
        const uint32_t r = s.packed ? static_cast<uint32_t>(word[k] & 0xFFFFu) : rad[k];
        const unsigned long long st = s.packed ? word[k] >> 16 : word[k];
        const bool hit = (hits >> k) & 1u, win = hit && st == (kTouched | seq);
        owner[k] = pore[k];
        if (win) s.state[w[k]] = ws_word(s.packed, pore[k] + 1, r);  // one 64-bit store: readers see either word
        else if (hit)  // the winner's pore: stored as the claimer already, or that of the winning touch's node
            owner[k] = st < kTouched ? static_cast<uint32_t>(st - 1) : __ldcg(gp + (st & kSeqMask) / 27) & ~kFace;
        const unsigned m = __ballot_sync(0xFFFFFFFFu, win && r == depth);
        if (lane == 0) s.won[(ck.e0 >> 5) + k] = m;
        count += __popc(m);
        ws_list_up(s, sh, l, win && r != depth, w[k], pore[k], r, (gen << s.time_shift) | seq);
    }
#pragma unroll
    for (int k = 0; k < PER; ++k) ws_list_ext(s, sh, l, owner[k] != pore[k], w[k], pore[k], (gen << 40) | (ck.e0 + k * 32 + lane));
    return count;
}

// One generation's phases, PER events a lane and strip.
template <int PER>
__device__ __forceinline__ void ws_claims(const WsState& s, WsGenShared& sh, WsLists& l, const uint32_t* gv, const uint32_t* gp,
                                          unsigned long long nev, uint32_t depth, unsigned long long gen) {
    const unsigned long long strips = (nev + PER * 32 - 1) / (PER * 32), step = static_cast<unsigned long long>(gridDim.x) * kGenWarps;
    // strips dealt to the blocks first, so that a generation of few strips spreads over the SMs
    unsigned long long c = (threadIdx.x >> 5) * static_cast<unsigned long long>(gridDim.x) + blockIdx.x;
    if (c >= strips) return;
    WsStrip next = ws_strip<PER>(c, nev);
    WsAhead ahead = ws_fetch<PER>(s, next, gv, gp, false);
    for (; c < strips; c += step) {
        const WsStrip ck = next;
        const WsAhead a = ahead;
        if (c + step < strips) {
            next = ws_strip<PER>(c + step, nev);
            ahead = ws_fetch<PER>(s, next, gv, gp, false);
        }
        ws_claim_strip<PER>(s, sh, l, ck, a, depth, gen);
    }
}

template <int PER>
__device__ __forceinline__ unsigned ws_resolves(const WsState& s, WsGenShared& sh, WsLists& l, const uint32_t* gv, const uint32_t* gp,
                                                unsigned long long c, unsigned long long c1, unsigned long long nev, uint32_t depth,
                                                unsigned long long gen) {
    if (c >= c1) return 0;
    unsigned count = 0;
    WsStrip next = ws_strip<PER>(c, nev);
    WsAhead ahead = ws_fetch<PER>(s, next, gv, gp, true);
    for (; c < c1; ++c) {
        const WsStrip ck = next;
        const WsAhead a = ahead;
        if (c + 1 < c1) {
            next = ws_strip<PER>(c + 1, nev);
            ahead = ws_fetch<PER>(s, next, gv, gp, true);
        }
        count += ws_resolve_strip<PER>(s, sh, l, ck, a, gp, depth, gen);
    }
    return count;
}

// The next frontier is written in event order: each warp resolves one contiguous range of strips and counts
// its claims of this depth, and behind a grid-wide barrier each block adds up the counts of the blocks before
// it. (A decoupled look-back in place of that barrier made the generations of 2^12 to 2^15 nodes 20 to 40 %
// slower.)
//
// Up to max_gens generations of one depth in a single cooperative launch, three grid-wide
// barriers per generation. ng[2] holds the two frontier sizes; the frontier starts on side
// `cur`. The launch ends early when the frontier has at most small_nodes nodes. out[0] =
// generations run, out[1] = the side holding the next frontier.
__global__ void __launch_bounds__(kGenThreads, 4) ws_generations(WsState s, uint32_t* gv0, uint32_t* gp0, uint32_t* gv1,
                                                             uint32_t* gp1, unsigned int* ng,
                                                             unsigned int* counts, uint32_t depth,
                                                             unsigned long long gen0, int max_gens, int cur,
                                                             unsigned small_nodes, unsigned long long* out) {
    namespace cg = cooperative_groups;
    cg::grid_group grid = cg::this_grid();
    __shared__ WsGenShared sh;
    const unsigned tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, lt = (1u << lane) - 1u;
    const bool first_thread = blockIdx.x == 0 && tid == 0;
    if (tid < 27) {
        int dx, dy, dz;
        stencil_offset(static_cast<int>(tid), 0, dx, dy, dz);
        sh.delta[tid] = (static_cast<uint32_t>(dz) * s.g.SX + dx) * s.g.SY + dy;  // modulo 2^32
    }
    WsLists lists{0, 0};
    __syncthreads();
    unsigned long long gen = gen0;
    int it = 0;
    for (; it < max_gens; ++it) {
        const unsigned long long nev = static_cast<unsigned long long>(__ldcg(ng + cur)) * 27;
        if (nev <= static_cast<unsigned long long>(small_nodes) * 27) break;  // ws_small goes on
        ++gen;
        const int hc = min(63, 63 - __clzll(nev / 27));
        unsigned long long t_start = 0;
        if (s.gen_hist && first_thread) {
            atomicAdd(&s.gen_hist[hc], 1ull);
            t_start = ws_clock();
        }
        const uint32_t* gv = cur ? gv1 : gv0;
        const uint32_t* gp = cur ? gp1 : gp0;
        uint32_t* nv = cur ? gv0 : gv1;
        uint32_t* np_ = cur ? gp0 : gp1;
        // one event a lane while the grid covers the generation in two rounds, else kStrip
        const bool one = nev <= 2ull * gridDim.x * kGenThreads;
        if (one) ws_claims<1>(s, sh, lists, gv, gp, nev, depth, gen);
        else ws_claims<kStrip>(s, sh, lists, gv, gp, nev, depth, gen);
        grid.sync();
        if (s.gen_hist && first_thread) {
            const unsigned long long t = ws_clock();
            atomicAdd(&s.gen_hist[64 + hc], t - t_start);
            t_start = t;
        }
        // warp w of block b resolves the strips [w0, w1)
        const unsigned strip = one ? 32 : 32 * kStrip;
        const unsigned long long strips = (nev + strip - 1) / strip, warps = static_cast<unsigned long long>(gridDim.x) * kGenWarps;
        const unsigned long long per = (strips + warps - 1) / warps;
        const unsigned long long w0 = min((static_cast<unsigned long long>(blockIdx.x) * kGenWarps + warp) * per, strips);
        const unsigned long long w1 = min(w0 + per, strips);
        unsigned count = one ? ws_resolves<1>(s, sh, lists, gv, gp, w0, w1, nev, depth, gen)
                             : ws_resolves<kStrip>(s, sh, lists, gv, gp, w0, w1, nev, depth, gen);
        if (lane == 0) sh.count[warp] = count;
        __syncthreads();
        unsigned before = 0, total = 0;  // the block's claims: of the warps before this one, of all
        for (int i = 0; i < kGenWarps; ++i) {
            if (i < static_cast<int>(warp)) before += sh.count[i];
            total += sh.count[i];
        }
        if (tid == 0) counts[blockIdx.x] = total;
        grid.sync();
        // the claims of the blocks before this one
        unsigned base = 0;
        for (unsigned b = tid; b < blockIdx.x; b += kGenThreads) base += __ldcg(counts + b);
        base = __reduce_add_sync(0xFFFFFFFFu, base);
        if (lane == 0) sh.base[warp] = base;
        __syncthreads();
        base = 0;
        for (int i = 0; i < kGenWarps; ++i) base += sh.base[i];
        if (blockIdx.x == gridDim.x - 1 && tid == 0) ng[cur ^ 1] = base + total;
        size_t pos = static_cast<size_t>(base) + before;
        if (count) {
            const unsigned long long b0 = w0 * (strip / 32), b1 = w1 * (strip / 32);  // the range's words of won bits
            for (unsigned long long b = b0; b < b1; b += 32) {
                const uint32_t bits = b + lane < b1 ? __ldcg(s.won + b + lane) : 0u;
                uint32_t incl = __popc(bits);
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, incl, o);
                    if (lane >= static_cast<unsigned>(o)) incl += t;
                }
                for (unsigned some = __ballot_sync(0xFFFFFFFFu, bits); some; some &= some - 1) {
                    const int q = __ffs(some) - 1;
                    const uint32_t m = __shfl_sync(0xFFFFFFFFu, bits, q), at = __shfl_sync(0xFFFFFFFFu, incl, q) - __popc(m);
                    if ((m >> lane) & 1u) {
                        const unsigned long long e = (b + q) * 32 + lane, i = e / 27;
                        const uint32_t v = __ldcg(gv + i) + sh.delta[e - i * 27];
                        nv[pos + at + __popc(m & lt)] = v;
                        np_[pos + at + __popc(m & lt)] = ws_node(s.g, v, __ldcg(gp + i) & ~kFace);
                    }
                }
                pos += __shfl_sync(0xFFFFFFFFu, incl, 31);
            }
        }
        grid.sync();
        if (s.gen_hist && first_thread) atomicAdd(&s.gen_hist[128 + hc], ws_clock() - t_start);
        cur ^= 1;
    }
    if (lists.ext) ws_flush_ext(s, sh, lists.ext);
    if (lists.up) ws_flush_up(s, sh, lists.up);
    if (first_thread) {
        out[0] = static_cast<unsigned long long>(it);
        out[1] = static_cast<unsigned long long>(cur);
    }
}

// --- small generations --------------------------------------------------------------------
//
// Most generations are small (a few to a few thousand nodes) and their time is latency: in
// ws_generations a generation of 2^6 to 2^10 nodes takes 10 to 14 us (three barriers over the whole
// grid, one launch and one host round trip per depth). ws_small runs them in one
// thread-block cluster, and goes from depth to depth by itself: it sorts a depth's bucket in
// shared memory, runs its generations and takes the next depth, until a bucket or a frontier is
// too large for it (the host then sorts that bucket and runs ws_generations until the frontier
// is small again). Generations of at most kSoloNodes nodes run in the cluster's first block
// alone, with the frontier in shared memory and block barriers; larger ones split their nodes
// over the blocks, one contiguous run each, with three cluster barriers.
// What bounds a generation: latency (a block barrier 50 cycles, a cluster barrier 400 and with it
// the wait for the atomics in flight, an L2 load 300 to 700), and one sector a clock and SM for the
// scattered state words; hence 16 blocks, and 64 nodes as the most for one block alone. From about
// 2000 nodes the whole grid is faster (2^11 nodes: 20 us here, 12 there). At 2^10 it is too, 11.3 against 14.5, but each
// change between the two costs a launch and a host round trip: with 1024 as the limit a 640 x 600 x 672
// spinodal took 277 ms, not 279, a 128^3 union 42.2, not 40.6.
// Whole stage, before and after (ms): 40 x 48 x 44 union 15.6 -> 5.2, 128^3 union 48.5 -> 30.7,
// 300 x 341 x 277 spinodal 135 -> 119.
constexpr int kSmallThreads = 512;
constexpr int kSmallWarps = kSmallThreads / 32;
constexpr int kSmallCluster = 16;       // blocks
constexpr int kSmallSort = 8192;        // bucket entries sorted in shared memory
constexpr unsigned kSoloNodes = 64;
constexpr unsigned kSmallNodes = 2048;
constexpr int kStage = kSmallNodes / kSmallCluster;  // nodes a block holds in shared memory
static_assert(kSoloNodes <= kStage && kStage <= kSmallThreads, "a block's nodes are staged whole, one a thread");
static_assert((kStage * 27 + kSmallThreads - 1) / kSmallThreads + 1 <= 32, "a thread's touch flags are one 32-bit word");
constexpr unsigned kSmallUps = 1024;    // claims of shallower voxels a block keeps until they go to their buckets
constexpr unsigned kLogSlab = 512;      // extension log entries a block of ws_small takes at a time

enum WsMode { kWsDone = 0, kWsRun = 1, kWsSort = 2, kWsBig = 3, kWsLimit = 4, kWsGrow = 5 };

struct WsCtl {  // where the flood stands
    unsigned long long gen;
    uint32_t di;   // index into the depth list
    uint32_t n;    // frontier nodes (kWsSort: entries of the bucket)
    uint32_t cur;  // side of the frontier
    uint32_t mode;
};

struct WsSmallArgs {
    uint32_t *gv0, *gp0, *gv1, *gp1;
    const uint32_t* depths;  // depths that can hold entries, deepest first
    uint32_t ndepths;
    const unsigned long long* boff;  // per depth: the first entry of its bucket
    unsigned long long max_gen;
};

struct WsSmallShared {
    uint32_t v[2][kStage], p[2][kStage];  // staged nodes
    unsigned long long up_time[kSmallUps], up_val[kSmallUps];  // claims of shallower voxels, as in a bucket
    uint32_t up_r[kSmallUps];                                  // their radii
    uint32_t ups;
    uint32_t won[kStage];    // per node: stencil positions of its same-depth claims
    uint32_t sum[kSmallWarps];
    uint32_t total[kSmallCluster];
    uint32_t delta[27];      // index step of a stencil position
    uint32_t log_base, log_used;  // the block's slab of the extension log
    uint32_t found_di, found_n;   // the next depth with entries and how many
    WsCtl ctl;
};

// Notes the extending touches of a warp (all 32 lanes call; ext = this lane has one) in the
// block's slab: a shared-memory counter instead of a round trip to the log's.
__device__ __forceinline__ void ws_small_note(const WsState& s, WsSmallShared& sh, bool ext, uint32_t w, uint32_t pore,
                                              unsigned long long t) {
    const unsigned m = __ballot_sync(0xFFFFFFFFu, ext);
    if (!m) return;
    const unsigned lane = threadIdx.x & 31;
    uint32_t first = 0;
    if (lane == 0) first = atomicAdd(&sh.log_used, static_cast<uint32_t>(__popc(m)));
    first = __shfl_sync(0xFFFFFFFFu, first, 0);
    if (!ext) return;
    const uint32_t pos = first + __popc(m & ((1u << lane) - 1u));
    if (pos < kLogSlab && sh.log_base + pos < s.log_cap)
        s.log[sh.log_base + pos] = make_ulonglong2(t, (static_cast<unsigned long long>(pore) << 32) | w);
    else ws_note(s, w, pore, t);  // slab full
}

// A new slab for the block when the present one is more than half used (or there is none).
__device__ __forceinline__ void ws_small_slab(const WsState& s, WsSmallShared& sh) {
    if (threadIdx.x == 0 && sh.log_used > kLogSlab / 2) {
        sh.log_base = static_cast<uint32_t>(min(atomicAdd(s.log_n, static_cast<unsigned long long>(kLogSlab)), 0x7FFFFFFFull));
        sh.log_used = 0;
    }
}

// Moves the block's list of claims of shallower voxels to their depths' buckets. Keeping them here
// over many generations takes the wait for the bucket's counter out of each of them.
__device__ __noinline__ void ws_small_flush(const WsState& s, WsSmallShared& sh) {
    __syncthreads();
    const uint32_t k = min(sh.ups, kSmallUps);
    for (uint32_t i = threadIdx.x; i < k; i += kSmallThreads) {
        const unsigned long long at = atomicAdd(&s.bpos[sh.up_r[i]], 1ull);
        s.ent_time[at] = sh.up_time[i];
        s.ent_val[at] = sh.up_val[i];
    }
    __syncthreads();
    if (threadIdx.x == 0) sh.ups = 0;
    __syncthreads();
}

// One generation of n nodes; returns the next frontier's size. cl: all blocks of the cluster, each
// a contiguous run of the nodes, staged from gv/gp; else one block, the frontier in sh.v[side].
// A thread takes an event at a time: a warp's lanes then meet three neighbours of a row in one
// 32-byte sector (an SM serves about one sector a clock, which bounds a block's generation).
__device__ __noinline__ uint32_t ws_small_generation(const WsState& s, WsSmallShared& sh, bool cl, const uint32_t* gv,
                                                     const uint32_t* gp, uint32_t* nv, uint32_t* np_, int side, uint32_t n,
                                                     uint32_t depth, unsigned long long gen) {
    namespace cg = cooperative_groups;
    const unsigned tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    uint32_t first = 0, m = n;  // the block's nodes
    if (cl) {
        const uint32_t per = (n + kSmallCluster - 1) / kSmallCluster;
        first = min(cg::this_cluster().block_rank() * per, n);
        m = min(per, n - first);
        side = 0;
        if (tid < m) {
            sh.v[0][tid] = __ldcg(gv + first + tid);
            sh.p[0][tid] = __ldcg(gp + first + tid);
        }
    }
    if (tid < m) sh.won[tid] = 0;
    __syncthreads();
    const uint32_t nev = m * 27, seq0 = first * 27;
    // claims, as ws_claim_strip; bit k of touched: this thread's k-th event touched an unclaimed
    // voxel. Two events a turn, their loads in flight together.
    uint32_t touched = 0;
#pragma unroll 1
    for (unsigned k = 0; k * kSmallThreads + warp * 32 < nev; k += 2) {
        unsigned long long word[2];
        uint32_t rad[2], w[2], pore[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const uint32_t e = (k + u) * kSmallThreads + tid, i = e < nev ? e / 27 : 0;
            const int j = static_cast<int>(e - i * 27);
            int dx, dy, dz;
            word[u] = 0;  // radius 0
            rad[u] = 0;
            w[u] = pore[u] = 0;
            if (e >= nev || !stencil_offset(j, s.d3q7, dx, dy, dz)) continue;
            const uint32_t v = sh.v[side][i], node = sh.p[side][i];
            pore[u] = node & ~kFace;
            w[u] = v + sh.delta[j];
            if (node & kFace) {
                int x, y, z;
                s.g.coords(v, x, y, z);
                if (!s.g.inside(x + dx, y + dy, z + dz)) {  // WC.cpp:140-144
                    s.pbound[pore[u]] = 1;
                    continue;
                }
            }
            word[u] = __ldcg(s.state + w[u]);
            if (!s.packed) rad[u] = __ldg(s.crad + w[u]);
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const uint32_t seq = seq0 + (k + u) * kSmallThreads + tid;
            const uint32_t r = s.packed ? static_cast<uint32_t>(word[u] & 0xFFFFu) : rad[u];
            const unsigned long long st = s.packed ? word[u] >> 16 : word[u];
            const bool in = r != 0 && r <= depth, ext = in && st < kTouched && st - 1 != pore[u];  // WC.cpp:152-156
            if (in && st >= kTouched) {
                atomicMin(&s.state[w[u]], ws_word(s.packed, kTouched | seq, r));
                touched |= 1u << (k + u);
            }
            if (__any_sync(0xFFFFFFFFu, ext)) ws_small_note(s, sh, ext, w[u], pore[u], (gen << 40) | seq);
        }
    }
    if (cl) cg::this_cluster().sync();
    else __syncthreads();
    // resolve the touches, as ws_resolve_strip; a claim of the same depth sets its stencil
    // position's bit in its node's word
#pragma unroll 1
    for (unsigned k = 0; k * kSmallThreads + warp * 32 < nev; k += 2) {
        if (!__any_sync(0xFFFFFFFFu, (touched >> k) & 3u)) continue;
        unsigned long long word[2];
        uint32_t rad[2], w[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            word[u] = 0;
            rad[u] = w[u] = 0;
            if (!((touched >> (k + u)) & 1u)) continue;
            const uint32_t e = (k + u) * kSmallThreads + tid, i = e / 27;
            w[u] = sh.v[side][i] + sh.delta[e - i * 27];
            word[u] = __ldcg(s.state + w[u]);
            if (!s.packed) rad[u] = __ldg(s.crad + w[u]);
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const uint32_t e = (k + u) * kSmallThreads + tid, i = e / 27, seq = seq0 + e;
            bool ext = false;
            uint32_t pore = 0;
            if ((touched >> (k + u)) & 1u) {
                pore = sh.p[side][i] & ~kFace;
                const uint32_t r = s.packed ? static_cast<uint32_t>(word[u] & 0xFFFFu) : rad[u];
                const unsigned long long st = s.packed ? word[u] >> 16 : word[u];
                if (st == (kTouched | seq)) {
                    s.state[w[u]] = ws_word(s.packed, pore + 1, r);
                    if (r == depth) {
                        atomicOr(&sh.won[i], 1u << (e - i * 27));
                    } else {  // to its depth's bucket, by way of the block's list
                        const uint32_t at = atomicAdd(&sh.ups, 1u);
                        if (at < kSmallUps) {
                            sh.up_time[at] = (gen << s.time_shift) | seq;
                            sh.up_val[at] = (static_cast<unsigned long long>(pore) << 32) | w[u];
                            sh.up_r[at] = r;
                        } else {
                            ws_append_entry(s, __activemask(), r, (gen << s.time_shift) | seq,
                                            (static_cast<unsigned long long>(pore) << 32) | w[u]);
                        }
                    }
                } else if (st < kTouched) {
                    ext = static_cast<uint32_t>(st - 1) != pore;
                } else {
                    const uint32_t node = static_cast<uint32_t>((st & kSeqMask) / 27);
                    ext = ((node - first < m ? sh.p[side][node - first] : __ldcg(gp + node)) & ~kFace) != pore;
                }
            }
            if (__any_sync(0xFFFFFFFFu, ext)) ws_small_note(s, sh, ext, w[u], pore, (gen << 40) | seq);
        }
    }
    __syncthreads();
    ws_small_slab(s, sh);
    // offsets in event order: nodes, then stencil positions
    uint32_t won = tid < m ? sh.won[tid] : 0u;
    uint32_t incl = __popc(won);
    const uint32_t mine = incl;
    if (warp * 32 < m) {
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= static_cast<unsigned>(o)) incl += t;
        }
    }
    if (lane == 31) sh.sum[warp] = incl;
    __syncthreads();
    const uint32_t sums = lane < kSmallWarps ? sh.sum[lane] : 0u;
    uint32_t next = __reduce_add_sync(0xFFFFFFFFu, sums);
    uint32_t pos = __reduce_add_sync(0xFFFFFFFFu, lane < warp ? sums : 0u) + incl - mine;
    if (cl) {
        cg::cluster_group cluster = cg::this_cluster();
        const unsigned rank = cluster.block_rank();
        if (tid < kSmallCluster) cluster.map_shared_rank(sh.total, tid)[rank] = next;
        cluster.sync();
        next = 0;
#pragma unroll 1
        for (unsigned b = 0; b < kSmallCluster; ++b) {
            if (b < rank) pos += sh.total[b];
            next += sh.total[b];
        }
    }
    if (won) {
        const uint32_t v = sh.v[side][tid], pore = sh.p[side][tid] & ~kFace;
        for (; won; won &= won - 1, ++pos) {
            const uint32_t w = v + sh.delta[__ffs(won) - 1], node = ws_node(s.g, w, pore);
            nv[pos] = w;
            np_[pos] = node;
            if (!cl && pos < kSoloNodes) {
                sh.v[side ^ 1][pos] = w;
                sh.p[side ^ 1][pos] = node;
            }
        }
    }
    if (sh.ups > kSmallUps / 2) ws_small_flush(s, sh);  // the same for the whole block: nobody adds now
    if (cl) cg::this_cluster().sync();
    else __syncthreads();
    return next;
}

// Shared memory of a bucket's sort, in the dynamic part (the cluster's first block uses it).
constexpr int kSortDigit = 6;  // bits of a radix pass: 64 digits x 32 warps of counters
struct WsSortShared {
    unsigned long long time[2][kSmallSort];
    uint16_t at[2][kSmallSort];
    uint16_t rank[kSmallSort];  // within the entry's warp and digit
    uint32_t count[(1 << kSortDigit) * (kSmallWarps + 1)];  // [digit][warp], a row of one more: fewer bank conflicts
    unsigned long long vary[kSmallWarps];
    uint32_t sum[kSmallWarps];
};
static_assert((1 << kSortDigit) * kSmallWarps == 2 * kSmallThreads, "two counters a thread");
constexpr uint32_t kRankSort = kSmallThreads / 4;  // buckets this small are sorted by counting

// Sorts the n entries of a depth's bucket by time (times are distinct) and writes the depth's
// first generation, in shared memory too. Up to kRankSort entries: each finds its rank by
// comparing itself with every other, four threads an entry. Larger: stable radix passes over the
// bits in which the times differ, each warp ranking its own run of the entries by ballots. (A bitonic sort,
// with a block barrier per step, took 5.4 us for 100 entries and 20 us for 1300.)
__device__ __noinline__ void ws_small_bucket(const WsState& s, WsSmallShared& sh, WsSortShared& so, unsigned long long off, uint32_t n,
                                uint32_t* gv, uint32_t* gp) {
    const unsigned tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, lt = (1u << lane) - 1u;
    auto put = [&](uint32_t pos, uint32_t at) {  // entry `at` becomes node `pos`
        const unsigned long long val = __ldcg(s.ent_val + off + at);
        const uint32_t v = static_cast<uint32_t>(val), node = ws_node(s.g, v, static_cast<uint32_t>(val >> 32));
        gv[pos] = v;
        gp[pos] = node;
        if (pos < kSoloNodes) {
            sh.v[0][pos] = v;
            sh.p[0][pos] = node;
        }
    };
    if (n <= kRankSort) {
        if (tid < n) so.time[0][tid] = __ldcg(s.ent_time + off + tid);
        __syncthreads();
        const uint32_t i = tid >> 2;
        const unsigned long long mine = i < n ? so.time[0][i] : 0ull;
        uint32_t below = 0;
        if (warp * 8 < n)
#pragma unroll 4
            for (uint32_t k = tid & 3; k < n; k += 4) below += so.time[0][k] < mine ? 1u : 0u;
        below += __shfl_xor_sync(0xFFFFFFFFu, below, 1);
        below += __shfl_xor_sync(0xFFFFFFFFu, below, 2);
        if (i < n && (tid & 3) == 0) put(below, i);
        __syncthreads();
        return;
    }
    // the bits in which the times differ
    unsigned long long vary = 0;
    const unsigned long long t0 = __ldcg(s.ent_time + off);
    for (uint32_t i = tid; i < n; i += kSmallThreads) {
        const unsigned long long t = __ldcg(s.ent_time + off + i);
        so.time[0][i] = t;
        so.at[0][i] = static_cast<uint16_t>(i);
        vary |= t ^ t0;
    }
    for (int o = 16; o > 0; o >>= 1) vary |= __shfl_xor_sync(0xFFFFFFFFu, vary, o);
    if (lane == 0) so.vary[warp] = vary;
    __syncthreads();
    vary = so.vary[lane % kSmallWarps];
    for (int o = 16; o > 0; o >>= 1) vary |= __shfl_xor_sync(0xFFFFFFFFu, vary, o);
    // warp w's run: steps of 32 entries
    const uint32_t steps = (n + kSmallThreads - 1) / kSmallThreads, run = warp * steps * 32;
    int src = 0;
    for (; vary; src ^= 1) {
        const int shift = __ffsll(static_cast<long long>(vary)) - 1;  // the next pass starts at a bit that varies
        vary = shift + kSortDigit < 64 ? vary & (~0ull << (shift + kSortDigit)) : 0ull;
        for (uint32_t i = tid; i < (1u << kSortDigit) * (kSmallWarps + 1); i += kSmallThreads) so.count[i] = 0;
        __syncthreads();
#pragma unroll 1
        for (uint32_t k = 0; k < steps && run + k * 32 < n; ++k) {
            const uint32_t i = run + k * 32 + lane;
            const bool in = i < n;
            const uint32_t d = in ? static_cast<uint32_t>(so.time[src][i] >> shift) & ((1u << kSortDigit) - 1u) : 0u;
            unsigned peers = __ballot_sync(0xFFFFFFFFu, in);
#pragma unroll
            for (int b = 0; b < kSortDigit; ++b) {
                const unsigned set = __ballot_sync(0xFFFFFFFFu, (d >> b) & 1u);
                peers &= (d >> b) & 1u ? set : ~set;
            }
            const int leader = __ffs(peers) - 1;
            uint32_t first = 0;
            if (in && static_cast<int>(lane) == leader) {  // the warp's own counter: no other warp writes it
                first = so.count[d * (kSmallWarps + 1) + warp];
                so.count[d * (kSmallWarps + 1) + warp] = first + __popc(peers);
            }
            first = __shfl_sync(0xFFFFFFFFu, first, leader & 31) + __popc(peers & lt);
            if (in) so.rank[i] = static_cast<uint16_t>(first);
            __syncwarp();
        }
        __syncthreads();
        // exclusive scan of the counters, digits first, then warps: two a thread
        uint32_t* two = so.count + (2 * tid / kSmallWarps) * (kSmallWarps + 1) + 2 * tid % kSmallWarps;
        const uint32_t c0 = two[0], c1 = two[1];
        uint32_t incl = c0 + c1;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= static_cast<unsigned>(o)) incl += t;
        }
        if (lane == 31) so.sum[warp] = incl;
        __syncthreads();
        uint32_t before = lane < warp ? so.sum[lane] : 0u;  // lane < warp < kSmallWarps
        before = __reduce_add_sync(0xFFFFFFFFu, before) + incl - c0 - c1;
        two[0] = before;
        two[1] = before + c0;
        __syncthreads();
#pragma unroll 1
        for (uint32_t k = 0; k < steps; ++k) {
            const uint32_t i = run + k * 32 + lane;
            if (i >= n) break;
            const unsigned long long t = so.time[src][i];
            const uint32_t d = static_cast<uint32_t>(t >> shift) & ((1u << kSortDigit) - 1u);
            const uint32_t pos = so.count[d * (kSmallWarps + 1) + warp] + so.rank[i];
            so.time[src ^ 1][pos] = t;
            so.at[src ^ 1][pos] = so.at[src][i];
        }
        __syncthreads();
    }
    for (uint32_t i = tid; i < n; i += kSmallThreads) put(i, so.at[src][i]);
    __syncthreads();
}

// Runs the flood from ctl (depth index, frontier) on; leaves in ctl where it stopped and why.
__global__ void __cluster_dims__(kSmallCluster, 1, 1) __launch_bounds__(kSmallThreads, 1)
    ws_small(WsState s, WsSmallArgs a, WsCtl* ctl) {
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    __shared__ WsSmallShared sh;
    extern __shared__ __align__(16) unsigned char dynamic[];
    WsSortShared& so = *reinterpret_cast<WsSortShared*>(dynamic);
    const unsigned tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, rank = cl.block_rank();
    if (tid < 27) {
        int dx, dy, dz;
        stencil_offset(static_cast<int>(tid), 0, dx, dy, dz);
        sh.delta[tid] = static_cast<uint32_t>((dz * static_cast<long long>(s.g.SX) + dx) * s.g.SY + dy);
    }
    if (tid == 0) {
        sh.log_used = kLogSlab;  // no slab yet
        sh.ups = 0;
    }
    WsCtl c = *ctl;
    bool staged = false;  // the first block: the frontier is in sh.v[cur]
    ws_small_slab(s, sh);
    __syncthreads();
    auto timed = [&](unsigned long long t0, uint32_t n) {  // the generation's class and time, in the claim slot
        if (!s.gen_hist || rank != 0 || tid != 0) return;
        const int hc = 31 - __clz(n);
        atomicAdd(&s.gen_hist[hc], 1ull);
        atomicAdd(&s.gen_hist[64 + hc], ws_clock() - t0);
    };
    for (;;) {
        if (rank == 0) {  // solo generations, bucket sorts and the way from depth to depth
            c.mode = kWsDone;
            for (;;) {
                // The host empties the log (and adds records) before it fills up. One thread looks for the
                // block: the other blocks may still be adding their first slabs to the counter, and
                // threads that read it for themselves could part ways here, at barriers that do not match.
                if ((c.n == 0 || (c.gen & 15) == 0) && __syncthreads_or(tid == 0 && 2ull * __ldcg(s.log_n) > s.log_cap)) {
                    c.mode = kWsGrow;
                    break;
                }
                if (c.n == 0) {  // the deepest depth with entries: the first warp looks at 32 at a time, for the block
                    if (warp == 0) {
                        uint32_t di = c.di, n0 = 0;
                        for (; di < a.ndepths; di += 32) {
                            uint32_t f = 0;
                            if (di + lane < a.ndepths) {
                                const uint32_t d = a.depths[di + lane];
                                f = static_cast<uint32_t>(__ldcg(s.bpos + d) - __ldg(a.boff + d));
                            }
                            const unsigned m = __ballot_sync(0xFFFFFFFFu, f != 0);
                            if (m) {
                                const int l = __ffs(m) - 1;
                                n0 = __shfl_sync(0xFFFFFFFFu, f, l);
                                di += l;
                                break;
                            }
                        }
                        if (lane == 0) {
                            sh.found_di = di;
                            sh.found_n = n0;
                        }
                    }
                    __syncthreads();
                    c.di = sh.found_di;
                    const uint32_t n0 = sh.found_n;
                    if (n0 == 0) break;  // done
                    c.n = n0;
                    if (n0 > kSmallSort) {
                        c.mode = kWsSort;
                        break;
                    }
                    c.cur = 0;
                    ws_small_bucket(s, sh, so, __ldg(a.boff + a.depths[c.di]), n0, a.gv0, a.gp0);
                    staged = true;
                }
                if (c.gen >= a.max_gen) {
                    c.mode = kWsLimit;
                    break;
                }
                if (c.n > kSoloNodes) {
                    c.mode = c.n > kSmallNodes ? kWsBig : kWsRun;
                    staged = false;
                    break;
                }
                uint32_t* gv = c.cur ? a.gv1 : a.gv0;
                uint32_t* gp = c.cur ? a.gp1 : a.gp0;
                if (!staged) {
                    if (tid < c.n) {
                        sh.v[c.cur][tid] = __ldcg(gv + tid);
                        sh.p[c.cur][tid] = __ldcg(gp + tid);
                    }
                    staged = true;
                    __syncthreads();
                }
                ++c.gen;
                const unsigned long long t0 = s.gen_hist ? ws_clock() : 0;
                const uint32_t n = ws_small_generation(s, sh, false, gv, gp, c.cur ? a.gv0 : a.gv1, c.cur ? a.gp0 : a.gp1,
                                                              static_cast<int>(c.cur), c.n, a.depths[c.di], c.gen);
                timed(t0, c.n);
                c.n = n;
                c.cur ^= 1;
                if (n == 0) {
                    ++c.di;
                    ws_small_flush(s, sh);
                }
            }
            if (c.mode != kWsRun) ws_small_flush(s, sh);
            if (tid == 0) sh.ctl = c;
        }
        cl.sync();
        if (rank != 0) c = *cl.map_shared_rank(&sh.ctl, 0);
        if (c.mode != kWsRun) break;
        while (c.n > kSoloNodes && c.n <= kSmallNodes && c.gen < a.max_gen) {
            ++c.gen;
            const unsigned long long t0 = s.gen_hist ? ws_clock() : 0;
            const uint32_t n = ws_small_generation(s, sh, true, c.cur ? a.gv1 : a.gv0, c.cur ? a.gp1 : a.gp0,
                                                         c.cur ? a.gv0 : a.gv1, c.cur ? a.gp0 : a.gp1, 0, c.n,
                                                         a.depths[c.di], c.gen);
            timed(t0, c.n);
            c.n = n;
            c.cur ^= 1;
            if ((c.gen & 15) == 0) break;  // the first block looks at the log
        }
        // every block's claims are in their buckets before the first block reads one
        ws_small_flush(s, sh);
        cl.sync();
        if (c.n == 0) ++c.di;
    }
    if (rank == 0 && tid == 0) *ctl = c;
    cl.sync();  // no block ends while another reads its shared memory
}

__global__ void ws_unpack_entries(const unsigned long long* __restrict__ val, size_t n, Grid g,
                                  uint32_t* __restrict__ gv, uint32_t* __restrict__ gp) {
    PMA_GRID_STRIDE(i, n) {
        const uint32_t v = static_cast<uint32_t>(val[i]);
        gv[i] = v;
        gp[i] = ws_node(g, v, static_cast<uint32_t>(val[i] >> 32));
    }
}

__global__ void ws_volumes(const unsigned long long* __restrict__ state, int packed,
                           const uint32_t* __restrict__ ext, size_t n, unsigned long long* __restrict__ pvol,
                           uint8_t* __restrict__ shared_flag) {
    // lanes of a warp claimed by the same pore combine their counts
    const unsigned lane = threadIdx.x & 31;
    PMA_GRID_STRIDE(v, n) {
        const uint32_t c = ws_claimer(packed, state[v]);
        const bool sh = ext[v] != 0;
        shared_flag[v] = sh;
        const uint32_t key = (c && !sh) ? c : 0u;
        const unsigned peers = __match_any_sync(__activemask(), key);
        if (key && static_cast<int>(lane) == __ffs(peers) - 1)
            atomicAdd(&pvol[key - 1], static_cast<unsigned long long>(__popc(peers)));
    }
}

// --- shared types -------------------------------------------------------------------------

// Extending pores of the shared voxel whose chain starts at record `rec`, with their first
// touch times, in slot order; returns how many (at most kMaxExt).
__device__ __forceinline__ int ws_chain(const uint32_t* __restrict__ ext_pore,
                                        const unsigned long long* __restrict__ ext_time,
                                        const uint32_t* __restrict__ ext_next, uint32_t rec, uint32_t* p,
                                        unsigned long long* t) {
    int m = 0;
    for (int hop = 0; hop < kMaxHops && rec != 0 && rec != kRecBusy; ++hop) {
        for (int k = 0; k < kSlots; ++k) {
            const size_t slot = static_cast<size_t>(rec - 1) * kSlots + k;
            const uint32_t pk = ext_pore[slot];
            if (pk == kNone) return m;
            if (p) {
                p[m] = pk;
                t[m] = ext_time[slot];
            }
            ++m;
        }
        rec = ext_next[rec - 1];
    }
    return m;
}

// Key length (claimer + extending pores) of each shared voxel, for the offsets of its key and
// of its prefix records.
__global__ void ws_key_lengths(const uint32_t* __restrict__ sv, size_t ns, const uint32_t* __restrict__ ext,
                               const uint32_t* __restrict__ ext_pore, const uint32_t* __restrict__ ext_next,
                               uint8_t* __restrict__ klen, unsigned long long* __restrict__ klen64) {
    PMA_GRID_STRIDE(i, ns) {
        const int len = ws_chain(ext_pore, nullptr, ext_next, ext[sv[i]], nullptr, nullptr) + 1;
        klen[i] = static_cast<uint8_t>(len);
        klen64[i] = static_cast<unsigned long long>(len);
    }
}

// Key of shared voxel i: [first extension, claimer, later extensions...] in pore indices, at
// kseq[koff[i] ..], and one record per prefix of length L = 2..len at record
// koff[i] - i + L - 2 (its hashes, creation time and voxel).
__global__ void ws_keys(const uint32_t* __restrict__ sv, size_t ns, const unsigned long long* __restrict__ state,
                        int packed,
                        const uint32_t* __restrict__ ext, const uint32_t* __restrict__ ext_pore,
                        const unsigned long long* __restrict__ ext_time, const uint32_t* __restrict__ ext_next,
                        const unsigned long long* __restrict__ koff, uint32_t* __restrict__ kseq,
                        unsigned long long* __restrict__ rh1, unsigned long long* __restrict__ rh2,
                        unsigned long long* __restrict__ rtime, uint32_t* __restrict__ rvox) {
    PMA_GRID_STRIDE(i, ns) {
        const uint32_t v = sv[i];
        uint32_t p[kMaxExt];
        unsigned long long t[kMaxExt];
        const int m = ws_chain(ext_pore, ext_time, ext_next, ext[v], p, t);
        for (int a = 1; a < m; ++a)  // insertion sort by time
            for (int b = a; b > 0 && t[b] < t[b - 1]; --b) {
                const unsigned long long tt = t[b];
                t[b] = t[b - 1];
                t[b - 1] = tt;
                const uint32_t pp = p[b];
                p[b] = p[b - 1];
                p[b - 1] = pp;
            }
        uint32_t key[kKeyMax];
        key[0] = p[0];
        key[1] = ws_claimer(packed, state[v]) - 1;
        for (int k = 1; k < m; ++k) key[k + 1] = p[k];
        const int len = m + 1;
        const unsigned long long base = koff[i];
        for (int k = 0; k < len; ++k) kseq[base + k] = key[k];
        const unsigned long long rbase = base - i;
        for (int L = 2; L <= len; ++L) {
            const unsigned long long r = rbase + (L - 2);
            unsigned long long h1, h2;
            list_hash(key, static_cast<uint32_t>(L), h1, h2);
            rh1[r] = h1;
            rh2[r] = h2;
            rtime[r] = t[L - 2];
            rvox[r] = static_cast<uint32_t>(i);
        }
    }
}

__global__ void ws_gather_h(const unsigned long long* __restrict__ h, const uint32_t* __restrict__ idx,
                            size_t n, unsigned long long* __restrict__ out) {
    PMA_GRID_STRIDE(i, n) out[i] = h[idx[i]];
}

// Prefix record r: its voxel, the start of that voxel's key and the prefix length.
struct RecRef {
    uint32_t vi;
    unsigned long long kbase;
    uint32_t L;
};

__device__ __forceinline__ RecRef ws_rec(uint32_t r, const uint32_t* __restrict__ rvox,
                                         const unsigned long long* __restrict__ koff) {
    RecRef x;
    x.vi = rvox[r];
    x.kbase = koff[x.vi];
    x.L = static_cast<uint32_t>(r - (x.kbase - x.vi)) + 2u;
    return x;
}

__global__ void ws_group_starts(const uint32_t* __restrict__ rec, size_t nr,
                                const unsigned long long* __restrict__ rh1,
                                const unsigned long long* __restrict__ rh2, const uint32_t* __restrict__ kseq,
                                const unsigned long long* __restrict__ koff, const uint32_t* __restrict__ rvox,
                                uint32_t* __restrict__ start, unsigned int* __restrict__ err) {
    PMA_GRID_STRIDE(i, nr) {
        const uint32_t r = rec[i];
        bool s = i == 0;
        if (!s) {
            const uint32_t q = rec[i - 1];
            s = rh1[r] != rh1[q] || rh2[r] != rh2[q];
            // equal first hashes, different second ones: sorted by the first hash alone, such
            // prefixes may interleave (the host then sorts by both)
            if (rh1[r] == rh1[q] && rh2[r] != rh2[q]) atomicOr(err, 64u);
            if (!s) {  // verify: same prefix
                const RecRef a = ws_rec(r, rvox, koff), b = ws_rec(q, rvox, koff);
                bool eq = a.L == b.L;
                for (uint32_t k = 0; eq && k < a.L; ++k) eq = kseq[a.kbase + k] == kseq[b.kbase + k];
                if (!eq) atomicOr(err, 4u);
            }
        }
        start[i] = s ? 1u : 0u;
    }
}

__global__ void ws_group_reduce(const uint32_t* __restrict__ rec, const uint32_t* __restrict__ excl,
                                const uint32_t* __restrict__ start, size_t nr,
                                const unsigned long long* __restrict__ rtime, const uint8_t* __restrict__ klen,
                                const unsigned long long* __restrict__ koff, const uint32_t* __restrict__ rvox,
                                unsigned long long* __restrict__ gtime, unsigned long long* __restrict__ gvol,
                                uint32_t* __restrict__ grep, uint32_t* __restrict__ final_group) {
    PMA_GRID_STRIDE(i, nr) {
        const uint32_t r = rec[i];
        const uint32_t g = excl[i] + start[i] - 1u;
        atomicMin(&gtime[g], rtime[r]);
        const RecRef a = ws_rec(r, rvox, koff);
        if (a.L == klen[a.vi]) {
            atomicAdd(&gvol[g], 1ull);
            final_group[a.vi] = g;
        }
        if (start[i]) grep[g] = r;
    }
}

__global__ void ws_labels(const unsigned long long* __restrict__ state, int packed, size_t n,
                          const uint32_t* __restrict__ pore_id, uint32_t* __restrict__ labels) {
    PMA_GRID_STRIDE(v, n) {
        const uint32_t c = ws_claimer(packed, state[v]);
        labels[v] = c ? pore_id[c - 1] : 0u;
    }
}

__global__ void ws_shared_labels(const uint32_t* __restrict__ sv, const uint32_t* __restrict__ final_group,
                                 const uint32_t* __restrict__ gid, size_t ns, uint32_t* __restrict__ labels) {
    PMA_GRID_STRIDE(i, ns) labels[sv[i]] = gid[final_group[i]];
}

// A type's pore ids in the order of its list: the prefix that its representative record stands for.
struct PrefixLists {
    const uint32_t* grep;
    const uint32_t* kseq;
    const unsigned long long* koff;
    const uint32_t* rvox;
    const uint32_t* pore_id;
    __device__ __forceinline__ uint32_t length(uint32_t g) const { return ws_rec(grep[g], rvox, koff).L; }
    __device__ __forceinline__ uint32_t pore(uint32_t g, uint32_t j) const {
        return pore_id[kseq[ws_rec(grep[g], rvox, koff).kbase + j]];
    }
};

// The dynamic shared-memory limit is a process-wide attribute of the kernel: set once per device.
void small_smem_attribute() {
    static std::mutex mutex;
    static std::vector<int> devices;
    int dev = 0;
    PMA_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(mutex);
    if (std::find(devices.begin(), devices.end(), dev) != devices.end()) return;
    PMA_CUDA(cudaFuncSetAttribute(ws_small, cudaFuncAttributeMaxDynamicSharedMemorySize, sizeof(WsSortShared)));
    PMA_CUDA(cudaFuncSetAttribute(ws_small, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    devices.push_back(dev);
}

template <class T>
T* buf(pma_ctx* ctx, const char* tag, size_t count) {
    return static_cast<T*>(ctx->scratch(tag, std::max<size_t>(count, 1) * sizeof(T)));
}

}  // namespace

pma_table* watershed(pma_ctx* ctx, const pma_table* pt, const uint32_t* crad2, pma_dims d,
                     pma_stencil st, uint32_t max_edt2, uint32_t* labels) {
    KernelTimer kt_stage(ctx, "stage_watershed");  // the whole stage, for the untimed remainder
    check_dims(d);
    PMA_REQUIRE(crad2 && labels, PMA_ERR_ARGUMENT, "pma_watershed: null device pointer");
    PMA_REQUIRE(pt->pores.size() < kFace, PMA_ERR_ARGUMENT, "pma_watershed: too many pores");
    cudaStream_t s = ctx->stream;
    const size_t n = voxels(d);
    const Grid g{d.sx, d.sy, d.sz};
    const unsigned G = grid_for(ctx, n);
    const size_t npores = pt->pores.size();
    const uint32_t nb = max_edt2 + 1;

    // Seeds (WatershedComputer.cpp:183-219), in pore-id order.
    std::vector<pma_pore> pores = pt->pores;
    std::sort(pores.begin(), pores.end(), [](const pma_pore& a, const pma_pore& b) { return a.id < b.id; });
    std::vector<uint32_t> seed_voxel(npores);
    std::vector<uint32_t> seed_hist(nb, 0);
    for (size_t k = 0; k < npores; ++k) {
        const pma_pore& p = pores[k];
        PMA_REQUIRE(g.inside(p.seed_x, p.seed_y, p.seed_z), PMA_ERR_ARGUMENT,
                    "pma_watershed: pore seed outside the image");
        PMA_REQUIRE(p.seed_r2 <= max_edt2, PMA_ERR_ARGUMENT, "pma_watershed: pore seed radius above max_edt2");
        seed_voxel[k] = static_cast<uint32_t>(g.idx(p.seed_x, p.seed_y, p.seed_z));
        seed_hist[p.seed_r2]++;
    }
    {
        std::vector<uint32_t> sv = seed_voxel;
        std::sort(sv.begin(), sv.end());
        PMA_REQUIRE(std::adjacent_find(sv.begin(), sv.end()) == sv.end(), PMA_ERR_ARGUMENT,
                    "pma_watershed: two pores share a seed voxel");
    }

    small_smem_attribute();
    int64_t* d_count = buf<int64_t>(ctx, "ws.count", 4);
    unsigned int* d_ng = reinterpret_cast<unsigned int*>(d_count + 3);  // two frontier sizes
    WsState ws;
    ws.g = g;
    ws.d3q7 = st == PMA_D3Q7 ? 1 : 0;
    ws.crad = crad2;
    ws.state = buf<unsigned long long>(ctx, "ws.state", n);
    ws.packed = max_edt2 < 65536u ? 1 : 0;  // radii up to max_edt2 fit the word's low 16 bits
    ws.ext = buf<uint32_t>(ctx, "ws.ext", n);
    ws.ext_count = reinterpret_cast<unsigned int*>(d_count + 1);
    ws.err = reinterpret_cast<unsigned int*>(d_count + 2);
    ws.spin_limit = ctx->limits.spin_limit;
    ws.gen_hist = nullptr;
    if (ctx->timing) {  // frontier sizes of the generations, for the timing report
        ws.gen_hist = buf<unsigned long long>(ctx, "ws.gen_hist", 192);
        PMA_CUDA(cudaMemsetAsync(ws.gen_hist, 0, 192 * 8, s));
    }
    ws.pbound = buf<unsigned int>(ctx, "ws.pbound", npores);
    // Shared-voxel records: a first guess of n/32; the pool doubles (copying the records)
    // whenever it is more than half used when the log is emptied, and a flood that still runs
    // out is redone with four times as many (up to two per voxel).
    const size_t max_records = std::min<size_t>(2 * n + 4096, 0x7FFFFFFF / kSlots);
    size_t ext_cap = std::min<size_t>(std::max<size_t>(n / 32, 4096), max_records);
    int ext_side = 0;  // which of two scratch tags holds the records
    auto ext_tag = [&](const char* base) { return std::string(base) + (ext_side ? ".1" : ".0"); };
    auto grow_records = [&](size_t used) {
        if (2 * used <= ws.ext_cap || ws.ext_cap >= max_records) return;
        const size_t old_cap = ws.ext_cap;
        const size_t cap2 = std::min<size_t>(std::max<size_t>(2 * old_cap, 4 * used), max_records);
        const std::string old_p = ext_tag("ws.ext_pore"), old_t = ext_tag("ws.ext_time"),
                          old_n = ext_tag("ws.ext_next");
        ext_side ^= 1;
        auto* np_ = buf<uint32_t>(ctx, ext_tag("ws.ext_pore").c_str(), cap2 * kSlots);
        auto* nt_ = buf<unsigned long long>(ctx, ext_tag("ws.ext_time").c_str(), cap2 * kSlots);
        auto* nn_ = buf<uint32_t>(ctx, ext_tag("ws.ext_next").c_str(), cap2);
        PMA_CUDA(cudaMemcpyAsync(np_, ws.ext_pore, old_cap * kSlots * 4, cudaMemcpyDeviceToDevice, s));
        PMA_CUDA(cudaMemcpyAsync(nt_, ws.ext_time, old_cap * kSlots * 8, cudaMemcpyDeviceToDevice, s));
        PMA_CUDA(cudaMemcpyAsync(nn_, ws.ext_next, old_cap * 4, cudaMemcpyDeviceToDevice, s));
        PMA_CUDA(cudaMemsetAsync(np_ + old_cap * kSlots, 0xFF, (cap2 - old_cap) * kSlots * 4, s));
        PMA_CUDA(cudaMemsetAsync(nt_ + old_cap * kSlots, 0xFF, (cap2 - old_cap) * kSlots * 8, s));
        PMA_CUDA(cudaMemsetAsync(nn_ + old_cap, 0, (cap2 - old_cap) * 4, s));
        ctx->release(old_p);
        ctx->release(old_t);
        ctx->release(old_n);
        ws.ext_pore = np_;
        ws.ext_time = nt_;
        ws.ext_next = nn_;
        ws.ext_cap = static_cast<uint32_t>(cap2);
    };
    // Extension log: emptied when it is more than half full at a host synchronisation point.
    const size_t log_cap = std::min<size_t>(n / 8 + (1u << 16), 1u << 30);
    ws.log = buf<ulonglong2>(ctx, "ws.log", log_cap);
    ws.log_cap = static_cast<uint32_t>(log_cap);
    ws.log_n = reinterpret_cast<unsigned long long*>(d_count);  // counts other things after the flood
    size_t used = 0;  // records in use when the log was last emptied
    auto record_extensions = [&](unsigned long long reserved) {
        const size_t noted = static_cast<size_t>(std::min<unsigned long long>(reserved, log_cap));
        ctx->count("ws.log_entries", static_cast<double>(noted));
        if (reserved > log_cap) ctx->count("ws.log_overflow", static_cast<double>(reserved - log_cap));
        unsigned int* h_used = static_cast<unsigned int*>(ctx->host_staging(128)) + 28;
        size_t at = 0;
        // each entry takes at most one new record: as many entries as records are free at a time
        while (at < noted) {
            size_t m = noted - at;
            if (ws.ext_cap < max_records) m = std::min<size_t>(m, std::max<size_t>(ws.ext_cap - std::min<size_t>(used, ws.ext_cap), 1));
            ws_record_extensions<<<grid_for(ctx, m), 256, 0, s>>>(ws, static_cast<uint32_t>(at), static_cast<uint32_t>(at + m));
            ctx->check_launch("ws_record_extensions");
            at += m;
            ReadBack rb;
            rb.add(h_used, ws.ext_count, 4);
            read_back(ctx, rb);
            used = *h_used;
            grow_records(used);
        }
        PMA_CUDA(cudaMemsetAsync(ws.log, 0xFF, noted * sizeof(ulonglong2), s));
        PMA_CUDA(cudaMemsetAsync(ws.log_n, 0, 8, s));
    };
    unsigned int h_err = 0;
    for (;;) {
        const size_t start_cap = ext_cap;
        used = 0;
        ws.ext_cap = static_cast<uint32_t>(ext_cap);
        ws.ext_pore = buf<uint32_t>(ctx, ext_tag("ws.ext_pore").c_str(), static_cast<size_t>(ws.ext_cap) * kSlots);
        ws.ext_time = buf<unsigned long long>(ctx, ext_tag("ws.ext_time").c_str(),
                                              static_cast<size_t>(ws.ext_cap) * kSlots);
        ws.ext_next = buf<uint32_t>(ctx, ext_tag("ws.ext_next").c_str(), ws.ext_cap);
        PMA_CUDA(cudaMemsetAsync(ws.ext_next, 0, static_cast<size_t>(ws.ext_cap) * 4, s));
        PMA_CUDA(cudaMemsetAsync(d_count, 0, 32, s));
        PMA_CUDA(cudaMemsetAsync(ws.log, 0xFF, log_cap * sizeof(ulonglong2), s));
        PMA_CUDA(cudaMemsetAsync(ws.ext_pore, 0xFF, static_cast<size_t>(ws.ext_cap) * kSlots * 4, s));
        PMA_CUDA(cudaMemsetAsync(ws.ext_time, 0xFF, static_cast<size_t>(ws.ext_cap) * kSlots * 8, s));
        PMA_CUDA(cudaMemsetAsync(ws.pbound, 0, std::max<size_t>(npores, 1) * 4, s));
        ws_init<<<G, 256, 0, s>>>(n, crad2, ws.packed, ws.state, ws.ext);
        ctx->check_launch("ws_init");

        // Buckets: capacity = voxels of that crad + seeds of that radius.
        unsigned int* hist = buf<unsigned int>(ctx, "ws.hist", nb);
        PMA_CUDA(cudaMemsetAsync(hist, 0, nb * 4ull, s));
        ws_histograms<<<G, 256, 0, s>>>(crad2, n, nb, hist);
        ctx->check_launch("ws_histograms");
        std::vector<unsigned int> h_hist(nb);
        PMA_CUDA(cudaMemcpyAsync(h_hist.data(), hist, nb * 4ull, cudaMemcpyDeviceToHost, s));
        ctx->sync();
        std::vector<unsigned long long> boff(nb + 1, 0);
        size_t max_bucket = 1;
        for (uint32_t b = 0; b < nb; ++b) {
            const unsigned long long c = static_cast<unsigned long long>(h_hist[b]) + seed_hist[b];
            boff[b + 1] = boff[b] + c;
            max_bucket = std::max<size_t>(max_bucket, c);
        }
        const unsigned long long total = boff[nb];
        auto* d_boff = buf<unsigned long long>(ctx, "ws.boff", nb + 1);
        ws.bpos = buf<unsigned long long>(ctx, "ws.bpos", nb);
        ws.ent_time = buf<unsigned long long>(ctx, "ws.ent_time", total);
        ws.ent_val = buf<unsigned long long>(ctx, "ws.ent_val", total);
        auto* srt_time = buf<unsigned long long>(ctx, "ws.srt_time", max_bucket);
        auto* srt_val = buf<unsigned long long>(ctx, "ws.srt_val", max_bucket);
        const size_t max_events = max_bucket * 27;
        // bucket entry times: events (and the seeds' pore indices) below 2^time_shift, so that a
        // depth's sort needs only time_shift + bits(generation) key bits
        ws.time_shift = 1;
        while (ws.time_shift < 41 && (1ull << ws.time_shift) <= std::max<size_t>(max_events, npores)) ++ws.time_shift;

        // event bits, whole strips; every word of a generation's strips is written before it is read
        const size_t max_strips = (max_events + kStrip * 32 - 1) / (kStrip * 32);
        ws.touched = buf<uint32_t>(ctx, "ws.touched", max_strips * kStrip);
        ws.won = buf<uint32_t>(ctx, "ws.won", max_strips * kStrip);
        PMA_CUDA(cudaMemcpyAsync(d_boff, boff.data(), (nb + 1) * 8ull, cudaMemcpyHostToDevice, s));
        std::vector<unsigned int> h_fill(nb, 0);
        if (npores) {
            std::vector<unsigned long long> a(3 * npores);
            for (size_t k = 0; k < npores; ++k) {
                const uint32_t b = pores[k].seed_r2;
                a[k] = boff[b] + h_fill[b]++;
                a[npores + k] = k;  // seeds come first in their bucket, in pore-id order
                a[2 * npores + k] = (static_cast<unsigned long long>(k) << 32) | seed_voxel[k];
            }
            auto* d_a = buf<unsigned long long>(ctx, "ws.seed_at", 3 * npores);
            PMA_CUDA(cudaMemcpyAsync(d_a, a.data(), 3 * npores * 8, cudaMemcpyHostToDevice, s));
            ws_seed_entries<<<grid_for(ctx, npores), 256, 0, s>>>(d_a, npores, ws.ent_time, ws.ent_val);
            ctx->check_launch("ws_seed_entries");
            uint32_t* d_seed = buf<uint32_t>(ctx, "ws.seedvox", npores);
            PMA_CUDA(cudaMemcpyAsync(d_seed, seed_voxel.data(), npores * 4, cudaMemcpyHostToDevice, s));
            ws_seed<<<grid_for(ctx, npores), 256, 0, s>>>(d_seed, npores, crad2, ws.packed, ws.state);
            ctx->check_launch("ws_seed");
            ctx->sync();
        }
        std::vector<unsigned long long> bpos(boff.begin(), boff.end() - 1);
        for (uint32_t b = 0; b < nb; ++b) bpos[b] += h_fill[b];
        PMA_CUDA(cudaMemcpyAsync(ws.bpos, bpos.data(), nb * 8ull, cudaMemcpyHostToDevice, s));
        ctx->sync();

        // Depth sweep (WatershedComputer.cpp:80-102).
        uint32_t* gvb[2] = {buf<uint32_t>(ctx, "ws.gv0", max_bucket), buf<uint32_t>(ctx, "ws.gv1", max_bucket)};
        uint32_t* gpb[2] = {buf<uint32_t>(ctx, "ws.gp0", max_bucket), buf<uint32_t>(ctx, "ws.gp1", max_bucket)};
        // cooperative grid: every block resident at once (grid-wide barriers)
        int per_sm = 0;
        PMA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, ws_generations, kGenThreads, 0));
        PMA_REQUIRE(per_sm > 0, PMA_ERR_CUDA, "pma_watershed: generation kernel does not fit an SM");
        // sized to the largest frontier (four strips a warp), so that the launches of small volumes
        // leave the rest of the GPU to other streams (batch lanes)
        const unsigned coop_grid = static_cast<unsigned>(std::max<size_t>(
            1, std::min<size_t>((max_strips + 4 * kGenWarps - 1) / (4 * kGenWarps),
                                static_cast<size_t>(ctx->num_sms) * std::min(per_sm, 8))));
        unsigned int* counts = buf<unsigned int>(ctx, "ws.counts", coop_grid);  // claims of each block's range
        // generations of this call at most: the context's bound, within the entry-time range
        const unsigned long long max_gen =
            std::min<unsigned long long>(ctx->limits.watershed_generations, kMaxGen - 1);
        // pinned words: frontier sizes and the record count, the launches' results, the flood's state
        unsigned int* h_small = static_cast<unsigned int*>(ctx->host_staging(128));
        auto* h_log_n = reinterpret_cast<unsigned long long*>(h_small + 4);
        auto* d_out = buf<unsigned long long>(ctx, "ws.coop_out", 2);
        unsigned long long* h_out = reinterpret_cast<unsigned long long*>(h_small + 8);
        auto* d_ctl = reinterpret_cast<WsCtl*>(buf<unsigned long long>(ctx, "ws.ctl", 3));
        static_assert(sizeof(WsCtl) == 24, "three words");
        WsCtl* h_ctl = reinterpret_cast<WsCtl*>(h_small + 16);
        // depths that can hold entries, deepest first
        std::vector<uint32_t> depths;
        for (int64_t depth = static_cast<int64_t>(nb) - 1; depth >= 0; --depth)
            if (boff[depth + 1] != boff[depth]) depths.push_back(static_cast<uint32_t>(depth));
        uint32_t* d_depths = buf<uint32_t>(ctx, "ws.depths", depths.size());
        if (!depths.empty())
            PMA_CUDA(cudaMemcpyAsync(d_depths, depths.data(), depths.size() * 4, cudaMemcpyHostToDevice, s));
        WsSmallArgs sa{gvb[0], gpb[0], gvb[1], gpb[1], d_depths, static_cast<uint32_t>(depths.size()), d_boff, max_gen};
        WsCtl c{0, 0, 0, 0, kWsRun};
        for (;;) {
            // small buckets and generations, depth after depth
            {
                KernelTimer kt(ctx, "ws_small");
                *h_ctl = c;
                PMA_CUDA(cudaMemcpyAsync(d_ctl, h_ctl, sizeof(c), cudaMemcpyHostToDevice, s));
                ws_small<<<kSmallCluster, kSmallThreads, sizeof(WsSortShared), s>>>(ws, sa, d_ctl);
                ctx->check_launch("ws_small");
                ctx->count("ws.small_launches", 1);
                ReadBack rb;
                rb.add(h_ctl, d_ctl, sizeof(c));
                rb.add(h_log_n, ws.log_n, 8);
                read_back(ctx, rb);
                c = *h_ctl;
            }
            if (c.mode == kWsDone || 2 * *h_log_n > ws.log_cap) record_extensions(*h_log_n);
            if (c.mode == kWsDone) break;
            PMA_REQUIRE(c.mode != kWsLimit, PMA_ERR_LIMIT, "pma_watershed: generation limit reached");
            if (c.mode == kWsGrow) {
                ctx->count("ws.log_stops", 1);
                continue;
            }
            const uint32_t dep = depths[c.di];
            int cur = static_cast<int>(c.cur);
            if (c.mode == kWsSort) {
                KernelTimer kt(ctx, "ws_depth_sort");
                cur = 0;
                int gen_bits = 0;
                while (gen_bits < 24 && (1ull << gen_bits) <= c.gen) ++gen_bits;
                sort_pairs(ctx, ws.ent_time + boff[dep], srt_time, ws.ent_val + boff[dep], srt_val,
                           static_cast<int64_t>(c.n), std::min(64, ws.time_shift + gen_bits));
                ws_unpack_entries<<<grid_for(ctx, c.n), 256, 0, s>>>(srt_val, c.n, g, gvb[cur], gpb[cur]);
                ctx->check_launch("ws_unpack_entries");
            }
            h_small[2] = c.n;
            PMA_CUDA(cudaMemcpyAsync(d_ng + cur, &h_small[2], 4, cudaMemcpyHostToDevice, s));
            // large generations of this depth, until the frontier is small
            KernelTimer kt(ctx, "ws_generations");
            while (c.n > kSmallNodes) {
                PMA_REQUIRE(c.gen < max_gen, PMA_ERR_LIMIT, "pma_watershed: generation limit reached");
                int gens = static_cast<int>(std::min<unsigned long long>(kGensPerLaunch, max_gen - c.gen));
                unsigned small_nodes = kSmallNodes;
                void* args[] = {&ws, &gvb[0], &gpb[0], &gvb[1], &gpb[1], &d_ng, &counts,
                                const_cast<uint32_t*>(&dep), &c.gen, &gens, &cur, &small_nodes, &d_out};
                PMA_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(ws_generations), coop_grid,
                                                     kGenThreads, args, 0, s));
                ctx->count_launch(1);
                ctx->count("ws.cooperative_launches", 1);
                ReadBack rb;
                rb.add(h_out, d_out, 16);
                rb.add(h_log_n, ws.log_n, 8);
                rb.add(h_small + 6, d_ng, 8);
                read_back(ctx, rb);
                c.gen += h_out[0];
                cur = static_cast<int>(h_out[1]);
                c.n = h_small[6 + cur];
                if (2 * *h_log_n > ws.log_cap) record_extensions(*h_log_n);
            }
            c.cur = static_cast<uint32_t>(cur);
            if (c.n == 0) ++c.di;
        }
        PMA_CUDA(cudaMemcpyAsync(&h_err, ws.err, 4, cudaMemcpyDeviceToHost, s));
        ctx->sync();
        if (!(h_err & 1u)) break;
        PMA_REQUIRE(start_cap < max_records, PMA_ERR_MEMORY, "pma_watershed: shared-voxel records exhausted");
        ext_cap = std::min<size_t>(std::max<size_t>(ws.ext_cap, start_cap * 4), max_records);
    }
    PMA_REQUIRE(!(h_err & 2u), PMA_ERR_INTERNAL, "pma_watershed: a shared voxel recorded more pores than touch it");
    PMA_REQUIRE(!(h_err & 8u), PMA_ERR_LIMIT, "pma_watershed: shared-voxel record allocation did not finish");
    if (ws.gen_hist) {
        unsigned long long hh[192];
        PMA_CUDA(cudaMemcpyAsync(hh, ws.gen_hist, sizeof(hh), cudaMemcpyDeviceToHost, s));
        ctx->sync();
        for (int b = 0; b < 64; ++b)
            if (hh[b]) {
                const std::string c = "ws.generations.frontier_2^" + std::to_string(b);
                ctx->count(c, static_cast<double>(hh[b]));
                ctx->count(c + ".claim_ms", hh[64 + b] * 1e-6);
                ctx->count(c + ".resolve_ms", hh[128 + b] * 1e-6);
            }
    }

    KernelTimer kt_tables(ctx, "ws_tables");  // to the end of the stage
    // Volumes, labels and shared voxels.
    auto* pvol = buf<unsigned long long>(ctx, "ws.pvol", npores);
    uint8_t* shared_flag = buf<uint8_t>(ctx, "ws.shared_flag", n);
    PMA_CUDA(cudaMemsetAsync(pvol, 0, std::max<size_t>(npores, 1) * 8, s));
    ws_volumes<<<G, 256, 0, s>>>(ws.state, ws.packed, ws.ext, n, pvol, shared_flag);
    ctx->check_launch("ws_volumes");
    std::vector<uint32_t> pore_id(std::max<size_t>(npores, 1));
    for (size_t k = 0; k < npores; ++k) pore_id[k] = pores[k].id;
    uint32_t* d_pid = buf<uint32_t>(ctx, "ws.pid", pore_id.size());
    PMA_CUDA(cudaMemcpyAsync(d_pid, pore_id.data(), pore_id.size() * 4, cudaMemcpyHostToDevice, s));
    ws_labels<<<G, 256, 0, s>>>(ws.state, ws.packed, n, d_pid, labels);
    ctx->check_launch("ws_labels");
    uint32_t* sv = buf<uint32_t>(ctx, "ws.sv", n);
    const int64_t nsh = select_flagged(ctx, thrust::counting_iterator<uint32_t>(0), shared_flag, sv,
                                       static_cast<int64_t>(n), d_count);

    pma_table* t = new pma_table;
    std::vector<unsigned long long> h_pvol(npores);
    std::vector<unsigned int> h_pbound(npores);
    if (npores) {
        PMA_CUDA(cudaMemcpyAsync(h_pvol.data(), pvol, npores * 8, cudaMemcpyDeviceToHost, s));
        PMA_CUDA(cudaMemcpyAsync(h_pbound.data(), ws.pbound, npores * 4, cudaMemcpyDeviceToHost, s));
        ctx->sync();
    }
    for (size_t k = 0; k < npores; ++k) {
        pma_pore p = pores[k];
        p.volume = h_pvol[k];
        p.is_boundary = h_pbound[k] ? 1 : 0;
        t->pores.push_back(p);
    }
    if (nsh == 0) return t;

    // Shared types on the device: key lengths, key and prefix-record offsets, keys and
    // prefix records, then the prefixes grouped by hash and ranked by creation time.
    uint8_t* klen = buf<uint8_t>(ctx, "ws.klen", nsh);
    auto* klen64 = buf<unsigned long long>(ctx, "ws.klen64", nsh);
    auto* koff = buf<unsigned long long>(ctx, "ws.koff", nsh);
    ws_key_lengths<<<grid_for(ctx, nsh), 256, 0, s>>>(sv, nsh, ws.ext, ws.ext_pore, ws.ext_next, klen, klen64);
    ctx->check_launch("ws_key_lengths");
    exclusive_sum(ctx, klen64, koff, nsh);
    unsigned long long kl[2] = {0, 0};
    PMA_CUDA(cudaMemcpyAsync(&kl[0], koff + nsh - 1, 8, cudaMemcpyDeviceToHost, s));
    PMA_CUDA(cudaMemcpyAsync(&kl[1], klen64 + nsh - 1, 8, cudaMemcpyDeviceToHost, s));
    ctx->sync();
    const unsigned long long nkey = kl[0] + kl[1];      // key elements of all shared voxels
    const unsigned long long nrec_u = nkey - static_cast<unsigned long long>(nsh);  // prefixes
    PMA_REQUIRE(nrec_u < 0xFFFFFFFFull, PMA_ERR_LIMIT, "pma_watershed: too many shared voxels");
    const int64_t nr = static_cast<int64_t>(nrec_u);
    uint32_t* kseq = buf<uint32_t>(ctx, "ws.kseq", nkey);
    auto* rh1 = buf<unsigned long long>(ctx, "ws.rh1", nr);
    auto* rh2 = buf<unsigned long long>(ctx, "ws.rh2", nr);
    auto* rtime = buf<unsigned long long>(ctx, "ws.rtime", nr);
    uint32_t* rvox = buf<uint32_t>(ctx, "ws.rvox", nr);
    ws_keys<<<grid_for(ctx, nsh), 256, 0, s>>>(sv, nsh, ws.state, ws.packed, ws.ext, ws.ext_pore, ws.ext_time, ws.ext_next,
                                               koff, kseq, rh1, rh2, rtime, rvox);
    ctx->check_launch("ws_keys");
    uint32_t* rec = buf<uint32_t>(ctx, "ws.rec", nr);
    uint32_t* rec2 = buf<uint32_t>(ctx, "ws.rec2", nr);
    type_iota<<<grid_for(ctx, nr), 256, 0, s>>>(rec, nr);
    ctx->check_launch("type_iota");
    // Equal prefixes become adjacent: a radix sort by the first hash (values: record ids),
    // unless two different prefixes share it (about n^2 / 2^65 likely), which ws_group_starts
    // flags; then stable sorts by the second hash and then the first.
    auto* kh = buf<unsigned long long>(ctx, "ws.kh", nr);
    auto* kh2 = buf<unsigned long long>(ctx, "ws.kh2", nr);
    uint32_t* gstart = buf<uint32_t>(ctx, "ws.gstart", nr);
    uint32_t* gexcl = buf<uint32_t>(ctx, "ws.gexcl", nr);
    sort_pairs(ctx, rh1, kh2, rec, rec2, nr);
    ws_group_starts<<<grid_for(ctx, nr), 256, 0, s>>>(rec2, nr, rh1, rh2, kseq, koff, rvox, gstart, ws.err);
    ctx->check_launch("ws_group_starts");
    PMA_CUDA(cudaMemcpyAsync(&h_err, ws.err, 4, cudaMemcpyDeviceToHost, s));
    ctx->sync();
    if (h_err & 64u) {
        PMA_CUDA(cudaMemsetAsync(ws.err, 0, 4, s));
        sort_pairs(ctx, rh2, kh2, rec, rec2, nr);
        ws_gather_h<<<grid_for(ctx, nr), 256, 0, s>>>(rh1, rec2, nr, kh);
        ctx->check_launch("ws_gather_h");
        sort_pairs(ctx, kh, kh2, rec2, rec, nr);
        PMA_CUDA(cudaMemcpyAsync(rec2, rec, nr * 4, cudaMemcpyDeviceToDevice, s));
        ws_group_starts<<<grid_for(ctx, nr), 256, 0, s>>>(rec2, nr, rh1, rh2, kseq, koff, rvox, gstart, ws.err);
        ctx->check_launch("ws_group_starts");
    }
    rec = rec2;  // records in group order from here on
    exclusive_sum(ctx, gstart, gexcl, nr);
    uint32_t last[2] = {0, 0};
    PMA_CUDA(cudaMemcpyAsync(&last[0], gexcl + nr - 1, 4, cudaMemcpyDeviceToHost, s));
    PMA_CUDA(cudaMemcpyAsync(&last[1], gstart + nr - 1, 4, cudaMemcpyDeviceToHost, s));
    PMA_CUDA(cudaMemcpyAsync(&h_err, ws.err, 4, cudaMemcpyDeviceToHost, s));
    ctx->sync();
    PMA_REQUIRE(!(h_err & 4u), PMA_ERR_INTERNAL, "pma_watershed: shared-type hash collision");
    const int64_t ngr = static_cast<int64_t>(last[0]) + last[1];
    auto* gtime = buf<unsigned long long>(ctx, "ws.gtime", ngr);
    auto* gvol = buf<unsigned long long>(ctx, "ws.gvol", ngr);
    uint32_t* grep = buf<uint32_t>(ctx, "ws.grep", ngr);
    uint32_t* final_group = buf<uint32_t>(ctx, "ws.fgroup", nsh);
    PMA_CUDA(cudaMemsetAsync(gtime, 0xFF, ngr * 8, s));
    PMA_CUDA(cudaMemsetAsync(gvol, 0, ngr * 8, s));
    ws_group_reduce<<<grid_for(ctx, nr), 256, 0, s>>>(rec, gexcl, gstart, nr, rtime, klen, koff, rvox, gtime,
                                                      gvol, grep, final_group);
    ctx->check_launch("ws_group_reduce");
    // ids in creation order (creation times are distinct), rows by ascending id
    uint32_t* d_gid = buf<uint32_t>(ctx, "ws.gid", ngr);
    type_rows(ctx, gtime, ngr, PrefixLists{grep, kseq, koff, rvox, d_pid}, gvol, d_gid, t);
    ws_shared_labels<<<grid_for(ctx, nsh), 256, 0, s>>>(sv, final_group, d_gid, nsh, labels);
    ctx->check_launch("ws_shared_labels");
    ctx->sync();
    return t;
}

void wait_selftest(pma_ctx* ctx, int* timed_out) {
    unsigned int* word = buf<unsigned int>(ctx, "ws.selftest", 2);
    PMA_CUDA(cudaMemsetAsync(word, 0, 2 * 4, ctx->stream));
    WsState ws{};
    ws.err = word + 1;
    ws.spin_limit = ctx->limits.spin_limit;
    ws_wait_selftest<<<1, 32, 0, ctx->stream>>>(ws, word);
    ctx->count_launch();
    ctx->check_launch("ws_wait_selftest");
    unsigned int h = 0;
    PMA_CUDA(cudaMemcpyAsync(&h, word + 1, 4, cudaMemcpyDeviceToHost, ctx->stream));
    ctx->sync();
    *timed_out = (h & 8u) ? 1 : 0;
}

}  // namespace pma
