// group_kernels.cuh -- persistent kernels over a group of independent tables
// (thousands of StaticMaps of uneven sizes in one slab, the batched pattern of
// per-partition group-by / join builds).
//
// One launch covers every table: the items of all tables are concatenated
// (table t owns items [offsets[t], offsets[t+1])) and dealt to the warps in
// chunks of at most 512 items, so work is balanced by items, not by tables, and
// the chunks in flight at one time are neighbours: the few tables they touch
// stay in L2, and the slab crosses HBM about once.  (One contiguous span per warp
// instead keeps the whole slab in play at once, so that every window is a random
// HBM read.)  Over many rounds chunk c must not simply go to warp c % warps: warps
// drift apart, and the tables in play grow past L2 with them.  Large batches deal
// the chunks by a counter, the next one to whichever warp is free.
// 4,096 tables of 280 M int32 pairs, a 4.8 GB slab, 561 M lookups, Insert and Find
// in ms: spans and cooperative windows 16.0 and 23.6; chunks of 256 by warp number,
// one lane a key (below) 11.0 and 7.7; by the counter 6.8 and 6.3 (7.6 and 7.4 GB
// read).  Clear, Insert and Find together by chunk size: 64 items 22.4, 128 15.9,
// 256 14.0, 512 13.8, 1,024 13.5, 2,048 15.8; 512 leaves room for wider slots.
// The warp searches the table of a chunk's first item together and each lane
// walks forward from there; the table's probe parameters stay in registers
// while it does not change.  Per key the algorithms are exactly the
// single-table ones.
#pragma once

#include "oa_insert.cuh"

namespace b2co {

struct GroupTable {
    uint64_t slot_offset;  // first slot of the table in the slab
    ProbeParams probe;
};

struct GroupArgs {
    void* slots;
    GroupTable const* tables;
    uint64_t const* offsets;  // count + 1 item offsets (device)
    uint32_t count;
    uint32_t probing, hash;  // the same for every table
    uint64_t empty_key;
    uint64_t empty_value;
    unsigned int* deal;  // chunks dealt after the first of every warp; null: chunk c goes to warp c % warps
};

__device__ __forceinline__ uint64_t group_warps() { return (uint64_t(gridDim.x) * blockDim.x) >> 5; }

// The chunks of a warp, in ascending order.  The counter's answer is asked for a
// chunk ahead.
struct GroupDeal {
    uint32_t ticket = 0;
    __device__ __forceinline__ void take(GroupArgs const& g)
    {
        if (g.deal && (threadIdx.x & 31) == 0) ticket = atomicAdd(g.deal, 1u);
    }
    __device__ __forceinline__ uint64_t next(GroupArgs const& g, uint64_t begin, uint32_t chunk)
    {
        if (!g.deal) return begin + group_warps() * chunk;
        uint64_t const c = group_warps() + __shfl_sync(0xffffffffu, ticket, 0);
        take(g);
        return c * chunk;
    }
};

// The table of item i (the last t with offsets[t] <= i), searched by the whole
// warp: 32 probes a round, so 1,024 tables take two rounds and 32,768 three.
__device__ __forceinline__ uint32_t group_table_of(uint64_t const* offsets, uint32_t count, uint64_t i)
{
    uint32_t const lane = threadIdx.x & 31;
    uint32_t lo = 0, left = count;  // the answer is in [lo, lo + left); offsets[lo] <= i
    while (left > 1) {
        uint32_t const step = (left + 31) / 32, at = lane * step;
        bool const below = at < left && __ldg(offsets + lo + at) <= i;
        uint32_t const last = 31 - __clz(__ballot_sync(0xffffffffu, below) | 1u);
        lo += last * step;
        left = left - last * step < step ? left - last * step : step;
    }
    return lo;
}

template <class S>
__device__ __forceinline__ OaArgs group_table_args(GroupArgs const& g, uint32_t t)
{
    OaArgs a;
    GroupTable const& d = g.tables[t];
    a.slots = static_cast<typename S::Raw*>(g.slots) + d.slot_offset;
    a.probe = d.probe;
    a.probe.probing = g.probing;
    a.probe.hash = g.hash;
    a.empty_key = g.empty_key;
    a.empty_value = g.empty_value;
    a.erased_key = g.empty_key;
    return a;
}

// A pair that is read once: first to leave L2.
template <class T>
__device__ __forceinline__ T ld_once(T const* p)
{
    return __ldcs(p);
}
__device__ __forceinline__ U128 ld_once(U128 const* p)
{
    ulonglong2 const v = __ldcs(reinterpret_cast<ulonglong2 const*>(p));
    return U128{v.x, v.y};
}

// Items per chunk: a multiple of 32 (every kernel's pass divides it), small
// enough that a small batch still reaches every warp.
constexpr uint32_t kGroupChunk = 512;
// Items of a batch whose chunks are dealt by the counter.  37 M items: 959 us with
// and without; 280 M: 13.8 and 18.9 ms.
constexpr uint64_t kGroupDealItems = 1ull << 25;
inline uint32_t group_chunk(uint64_t n, uint64_t warps)
{
    uint64_t const share = ((n + warps - 1) / warps + 31) / 32 * 32;
    return share < kGroupChunk ? uint32_t(share ? share : 32) : kGroupChunk;
}
__device__ __forceinline__ uint64_t group_warp()
{
    return (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
}

// A lane's place in the concatenation: the table of its item, with what its
// probing needs, walked forward as the items ascend.
template <class S, int B>
struct GroupCursor {
    uint32_t t;
    uint64_t next_off;
    OaArgs a;
    __device__ __forceinline__ void start(GroupArgs const& g, uint64_t begin)  // the whole warp
    {
        t = group_table_of(g.offsets, g.count, begin);
        next_off = __ldg(g.offsets + t + 1);
        a = group_table_args<S>(g, t);
    }
    __device__ __forceinline__ void advance(GroupArgs const& g, uint64_t i)
    {
        if (i < next_off) return;
        do {
            ++t;
            next_off = __ldg(g.offsets + t + 1);
        } while (i >= next_off);
        a = group_table_args<S>(g, t);
    }
};

// One lane per key, its window read as whole sectors (oa_sector.cuh); a key whose
// window settles nothing is queued in the warp's shared-memory ring with its
// table and followed a full pass at a time, one window each.  Bound by the L2
// requests of the windows, as the single-table kernel: 89 Gkeys/s over the 4,096
// tables above.  Keys and results leave L2 first (18.7 against 19.2 ms for Clear,
// Insert and Find).  Asking L2 for the slab ahead of the chunks with bulk prefetches
// was slower (10.0 against 7.7 ms).  Five blocks an SM: 15.5 against 14.0 ms for
// all three.  Blocks of up to 256 threads.
template <class S, int B, bool CONTAINS>
__global__ void __launch_bounds__(256, 4) k_group_find_lane(__grid_constant__ const GroupArgs g, void const* keys,
                                                            void* out, uint64_t n, uint32_t chunk)
{
    using Raw = typename S::Raw;
    using Key = typename Io<S>::Key;
    constexpr uint32_t RING = kSectorRing - 1;
    __shared__ uint64_t qkey[8][kSectorRing], qpos[8][kSectorRing];
    __shared__ uint32_t qtab[8][kSectorRing], qinit[8][kSectorRing], qidx[8][kSectorRing];

    uint32_t const lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    GroupDeal deal;
    deal.take(g);
    uint64_t begin = group_warp() * chunk, at = begin, end = begin + chunk < n ? begin + chunk : n;
    Key const* const kin = static_cast<Key const*>(keys);
    uint64_t const empty = S::is_set ? g.empty_key : g.empty_value;
    uint32_t head = 0, count = 0;

    auto store = [&](uint64_t pos, bool hit, uint64_t payload) {
        if constexpr (CONTAINS) reinterpret_cast<uint8_t*>(out)[pos] = hit;
        else __stcs(reinterpret_cast<typename Io<S>::Payload*>(out) + pos, typename Io<S>::Payload(hit ? payload : empty));
    };
    GroupCursor<S, B> cur;
    uint64_t next_key = 0;
    if (begin < n) {
        cur.start(g, begin);
        next_key = at + lane < end ? uint64_t(__ldcs(kin + at + lane)) : 0;
    }
    for (;;) {
        uint64_t key, pos;
        uint32_t tab, init, idx;
        Raw const* slots;
        bool live;
        if (count >= 32 || begin >= n) {
            if (count == 0) break;
            __syncwarp();
            uint32_t const take = count < 32 ? count : 32;
            live = lane < take;
            uint32_t const e = (head + (live ? lane : 0u)) & RING;
            key = qkey[warp][e];
            pos = qpos[warp][e];
            tab = qtab[warp][e];
            init = qinit[warp][e];
            idx = qidx[warp][e];
            __syncwarp();
            head = (head + take) & RING;
            count -= take;
            OaArgs const a = group_table_args<S>(g, tab);
            slots = static_cast<Raw const*>(a.slots);
            idx = probe_next(idx, probe_step<S::key_bytes, B>(a.probe, key), a.probe.capacity);
            if (live && idx == init) {  // a whole cycle: not present
                store(pos, false, empty);
                live = false;
            }
        } else {
            pos = at + lane;
            live = pos < end;
            key = next_key;
            if (live) cur.advance(g, pos);
            tab = cur.t;
            slots = static_cast<Raw const*>(cur.a.slots);
            init = idx = probe_init<S::key_bytes, B>(cur.a.probe, key);
            at += 32;
            if (at >= end) {  // the next chunk
                begin = deal.next(g, begin, chunk);
                at = begin;
                end = begin + chunk < n ? begin + chunk : n;
                if (begin < n) cur.start(g, begin);
            }
            next_key = begin < n && at + lane < end ? uint64_t(__ldcs(kin + at + lane)) : 0;
        }
        bool open = false;
        if (live) {
            SectorWindow<S, B> w;
            w.template load<false, true>(slots + idx);
            int const j = w.first_stop(key, g.empty_key);
            if (j >= 0) {
                Raw const slot = w.pick(j);
                store(pos, S::key(slot) != g.empty_key, S::value(slot));
            } else {
                open = true;
            }
        }
        uint32_t const m = __ballot_sync(0xffffffffu, open);
        if (open) {
            uint32_t const e = (head + count + __popc(m & ((1u << lane) - 1u))) & RING;
            qkey[warp][e] = key;
            qpos[warp][e] = pos;
            qtab[warp][e] = tab;
            qinit[warp][e] = init;
            qidx[warp][e] = idx;
        }
        count += __popc(m);
    }
}

template <class S, int B, int G, bool CONTAINS>
__global__ void __launch_bounds__(256) k_group_find(__grid_constant__ const GroupArgs g, void const* keys,
                                                    void* out, uint64_t n, uint32_t chunk)
{
    uint64_t const stride = group_warps() * chunk;
    using Raw = typename S::Raw;
    constexpr int ROUNDS = (B + G - 1) / G;
    constexpr uint32_t TILES = 32 / G;
    uint32_t const lane = threadIdx.x & 31, r = lane % G, tile_lane0 = lane & ~uint32_t(G - 1), tile = lane / G;
    GroupCursor<S, B> cur;
    uint64_t end = 0;
    for (uint64_t i0 = group_warp() * chunk, begin = i0; begin < n;) {
        if (i0 == begin) {
            end = begin + chunk < n ? begin + chunk : n;
            cur.start(g, begin);
        }
        uint64_t const i = i0 + tile;
        bool const live = i < end;
        if (live) cur.advance(g, i);
        OaArgs const& a = cur.a;
        uint64_t const key = live ? uint64_t(__ldg(reinterpret_cast<typename Io<S>::Key const*>(keys) + i)) : 0;
        uint32_t const init = live ? probe_init<S::key_bytes, B>(a.probe, key) : 0;
        Raw const* slots = reinterpret_cast<Raw const*>(a.slots);
        Raw w[ROUNDS];
        if (live) {
#pragma unroll
            for (int k = 0; k < ROUNDS; ++k)
                if (int(r) + k * G < B) w[k] = ld_ro(slots + init + r + k * G);
        }
        TileResult res{0, false, !live};
        tile_resolve<S, B, G, ROUNDS>(a, w, key, r, tile_lane0, !live, res);
        if (__any_sync(0xffffffffu, !res.done)) res = tile_continue<S, B, G, ROUNDS>(a, slots, key, init, r, tile_lane0, res);
        if (r == 0 && live) {
            if constexpr (CONTAINS) reinterpret_cast<uint8_t*>(out)[i] = res.hit;
            else reinterpret_cast<typename Io<S>::Payload*>(out)[i] =
                typename Io<S>::Payload(res.hit ? res.payload : empty_payload<S>(a));
        }
        i0 += TILES;
        if (i0 >= end) i0 = begin += stride;
    }
}

// The group lookup in the single-table default's shape: G lanes share a
// window, each tile keeps Q keys in flight, and a key whose first window
// settles nothing is queued in the warp's shared-memory ring with its table
// and followed a pass at a time (a pass waits on one window load).  Each
// q-slot of a tile walks forward through the tables on its own, so a pass may
// span a table boundary.  Blocks of up to 256 threads.
template <class S, int B, int G, int Q, bool CONTAINS>
__global__ void __launch_bounds__(256) k_group_find_q(__grid_constant__ const GroupArgs g, void const* keys,
                                                    void* out, uint64_t n, uint32_t chunk)
{
    static_assert(Q <= G && G >= 2 && G <= 8, "tile shape");
    using Raw = typename S::Raw;
    constexpr int ROUNDS = (B + G - 1) / G;
    constexpr uint32_t TILES = 32 / G;
    constexpr uint32_t PASS = TILES * Q;
    static_assert(2 * PASS <= kDeferRing, "the ring must hold a pass on top of a partial one");
    constexpr uint32_t RING = kDeferRing - 1;
    __shared__ uint64_t qkey[8][kDeferRing], qpos[8][kDeferRing];
    __shared__ uint32_t qtab[8][kDeferRing], qinit[8][kDeferRing], qidx[8][kDeferRing];

    uint32_t const lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t const r = lane % G, tile_lane0 = lane & ~uint32_t(G - 1), tile = lane / G;
    uint32_t head = 0, count = 0;
    using Key = typename Io<S>::Key;
    Key const* kin = static_cast<Key const*>(keys);

    auto write = [&](uint64_t pos, bool hit, Raw const& slot, uint64_t empty) {
        if constexpr (CONTAINS) reinterpret_cast<uint8_t*>(out)[pos] = hit;
        else reinterpret_cast<typename Io<S>::Payload*>(out)[pos] = typename Io<S>::Payload(hit ? S::value(slot) : empty);
    };
    auto enqueue = [&](bool unsettled, uint64_t key, uint32_t tab, uint32_t init, uint32_t idx, uint64_t pos) {
        uint32_t const m = __ballot_sync(0xffffffffu, unsettled);
        if (unsettled) {
            uint32_t const e = (head + count + __popc(m & ((1u << lane) - 1u))) & RING;
            qkey[warp][e] = key;
            qtab[warp][e] = tab;
            qinit[warp][e] = init;
            qidx[warp][e] = idx;
            qpos[warp][e] = pos;
        }
        count += __popc(m);
    };
    uint64_t const empty = S::is_set ? g.empty_key : g.empty_value;
    auto follow = [&]() {
        __syncwarp();
        uint32_t const take = count < PASS ? count : PASS;
        uint64_t key[Q], pos[Q];
        uint32_t tab[Q], init[Q], idx[Q];
        bool live[Q];
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            uint32_t const j = q * TILES + tile;
            live[q] = j < take;
            uint32_t const e = (head + (live[q] ? j : 0u)) & RING;
            key[q] = qkey[warp][e];
            tab[q] = qtab[warp][e];
            init[q] = qinit[warp][e];
            idx[q] = qidx[warp][e];
            pos[q] = qpos[warp][e];
        }
        __syncwarp();
        head = (head + take) & RING;
        count -= take;
        Raw w[Q][ROUNDS];
        Raw const* base[Q];
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            GroupTable const& T = g.tables[live[q] ? tab[q] : 0u];
            base[q] = static_cast<Raw const*>(g.slots) + T.slot_offset;
            if (live[q]) {
                idx[q] = probe_next(idx[q], probe_step<S::key_bytes, B>(T.probe, key[q]), T.probe.capacity);
                if (idx[q] == init[q]) {  // a whole cycle: not present
                    if (r == 0) write(pos[q], false, Raw{}, empty);
                    live[q] = false;
                }
            }
            load_range<S, B, G, ROUNDS>(base[q], idx[q], 0, B, r, !live[q], w[q]);
        }
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            int own;
            Raw mine{};
            int const st = tile_first_stop<S, B, G, ROUNDS>(w[q], !live[q], key[q], g.empty_key, r, own, mine);
            if (live[q] && st != kNoStop && own == st) write(pos[q], S::key(mine) != g.empty_key, mine, empty);
            enqueue(live[q] && st == kNoStop && r == 0, key[q], tab[q], init[q], idx[q], pos[q]);
        }
    };

    uint64_t const stride = group_warps() * chunk;
    uint32_t tq[Q];
    uint64_t nextq[Q], end = 0;
    for (uint64_t i0 = group_warp() * chunk, begin = i0; begin < n;) {
        if (i0 == begin) {
            end = begin + chunk < n ? begin + chunk : n;
            tq[0] = group_table_of(g.offsets, g.count, begin);
            nextq[0] = __ldg(g.offsets + tq[0] + 1);
#pragma unroll
            for (int q = 1; q < Q; ++q) tq[q] = tq[0], nextq[q] = nextq[0];
        }
        uint64_t key[Q];
        uint32_t idx[Q];
        bool live[Q];
        uint32_t my_init = 0;
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            uint64_t const i = i0 + q * TILES + tile;
            live[q] = i < end;
            if (live[q] && i >= nextq[q]) {
                do {
                    ++tq[q];
                    nextq[q] = __ldg(g.offsets + tq[q] + 1);
                } while (i >= nextq[q]);
            }
            key[q] = live[q] ? uint64_t(__ldg(kin + i)) : 0;
            if (int(r) == q && live[q]) my_init = probe_init<S::key_bytes, B>(g.tables[tq[q]].probe, key[q]);
        }
        Raw w[Q][ROUNDS];
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            idx[q] = __shfl_sync(0xffffffffu, my_init, tile_lane0 + q);
            Raw const* base = static_cast<Raw const*>(g.slots) + g.tables[tq[q]].slot_offset;
            load_range<S, B, G, ROUNDS>(base, idx[q], 0, B, r, !live[q], w[q]);
        }
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            int own;
            Raw mine{};
            uint64_t const i = i0 + q * TILES + tile;
            int const st = tile_first_stop<S, B, G, ROUNDS>(w[q], !live[q], key[q], g.empty_key, r, own, mine);
            if (live[q] && st != kNoStop && own == st) write(i, S::key(mine) != g.empty_key, mine, empty);
            enqueue(live[q] && st == kNoStop && r == 0, key[q], tq[q], idx[q], idx[q], i);
        }
        while (count >= PASS) follow();
        i0 += PASS;
        if (i0 >= end) i0 = begin += stride;
    }
    while (count > 0) follow();
}

// Every lane learns where the first deciding slot of its window is (the slot among
// the window's sectors | 32: empty | 64: found; 0: none), the warp reading its 32
// windows a sector a lane as k_insert_tile does.
template <class S, int B>
__device__ __forceinline__ uint32_t tile_first_slot(bool live, uint64_t key, uint64_t empty_key,
                                                    typename S::Raw const* window)
{
    constexpr int G = kTileLanes<S, B>;
    constexpr uint32_t TILES = 32 / G, TM = (1u << G) - 1u, N = 32 / S::bytes;
    static_assert(SectorWindow<S, B>::NS <= G && G * N <= 32, "tile shape");
    uint32_t const lane = threadIdx.x & 31, r = lane % G, tile = lane / G;
    uint32_t const own_q = lane / TILES, own_shift = (lane % TILES) * G;  // who reads this lane's window
    uint32_t const live_mask = __ballot_sync(0xffffffffu, live);
    Sector w[G];
    uint64_t k[G];
    uint32_t valid[G];  // the slots of this lane's sector that lie in the window
#pragma unroll
    for (int q = 0; q < G; ++q) {
        uint32_t const src = q * TILES + tile;
        k[q] = S::key_bytes <= 4 ? uint64_t(__shfl_sync(0xffffffffu, uint32_t(key), src))
                                 : __shfl_sync(0xffffffffu, (unsigned long long)key, src);
        uintptr_t const addr = __shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(window), src);
        valid[q] = ((((1u << B) - 1u) << (uint32_t(addr & 31) / S::bytes)) >> (r * N)) & ((1u << N) - 1u);
        if (!((live_mask >> src) & 1u)) valid[q] = 0;
        if (valid[q]) w[q] = ld_sector<true, false>(reinterpret_cast<void const*>((addr & ~uintptr_t(31)) + r * 32));
    }
    uint32_t mine = 0;
#pragma unroll
    for (int q = 0; q < G; ++q) {
        uint32_t info = 0;
        if (valid[q]) {
            uint32_t stops = 0, empties = 0;
#pragma unroll
            for (int i = 0; i < int(N); ++i) {
                uint64_t const sk = S::key(sector_slot<S>(w[q], i));
                if (sk == empty_key) empties |= 1u << i;
                else if (S::key_eq(sk, k[q])) stops |= 1u << i;
            }
            stops = (stops | empties) & valid[q];
            if (stops) {
                uint32_t const i = uint32_t(__ffs(stops) - 1);
                info = i | (((empties >> i) & 1u) ? 96u : 64u);
            }
        }
        uint32_t const m = (__ballot_sync(0xffffffffu, info != 0) >> own_shift) & TM;
        uint32_t const first = m ? uint32_t(__ffs(m) - 1) : 0u;
        uint32_t const got = __shfl_sync(0xffffffffu, info, own_shift + first);
        if (uint32_t(q) == own_q && m) mine = got + first * N;
    }
    return mine;
}

// Insert into every table: k_insert_sector's pass with the item's own table, or with
// TILED k_insert_tile's, the window's address handed to its tile.
template <class S, int B, bool TILED>
__global__ void __launch_bounds__(256, TILED ? 3 : 4)
    k_group_insert(__grid_constant__ const GroupArgs g, void const* pairs, uint64_t n, uint32_t chunk,
                   unsigned long long* failed_counter)
{
    using Raw = typename S::Raw;
    constexpr uint32_t RING = kSectorRing - 1;
    __shared__ Raw qpair[8][kSectorRing];
    __shared__ uint32_t qtab[8][kSectorRing], qinit[8][kSectorRing], qidx[8][kSectorRing];

    uint32_t const lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    GroupDeal deal;
    deal.take(g);
    uint64_t begin = group_warp() * chunk, at = begin, end = begin + chunk < n ? begin + chunk : n;
    Raw const* const pin = static_cast<Raw const*>(pairs);
    uint32_t head = 0, count = 0, failed = 0;
    GroupCursor<S, B> cur;
    Raw next_pair{};
    if (begin < n) {
        cur.start(g, begin);
        if (at + lane < end) next_pair = ld_once(pin + at + lane);
    }
    for (;;) {
        Raw pr;
        uint32_t tab, init, idx;
        Raw* slots;
        bool live;
        if (count >= 32 || begin >= n) {
            if (count == 0) break;
            __syncwarp();
            uint32_t const take = count < 32 ? count : 32;
            live = lane < take;
            uint32_t const e = (head + (live ? lane : 0u)) & RING;
            pr = qpair[warp][e];
            tab = qtab[warp][e];
            init = qinit[warp][e];
            idx = qidx[warp][e];
            __syncwarp();
            head = (head + take) & RING;
            count -= take;
            OaArgs const a = group_table_args<S>(g, tab);
            slots = static_cast<Raw*>(a.slots);
            idx = probe_next(idx, probe_step<S::key_bytes, B>(a.probe, S::key(pr)), a.probe.capacity);
            if (live && idx == init) {  // a whole cycle: the table is full for this key
                ++failed;
                live = false;
            }
        } else {
            live = at + lane < end;
            pr = next_pair;
            if (live) cur.advance(g, at + lane);
            tab = cur.t;
            slots = static_cast<Raw*>(cur.a.slots);
            init = idx = probe_init<S::key_bytes, B>(cur.a.probe, S::key(pr));
            if (live && S::key(pr) == g.empty_key) {  // the empty key itself: FAILED
                ++failed;
                live = false;
            }
            at += 32;
            if (at >= end) {
                begin = deal.next(g, begin, chunk);
                at = begin;
                end = begin + chunk < n ? begin + chunk : n;
                if (begin < n) cur.start(g, begin);
            }
            if (begin < n && at + lane < end) next_pair = ld_once(pin + at + lane);
        }
        int verdict = kOpen;
        uint64_t const key = S::key(pr);
        // the window's first deciding slot: its place in the window, and the slot (TILED: only whether it is empty)
        int j = -1;
        Raw cur{};
        if constexpr (TILED) {
            uint32_t const at = tile_first_slot<S, B>(live, key, g.empty_key, slots + idx);
            if (live && at) {
                j = int(at & 31u) - int(uint32_t(reinterpret_cast<uintptr_t>(slots + idx) & 31) / S::bytes);
                cur = S::make((at & 32u) ? g.empty_key : ~g.empty_key, 0);
            }
        } else if (live) {
            SectorWindow<S, B> w;
            w.template load<true, true>(slots + idx);
            int const at = w.first_stop(key, g.empty_key);
            if (at >= 0) cur = w.pick(at), j = at - int(w.off);
        }
        if (j >= 0) {
            verdict = kDuplicate;
            if (S::key(cur) == g.empty_key) {
                OaArgs a{};
                a.empty_key = g.empty_key;
                a.empty_value = g.empty_value;
                verdict = sector_claim<S, B>(a, slots + idx, key, S::value(pr), j, cur);
            }
            failed += verdict == kDuplicate;
        }
        bool const open = live && verdict == kOpen;
        uint32_t const m = __ballot_sync(0xffffffffu, open);
        if (open) {
            uint32_t const e = (head + count + __popc(m & ((1u << lane) - 1u))) & RING;
            qpair[warp][e] = pr;
            qtab[warp][e] = tab;
            qinit[warp][e] = init;
            qidx[warp][e] = idx;
        }
        count += __popc(m);
    }
    if (failed_counter) block_add_counter(failed_counter, failed);
}

}  // namespace b2co
