// oa_sector.cuh -- the default lookup and write kernels of the open-addressing
// containers: one key per lane, its window read as whole 32-byte sectors.
//
// What bounds these operations while the table is in L2 is what a bucket window
// costs an SM: instructions and L1 requests.  A window of B slots is read here
// as the 32-byte sectors it covers, a sector a load (ld.global.v4.u64): five
// 16-byte slots are three loads, five 8-byte slots two, where one lane per slot
// took five lanes' worth of compares and shuffles.  A lane works alone, so a pass
// serves 32 keys of a warp with no shuffles, and results leave coalesced.  Keys
// whose window decides nothing are queued in shared memory and followed a full
// pass at a time, one window each, through the same code, so a pass waits on one
// window load only, whatever the load factor.  The last 32 keys of a warp leave the
// queue for good: nothing is left to fill a pass with, and a lane that walks on by
// itself waits for its windows alone (20,000 lookups of a 1.2 GB table at load 0.95:
// 35 to 18 us; 20,000 InsertOrAssigns of present keys in buckets of one slot, 24 MB:
// 12.6 to 6.1).
//
// Measured on one B200, 16 M lookups at 50% hits: 97 Gkeys/s on a 20 MB table of
// 8-byte slots (two lanes a window: 92) and 67 on an 80 MB table of 16-byte slots
// (46); 1.3 M inserts into a 20 MB table 38 Gpairs/s (slot by slot: 30).  Which
// tables and batches take these kernels is decided in oa_inst.cuh.
//
// Every loop is bounded by the probe cycle, so no kernel can spin.
#pragma once

#include "oa_kernels.cuh"

namespace b2co {

struct alignas(32) Sector {
    unsigned long long w[4];
};

// A sector, coherently (L2, never a stale L1 line) for kernels that race with
// writers, else through the read-only path.  A missed sector brings 64 bytes
// from HBM, or 128 with WIDE, where the neighbours will be wanted as well.
#ifndef B2CO_WIDE_FILL
#define B2CO_WIDE_FILL "128B"
#endif
template <bool COHERENT, bool WIDE>
__device__ __forceinline__ Sector ld_sector(void const* p)
{
    Sector v;
#define B2CO_LD_SECTOR(volatility, op, fill, clobber)                                     \
    asm volatility("ld." op ".L2::" fill ".v4.u64 {%0, %1, %2, %3}, [%4];"                \
                   : "=l"(v.w[0]), "=l"(v.w[1]), "=l"(v.w[2]), "=l"(v.w[3])               \
                   : "l"(p)                                                               \
                   clobber)
    if constexpr (COHERENT && WIDE) B2CO_LD_SECTOR(volatile, "relaxed.gpu.global", B2CO_WIDE_FILL, : "memory");
    else if constexpr (COHERENT) B2CO_LD_SECTOR(volatile, "relaxed.gpu.global", "64B", : "memory");
    else if constexpr (WIDE) B2CO_LD_SECTOR(, "global.nc", B2CO_WIDE_FILL, );
    else B2CO_LD_SECTOR(, "global.nc", "64B", );
#undef B2CO_LD_SECTOR
    return v;
}

template <class S>
__device__ __forceinline__ typename S::Raw sector_slot(Sector const& w, int i)
{
    if constexpr (S::bytes == 16) return U128{w.w[2 * i], w.w[2 * i + 1]};
    else if constexpr (S::bytes == 8) return w.w[i];
    else if constexpr (S::bytes == 4) return typename S::Raw(w.w[i / 2] >> (32 * (i % 2)));
    else return typename S::Raw(w.w[i / 4] >> (16 * (i % 4)));
}

constexpr uint32_t gcd_u32(uint32_t a, uint32_t b) { return b == 0 ? a : gcd_u32(b, a % b); }

// A bucket window of B slots as the aligned 32-byte sectors it covers.  The
// sectors may hold slots beside the window; they are masked (slot storage is a
// multiple of 32 bytes, so no load leaves it).
template <class S, int B>
struct SectorWindow {
    using Raw = typename S::Raw;
    static constexpr int N = 32 / S::bytes;                                 // slots per sector
    static constexpr uint32_t kStep = gcd_u32(uint32_t(B) * S::bytes, 32);  // window starts are multiples of this
    static constexpr int NS = int((32 - kStep + uint32_t(B) * S::bytes + 31) / 32);  // sectors that may be covered
    static_assert(NS * N <= 32, "slot mask");
    Sector s[NS];
    uint32_t off;  // the window's first slot within its first sector

    template <bool COHERENT, bool WIDE = false>
    __device__ __forceinline__ void load(Raw const* win)
    {
        uintptr_t const addr = reinterpret_cast<uintptr_t>(win);
        off = uint32_t(addr & 31) / S::bytes;
        char const* p = reinterpret_cast<char const*>(addr & ~uintptr_t(31));
#pragma unroll
        for (int i = 0; i < NS; ++i) {
            // the last sector is covered only when the window starts late enough in the first
            bool const need = i == 0 || off + B > uint32_t(i) * N;
            if (need) s[i] = ld_sector<COHERENT, WIDE>(p + 32 * i);
        }
    }
    __device__ __forceinline__ Raw slot(int j) const { return sector_slot<S>(s[j / N], j % N); }
    // First slot of the window, in scan order, that is empty or holds an equal
    // key: its place among the loaded slots (window slot + off), or -1.
    __device__ __forceinline__ int first_stop(uint64_t key, uint64_t empty_key) const
    {
        uint32_t m = 0;
#pragma unroll
        for (int j = 0; j < NS * N; ++j) {
            uint64_t const k = S::key(slot(j));
            if (k == empty_key || S::key_eq(k, key)) m |= 1u << j;
        }
        m &= ((1u << B) - 1u) << off;
        return __ffs(m) - 1;
    }
    // Slot j of the loaded ones (an unrolled select: a computed index would move
    // the window to local memory).
    __device__ __forceinline__ Raw pick(int j) const
    {
        Raw r = slot(0);
#pragma unroll
        for (int i = 1; i < NS * N; ++i)
            if (j == i) r = slot(i);
        return r;
    }
};

// A window of one slot: the slot alone, compared once and not with its sector's
// others.
template <class S>
struct SectorWindow<S, 1> {
    using Raw = typename S::Raw;
    static constexpr int NS = 1;
    Raw s;
    static constexpr uint32_t off = 0;

    template <bool COHERENT, bool WIDE = false>
    __device__ __forceinline__ void load(Raw const* win)
    {
        s = COHERENT ? ld_rw(win) : ld_ro(win);
    }
    __device__ __forceinline__ int first_stop(uint64_t key, uint64_t empty_key) const
    {
        uint64_t const k = S::key(s);
        return k == empty_key || S::key_eq(k, key) ? 0 : -1;
    }
    __device__ __forceinline__ Raw pick(int) const { return s; }
};

constexpr uint32_t kSectorRing = 64;  // queued keys per warp: a pass may add 31 + 32

// ----------------------------------------------------------------------------
// Find / Contains, with or without a stencil
// ----------------------------------------------------------------------------

#ifndef B2CO_SECTOR_FIND_MINB
#define B2CO_SECTOR_FIND_MINB(NS) ((NS) >= 3 ? 4 : 5)
#endif

template <class S, int B, bool CONTAINS, bool KEEP>
__global__ void __launch_bounds__(256, B2CO_SECTOR_FIND_MINB((SectorWindow<S, B>::NS)))
    k_find_sector(__grid_constant__ const OaArgs a, void const* keys, uint8_t const* stencil, void* out, uint32_t n)
{
    using Raw = typename S::Raw;
    constexpr uint32_t RING = kSectorRing - 1;
    __shared__ uint64_t qkey[8][kSectorRing];
    __shared__ uint32_t qinit[8][kSectorRing], qidx[8][kSectorRing], qpos[8][kSectorRing];

    uint32_t const lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t const stride = gridDim.x * blockDim.x;  // keys of one pass of the whole grid
    uint32_t base = blockIdx.x * blockDim.x + (threadIdx.x & ~31u);
    uint32_t head = 0, count = 0;  // queue state, the same on every lane
    Raw const* const slots = reinterpret_cast<Raw const*>(a.slots);

    // whether an earlier lookup has answered key i already (OaArgs::keep_misses 2)
    auto answered = [&](uint32_t i) {
        if (!KEEP || a.keep_misses < 2) return false;
        if constexpr (CONTAINS) return reinterpret_cast<uint8_t const*>(out)[i] != 0;
        else return uint64_t(reinterpret_cast<typename Io<S>::Payload const*>(out)[i]) != empty_payload<S>(a);
    };
    // the next pass's key is loaded one pass ahead
    bool next_done = base + lane < n && answered(base + lane);
    uint64_t next_key = base + lane < n ? Io<S>::load_key(keys, base + lane) : 0;
    // a key's window at slot idx; whether it decided nothing
    auto look = [&](uint64_t key, uint32_t idx, uint32_t pos) {
        SectorWindow<S, B> w;
        w.template load<false>(slots + idx);
        int const j = w.first_stop(key, a.empty_key);
        if (j < 0) return true;
        Raw const slot = w.pick(j);
        store_result<S, CONTAINS>(a, KEEP, out, pos, S::key(slot) != a.empty_key, S::value(slot));
        return false;
    };
    for (;;) {
        uint64_t key;
        uint32_t init, idx, pos;
        bool live;
        if (count >= 32 || base >= n) {
            if (base >= n && count <= 32) break;
            __syncwarp();  // the queue writes precede these reads
            uint32_t const take = count < 32 ? count : 32;
            live = lane < take;
            uint32_t const e = (head + (live ? lane : 0u)) & RING;
            key = qkey[warp][e];
            init = qinit[warp][e];
            idx = qidx[warp][e];
            pos = qpos[warp][e];
            __syncwarp();  // every read of the taken entries precedes their reuse
            head = (head + take) & RING;
            count -= take;
            idx = probe_next(idx, probe_step<S::key_bytes, B>(a.probe, key), a.probe.capacity);
            if (live && idx == init) {  // full cycle: not present
                store_result<S, CONTAINS>(a, KEEP, out, pos, false, 0);
                live = false;
            }
        } else {
            pos = base + lane;
            key = next_key;
            live = pos < n && !next_done;
            if (stencil && live && !stencil[pos]) {
                store_result<S, CONTAINS>(a, KEEP, out, pos, false, 0);
                live = false;
            }
            init = idx = probe_init<S::key_bytes, B>(a.probe, key);
            base += stride;
            next_done = base < n && base + lane < n && answered(base + lane);
            next_key = base < n && base + lane < n ? Io<S>::load_key(keys, base + lane) : 0;
        }
        bool const open = live && look(key, idx, pos);
        uint32_t const m = __ballot_sync(0xffffffffu, open);
        if (open) {
            uint32_t const e = (head + count + __popc(m & ((1u << lane) - 1u))) & RING;
            qkey[warp][e] = key;
            qinit[warp][e] = init;
            qidx[warp][e] = idx;
            qpos[warp][e] = pos;
        }
        count += __popc(m);
    }
    __syncwarp();
    if (lane < count) {  // the last keys walk on, each with its lane
        uint32_t const e = (head + lane) & RING;
        uint64_t const key = qkey[warp][e];
        uint32_t const init = qinit[warp][e], step = probe_step<S::key_bytes, B>(a.probe, key);
        uint32_t idx = qidx[warp][e];
        do {
            idx = probe_next(idx, step, a.probe.capacity);
            if (idx == init) {
                store_result<S, CONTAINS>(a, KEEP, out, qpos[warp][e], false, 0);
                break;
            }
        } while (look(key, idx, qpos[warp][e]));
    }
}

// ----------------------------------------------------------------------------
// Insert / InsertIf / InsertOrAssign, InsertAndFind (race), first-wins placement
// ----------------------------------------------------------------------------

enum { kInsPlain = 0, kInsAssign = 1, kInsIafRace = 2, kInsIafPlace = 3, kInsMark = 4, kInsMarkAssign = 5 };

// Outputs of one insert-family launch (only the mode's fields are used).
struct InsOut {
    Counters counters;   // plain/assign
    void* found;         // race: payload found or inserted
    uint8_t* inserted;   // race: 1 = this input inserted the key; mark: cleared where the key is present
    uint32_t* pos;       // place: slot of every input (kNoSlot = failed)
    uint32_t* newbits;   // place: slots claimed by this batch
    uint32_t* owner;     // place: claiming input of each claimed slot (claim_bit 0 only)
    uint32_t claim_bit;  // place: flag OR-ed into pos[] of the claiming input (0 = none)
};

// What a decided key leaves behind, by mode; one per thread.
template <class S, int MODE>
struct InsRecord {
    uint32_t failed = 0, assigned = 0, selected = 0;
    __device__ __forceinline__ void operator()(OaArgs const& a, InsOut const& o, uint32_t i, int verdict, uint32_t where,
                                               uint64_t found)
    {
        if constexpr (MODE == kInsPlain || MODE == kInsAssign) {
            // Insert succeeds only on SUCCESS (open_addressing_ref_impl.h:282-285);
            // InsertOrAssign counts a duplicate as an assignment instead.
            failed += MODE == kInsAssign ? verdict == kFailed : verdict != kSuccess;
            assigned += verdict == kDuplicate;
            ++selected;
        } else if constexpr (MODE == kInsIafRace) {
            Io<S>::store_payload(o.found, i, verdict == kFailed ? empty_payload<S>(a) : found);
            o.inserted[i] = verdict == kSuccess;
        } else if constexpr (MODE == kInsIafPlace) {
            uint32_t const p = verdict == kFailed ? kNoSlot : where;
            if (verdict == kSuccess) {
                atomicOr(o.newbits + (p >> 5), 1u << (p & 31));
                if (!o.claim_bit) o.owner[p] = i;  // tables without room for the claim bit
            }
            o.pos[i] = verdict == kSuccess ? (p | o.claim_bit) : p;
        } else {
            if (verdict == kDuplicate) o.inserted[i] = 0;
        }
    }
    __device__ __forceinline__ void finish(InsOut const& o) const  // every thread of the block
    {
        if constexpr (MODE == kInsPlain || MODE == kInsAssign) {
            if (o.counters.sum) {
                block_add_counter(o.counters.sum + kCountFailed, failed);
                if (MODE == kInsAssign) {
                    block_add_counter(o.counters.sum + kCountAssigned, assigned);
                }
                if (o.counters.host) block_add_counter(o.counters.sum + kCountSelected, selected);
                finish_counters(o.counters);
            }
        }
    }
};

enum { kOpen = 3 };  // no verdict yet: the key goes on to its next window

// Claims slot j of a window that was seen empty, or scans on from it as the
// reference does (InsertVerdict, open_addressing_ref_impl.h:489-532): a lost
// CAS goes on after that slot unless the winner holds an equal key.  Returns
// the verdict (kOpen: the window is exhausted) with the deciding slot in j and,
// for a duplicate met by a CAS, its contents in `old`.
template <class S, int B>
__device__ __forceinline__ int sector_claim(OaArgs const& a, typename S::Raw* win, uint64_t key, uint64_t val, int& j,
                                            typename S::Raw& old)
{
    using Raw = typename S::Raw;
    Raw expected = S::make(a.empty_key, a.empty_value);
    old = cas_slot(win + j, expected, insert_desired<S>(expected, key, val));
    if (raw_eq(old, expected)) return kSuccess;
    if (S::key_eq(S::key(old), key)) return kDuplicate;
    // rare: the slot was taken by another key, or is empty with another payload
    if (S::bytes < 16 || S::key(old) != a.empty_key) ++j;
    for (; j < B; ++j) {
        Raw cur = ld_rw(win + j);
        uint64_t const k = S::key(cur);
        if (S::key_eq(k, key)) {
            old = cur;
            return kDuplicate;
        }
        if (k != a.empty_key || !insert_expected<S>(a, cur, expected)) continue;
        old = cas_slot(win + j, expected, insert_desired<S>(cur, key, val));
        if (raw_eq(old, expected)) return kSuccess;
        if (S::key_eq(S::key(old), key)) return kDuplicate;
    }
    return kOpen;
}

// What an owner does with its window's first deciding slot `cur` (window slot j):
// claims it when it is empty, otherwise its key is present.  Returns the verdict,
// kOpen when the window turned out exhausted after all.
template <class S, int B, int MODE>
__device__ __forceinline__ int sector_decide(OaArgs const& a, typename S::Raw* win, int& j, typename S::Raw cur,
                                             uint64_t key, uint64_t val, uint64_t& found)
{
    bool const empty = S::key(cur) == a.empty_key;
    if constexpr (MODE == kInsMark || MODE == kInsMarkAssign) {
        if (empty) return kFailed;  // absent: nothing is written
        if constexpr (MODE == kInsMarkAssign) assign_payload<S>(win + j, key, val);
        return kDuplicate;
    } else {
        int const verdict = empty ? sector_claim<S, B>(a, win, key, val, j, cur) : int(kDuplicate);
        if (verdict == kDuplicate) {
            if constexpr (MODE == kInsAssign) assign_payload<S>(win + j, key, val);
            if constexpr (MODE == kInsIafRace) found = S::value(settle<S>(a, win + j, cur));
        } else if (verdict == kSuccess) {
            found = S::is_set ? key : val;
        }
        return verdict;
    }
}

// What became of a pair that its lane followed to the end by itself.
struct WalkEnd {
    uint64_t found;
    int verdict;
    uint32_t where;
};

// Follows a pair from the window at slot idx, which decided nothing, to the end.
template <class S, int B, int MODE>
__device__ __forceinline__ WalkEnd sector_walk(OaArgs const& a, typename S::Raw* slots, typename S::Raw pr, uint32_t init,
                                            uint32_t idx)
{
    uint32_t const step = probe_step<S::key_bytes, B>(a.probe, S::key(pr));
    WalkEnd e{0, kFailed, 0};
    for (;;) {
        idx = probe_next(idx, step, a.probe.capacity);
        if (idx == init) {  // a whole cycle: the table is full for this key
            e.verdict = kFailed;
            return e;
        }
        SectorWindow<S, B> w;
        w.template load<true>(slots + idx);
        int j = w.first_stop(S::key(pr), a.empty_key);
        if (j < 0) continue;
        typename S::Raw const cur = w.pick(j);
        j -= int(w.off);
        e.verdict = sector_decide<S, B, MODE>(a, slots + idx, j, cur, S::key(pr), S::value(pr), e.found);
        e.where = idx + uint32_t(j);
        if (e.verdict != kOpen) return e;
    }
}

template <class S, int B, int MODE>
__device__ __noinline__ WalkEnd sector_walk_call(OaArgs const& a, typename S::Raw* slots, typename S::Raw pr,
                                                 uint32_t init, uint32_t idx)
{
    return sector_walk<S, B, MODE>(a, slots, pr, init, idx);
}

// The last queued pairs of a warp, at most one a lane.  CALL: out of line, which
// costs a small batch about a microsecond.
template <class S, int B, int MODE, bool CALL>
__device__ __forceinline__ void insert_rest(OaArgs const& a, InsOut const& o, InsRecord<S, MODE>& record,
                                            typename S::Raw* slots, typename S::Raw const* qpair, uint32_t const* qinit,
                                            uint32_t const* qidx, uint32_t const* qpos, uint32_t head, uint32_t count)
{
    uint32_t const lane = threadIdx.x & 31;
    __syncwarp();  // the queue writes precede these reads
    if (lane < count) {
        uint32_t const e = (head + lane) & (kSectorRing - 1);
        WalkEnd const end = CALL ? sector_walk_call<S, B, MODE>(a, slots, qpair[e], qinit[e], qidx[e])
                                 : sector_walk<S, B, MODE>(a, slots, qpair[e], qinit[e], qidx[e]);
        record(a, o, qpos[e], end.verdict, end.where, end.found);
    }
    __syncwarp();
}

#ifndef B2CO_SECTOR_WRITE_MINB
#define B2CO_SECTOR_WRITE_MINB(NS) ((NS) >= 3 ? 4 : 5)
#endif

template <class S, int B, int MODE>
__global__ void __launch_bounds__(256, B2CO_SECTOR_WRITE_MINB((SectorWindow<S, B>::NS)))
    k_insert_sector(__grid_constant__ const OaArgs a, void const* pairs, uint8_t const* stencil, uint32_t n,
                    __grid_constant__ const InsOut o)
{
    using Raw = typename S::Raw;
    constexpr uint32_t RING = kSectorRing - 1;
    __shared__ Raw qpair[8][kSectorRing];
    __shared__ uint32_t qinit[8][kSectorRing], qidx[8][kSectorRing], qpos[8][kSectorRing];

    uint32_t const lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t const stride = gridDim.x * blockDim.x;
    uint32_t base = blockIdx.x * blockDim.x + (threadIdx.x & ~31u);
    uint32_t head = 0, count = 0;
    Raw* const slots = reinterpret_cast<Raw*>(a.slots);
    InsRecord<S, MODE> record;

    // the next pass's pair is loaded one pass ahead
    bool next_in = base + lane < n && (!stencil || stencil[base + lane]);
    Raw next_pair = next_in ? Io<S>::load_pair(pairs, base + lane) : Raw{};
    for (;;) {
        Raw pr;
        uint32_t init, idx, pos;
        bool live;
        if (count >= 32 || base >= n) {
            if (base >= n && count <= 32) break;
            __syncwarp();  // the queue writes precede these reads
            uint32_t const take = count < 32 ? count : 32;
            live = lane < take;
            uint32_t const e = (head + (live ? lane : 0u)) & RING;
            pr = qpair[warp][e];
            init = qinit[warp][e];
            idx = qidx[warp][e];
            pos = qpos[warp][e];
            __syncwarp();  // every read of the taken entries precedes their reuse
            head = (head + take) & RING;
            count -= take;
            idx = probe_next(idx, probe_step<S::key_bytes, B>(a.probe, S::key(pr)), a.probe.capacity);
            if (live && idx == init) {  // a whole cycle: the table is full for this key
                record(a, o, pos, kFailed, 0, 0);
                live = false;
            }
        } else {
            pos = base + lane;
            pr = next_pair;
            live = next_in;
            if (live && S::key(pr) == a.empty_key) {  // the empty key itself: FAILED
                record(a, o, pos, kFailed, 0, 0);
                live = false;
            }
            init = idx = probe_init<S::key_bytes, B>(a.probe, S::key(pr));
            base += stride;
            next_in = base < n && base + lane < n && (!stencil || stencil[base + lane]);
            next_pair = next_in ? Io<S>::load_pair(pairs, base + lane) : Raw{};
        }
        int verdict = kOpen;
        if (live) {
            uint64_t const key = S::key(pr);
            SectorWindow<S, B> w;
            w.template load<true>(slots + idx);
            int j = w.first_stop(key, a.empty_key);
            if (j >= 0) {
                Raw const cur = w.pick(j);
                j -= int(w.off);
                uint64_t found = 0;
                verdict = sector_decide<S, B, MODE>(a, slots + idx, j, cur, key, S::value(pr), found);
                if (verdict != kOpen) record(a, o, pos, verdict, idx + uint32_t(j), found);
            }
        }
        bool const open = live && verdict == kOpen;
        uint32_t const m = __ballot_sync(0xffffffffu, open);
        if (open) {
            uint32_t const e = (head + count + __popc(m & ((1u << lane) - 1u))) & RING;
            qpair[warp][e] = pr;
            qinit[warp][e] = init;
            qidx[warp][e] = idx;
            qpos[warp][e] = pos;
        }
        count += __popc(m);
    }
    insert_rest<S, B, MODE, false>(a, o, record, slots, qpair[warp], qinit[warp], qidx[warp], qpos[warp], head, count);
    record.finish(o);
}

}  // namespace b2co
