// multi.cu -- StaticMultiset<Key> and StaticMultimap<Key, Value> (Key, Value
// int32 or int64) for B200.  The reference's containers expose no slot layout,
// so the storage here is designed for the GPU, and only the observable rules
// follow the reference (include/static_multiset.h, include/static_multimap.h,
// static_multimap_ref.h):
//
// StaticMultiset: an `ordered` array of the accepted keys in insertion order
// (RetrieveAll) plus a key -> count table (multi_common.cuh) sized for the
// capacity.  Insert ranks the valid selected keys in input order with a
// device-wide scan, keeps the first (capacity - size), appends them and adds 1
// to each key's count; every query is one table probe.
//
// StaticMultimap: a dense pair array in accepted insertion order
// (RetrieveAll) plus, built lazily at the first query after an insert, a
// grouped index: a table of the distinct keys, each with the length and the
// place of its run in a CSR array that holds every key's values ascending.
// Find is then the first value of the key's run (its minimum), Count its length
// and Retrieve a copy of the run -- no per-query sorting.
//
// The index is built by grouping first and sorting inside the groups: runs are
// short as a rule, so the values of a tile of runs are sorted in shared memory,
// where sorting all (value, key) records together takes one pass over memory per
// byte of both (16.8 M int64 pairs over 4.2 M keys: twelve passes, 4.9 ms, against 125 us
// for sorting the runs).  The pairs of large batches are grouped partition by
// partition (475 us for those pairs: survey 55, route 187, build 225), others in a
// table that all blocks share (1,700 us).
#include <algorithm>
#include <cmath>
#include <cstddef>
#include <new>

#include "multi_common.cuh"
#include "run_probe.h"

using namespace b2co;
using namespace b2co::multi;

namespace {

constexpr uint64_t kMaxElements = 1ull << 31;

cudaStream_t cs(b2co_stream s) { return reinterpret_cast<cudaStream_t>(s); }

uint64_t mask_bits(uint64_t v, uint32_t bytes) { return bytes >= 8 ? v : (v & ((1ull << (8 * bytes)) - 1)); }

// Device scratch grown on demand.
struct Scratch {
    void* p = nullptr;
    uint64_t bytes = 0;
    int reserve(uint64_t need)
    {
        if (need <= bytes) return B2CO_OK;
        if (p) cudaFree(p);
        p = nullptr;
        bytes = 0;
        cudaError_t e = cudaMalloc(&p, need);
        if (e != cudaSuccess) return cuda_fail(e, "multi-container scratch");
        bytes = need;
        return B2CO_OK;
    }
    void release()
    {
        if (p) cudaFree(p);
        p = nullptr;
        bytes = 0;
    }
    template <class T>
    T* as() const { return static_cast<T*>(p); }
};

int read_word(uint64_t const* dev, uint64_t* host_pinned, cudaStream_t s, uint64_t* out)
{
    B2CO_CUDA(cudaMemcpyAsync(host_pinned, dev, sizeof(uint64_t), cudaMemcpyDeviceToHost, s));
    B2CO_CUDA(cudaStreamSynchronize(s));
    *out = *host_pinned;
    return B2CO_OK;
}

template <class F, class A>
int apply_scanned(F f, A act, uint64_t n, uint64_t const* tile_offsets, cudaStream_t s)
{
    if (n == 0) return B2CO_OK;
    k_tile_apply<<<uint32_t((n + kTile - 1) / kTile), kThreads, 0, s>>>(f, act, n, tile_offsets);
    B2CO_CUDA(cudaGetLastError());
    return B2CO_OK;
}

// ---------------------------------------------------------------------------
// StaticMultiset
// ---------------------------------------------------------------------------

template <int KB>
struct MsetFlag {  // a valid selected key -> 1, a selected sentinel key -> 2^32
    KeyWord<KB> const* keys;
    uint8_t const* stencil;
    KeyWord<KB> empty;
    __device__ uint64_t operator()(uint64_t i) const
    {
        if (stencil && !stencil[i]) return 0;
        return keys[i] == empty ? (1ull << 32) : 1ull;
    }
};

template <int KB>
struct MsetAppend {
    KeyTable<KB> t;
    KeyWord<KB> const* keys;
    KeyWord<KB>* ordered;
    uint64_t size, accepted;
    __device__ void operator()(uint64_t i, uint64_t v, uint64_t prefix) const
    {
        if (v != 1) return;
        uint64_t const rank = prefix & 0xffffffffull;
        if (rank >= accepted) return;
        ordered[size + rank] = keys[i];
        table_add<KB>(t, keys[i], 1u);
    }
};

template <int KB>
struct MsetCount {
    KeyTable<KB> t;
    KeyWord<KB> const* keys;
    __device__ uint64_t operator()(uint64_t i) const
    {
        uint64_t const s = table_find<KB>(t, keys[i]);
        return s == ~0ull ? 0 : t.counts[s];
    }
};

template <int KB>
struct MsetRetrieve {
    KeyWord<KB> const* keys;
    KeyWord<KB>* probe_out;
    KeyWord<KB>* match_out;
    __device__ void operator()(uint64_t i, uint64_t count, uint64_t offset) const
    {
        KeyWord<KB> const k = keys[i];
        for (uint64_t j = 0; j < count; ++j) {
            probe_out[offset + j] = k;
            match_out[offset + j] = k;
        }
    }
};

// mode: 0 contains (u8), 1 find (key), 2 count each (u64), 3 count each, 0 -> 1 (u64)
template <int KB, int MODE>
__global__ void __launch_bounds__(256) k_mset_query(KeyTable<KB> t, KeyWord<KB> const* keys, uint8_t const* stencil,
                                                    void* out, uint64_t n)
{
    uint64_t const stride = uint64_t(gridDim.x) * blockDim.x;
    for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) {
        bool const sel = !stencil || stencil[i];
        KeyWord<KB> const k = keys[i];
        uint64_t c = 0;
        if (sel) {
            uint64_t const s = table_find<KB>(t, k);
            c = s == ~0ull ? 0 : t.counts[s];
        }
        if constexpr (MODE == 0) static_cast<uint8_t*>(out)[i] = c > 0;
        else if constexpr (MODE == 1) static_cast<KeyWord<KB>*>(out)[i] = c > 0 ? k : t.empty;
        else if constexpr (MODE == 2) static_cast<unsigned long long*>(out)[i] = c;
        else static_cast<unsigned long long*>(out)[i] = c ? c : 1;
    }
}

// ---------------------------------------------------------------------------
// StaticMultimap
// ---------------------------------------------------------------------------

template <int VB>
__device__ __forceinline__ unsigned long long order_bits(uint64_t v)
{
    if constexpr (VB == 4) return (v & 0xffffffffull) ^ 0x80000000ull;
    else return v ^ 0x8000000000000000ull;
}
template <int VB>
__device__ __forceinline__ uint64_t from_order_bits(unsigned long long b)
{
    if constexpr (VB == 4) return (b ^ 0x80000000ull) & 0xffffffffull;
    else return b ^ 0x8000000000000000ull;
}

template <int KB, int VB>
struct MmapSelect {
    uint8_t const* stencil;
    __device__ uint64_t operator()(uint64_t i) const { return !stencil || stencil[i] ? 1 : 0; }
};

template <int KB, int VB>
__global__ void __launch_bounds__(256) k_mmap_validate(typename SlotT<KB, VB>::Raw const* pairs, uint8_t const* stencil,
                                                       uint64_t n, uint64_t ek, uint64_t ev, unsigned int* status)
{
    using S = SlotT<KB, VB>;
    uint64_t const stride = uint64_t(gridDim.x) * blockDim.x;
    bool bad = false;
    for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) {
        if (stencil && !stencil[i]) continue;
        typename S::Raw const r = pairs[i];
        bad |= S::key(r) == ek || S::value(r) == ev;
    }
    if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicOr(status, 1u);
}

template <int KB, int VB>
struct MmapAppend {
    typename SlotT<KB, VB>::Raw const* pairs;
    typename SlotT<KB, VB>::Raw* dense;
    uint64_t size, accepted;
    __device__ void operator()(uint64_t i, uint64_t v, uint64_t rank) const
    {
        using S = SlotT<KB, VB>;
        if (!v || rank >= accepted) return;
        typename S::Raw const r = pairs[i];
        dense[size + rank] = S::make(S::key(r), S::value(r));  // padding bytes normalized
    }
};

// Insert without a stencil: pair i is the i-th accepted one, so one kernel checks
// every pair and appends the first `accepted`.  A bad pair rejects the batch by
// leaving the container's size as it was; what lies past it is never read.
// (16.8 M int64 pairs: 81 us; checking, ranking and appending in passes of their
// own read the pairs twice and took 187.)
template <int KB, int VB>
__global__ void __launch_bounds__(256) k_mmap_append(typename SlotT<KB, VB>::Raw const* pairs, uint64_t n, uint64_t ek,
                                                     uint64_t ev, typename SlotT<KB, VB>::Raw* dense, uint64_t accepted,
                                                     unsigned int* status)
{
    using S = SlotT<KB, VB>;
    uint64_t const stride = uint64_t(gridDim.x) * blockDim.x;
    bool bad = false;
    for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) {
        typename S::Raw const r = pairs[i];
        bad |= S::key(r) == ek || S::value(r) == ev;
        if (i < accepted) dense[i] = S::make(S::key(r), S::value(r));  // padding bytes normalized
    }
    if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicOr(status, 1u);
}

// ---- grouped index ---------------------------------------------------------

template <int KB>
__device__ __forceinline__ uint64_t run_hash(KeyWord<KB> k)
{
    if constexpr (KB == 4) return uint64_t(fmix32(k, 0)) << 32;
    else return fmix64(k, 0);
}

// One distinct key: its run is csr[offset, offset + count).
template <int KB>
struct alignas(16) RunSlot {
    KeyWord<KB> key;
    uint32_t count, offset;
};

// A key's probing starts at the leading bits of its hash and goes round the
// region (a power of two of slots) that it starts in: the whole table, or the
// part of it that one block builds in shared memory.  A table of full size is at
// most half full; one that was sized by an estimate, and every region that a
// block built, at most three quarters (region_crowded).
// Slots of 8-byte keys are one 16-byte word: adding to a key or asking for it
// touches one sector, not one each for key and run.  4-byte keys lie apart from
// their runs: a quarter of the bytes serve Contains, and every miss (2 M queries of
// 16.8 M distinct keys: Contains 46 us against 74, Count 77 against 90).
template <int KB>
struct RunTable {
    unsigned char* slots;  // kSlotBytes a slot
    uint64_t mask;    // table size - 1 (a power of two)
    uint64_t region;  // region size - 1
    uint32_t shift;   // 64 - log2(table size)
    KeyWord<KB> empty;

    __device__ __forceinline__ KeyWord<KB>* key(uint64_t s) const
    {
        return reinterpret_cast<KeyWord<KB>*>(slots + s * (KB == 8 ? 16 : 4));
    }
    __device__ __forceinline__ uint32_t* count(uint64_t s) const  // its offset follows
    {
        return reinterpret_cast<uint32_t*>(KB == 8 ? slots + s * 16 + 8 : slots + (mask + 1) * 4 + s * 8);
    }
    __device__ __forceinline__ void put(uint64_t s, KeyWord<KB> k, uint32_t c, uint32_t offset) const
    {
        if constexpr (KB == 8) {
            *reinterpret_cast<RunSlot<KB>*>(slots + s * 16) = RunSlot<KB>{k, c, offset};
        } else {
            *key(s) = k;
            *reinterpret_cast<uint2*>(count(s)) = make_uint2(c, offset);
        }
    }
    __device__ __forceinline__ uint64_t start(KeyWord<KB> k) const { return run_hash<KB>(k) >> shift; }
    __device__ __forceinline__ uint64_t next(uint64_t s) const { return next_in_region(s, region); }
};
template <int KB>
constexpr uint64_t kSlotBytes = KB == 8 ? 16 : 12;

// The key's slot contents; false (and count 0) when absent.  Bounded by the
// region, whatever the table holds.
template <int KB>
__device__ __forceinline__ bool find_run(RunTable<KB> const& t, KeyWord<KB> k, RunSlot<KB>& out)
{
    out.count = 0;
    if (k == t.empty) return false;
    return walk_region(uint32_t(t.start(k)), uint32_t(t.region), [&](uint32_t s) {  // at most 2^32 slots
        KeyWord<KB> found;
        uint2 run;
        if constexpr (KB == 8) {
            uint4 const v = __ldg(reinterpret_cast<uint4 const*>(t.key(s)));
            found = v.x | ((unsigned long long)v.y << 32);
            run = make_uint2(v.z, v.w);
        } else {
            found = __ldg(t.key(s));
            if (found == k) run = __ldg(reinterpret_cast<uint2 const*>(t.count(s)));
        }
        if (found == k) {
            out = RunSlot<KB>{k, run.x, run.y};
            return int(kProbeHit);
        }
        return int(found == t.empty ? kProbeMiss : kProbeOn);
    });
}

template <int KB>
__global__ void __launch_bounds__(256) k_run_clear(RunTable<KB> t)
{
    uint64_t const n = t.mask + 1, stride = uint64_t(gridDim.x) * blockDim.x;
    for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) t.put(i, t.empty, 0u, 0u);
}

// Counters of one build: runs << 32 | values, then the runs too long for the
// tile sort, then (found by the long-run sort) the runs left to the radix sort
// and their values.
struct RunCounters {
    unsigned long long cursor;
    unsigned int nlong, ngiant;
    unsigned long long giant_values;
    unsigned int crowded, pad;
};

constexpr uint32_t kNoPlace = 0xffffffffu;  // no rank in a run: runs have fewer pairs
constexpr uint32_t kMaxProbes = 128;  // of a table sized by an estimate

// Every pair joins its key's slot (a warp's pairs of one key with one atomic: 1 M pairs
// under Zipf(1.1) keys 146 us without that); place[i] = (slot, rank of the pair in its run).
// A key that finds no place within kMaxProbes slots sets *crowded: the table is
// too small for the keys, and the host builds again with a full-size one.
template <int KB, int VB>
__global__ void __launch_bounds__(256) k_run_count(RunTable<KB> t, typename SlotT<KB, VB>::Raw const* dense, uint64_t n,
                                                   uint2* place, unsigned int* crowded)
{
    using S = SlotT<KB, VB>;
    uint64_t const stride = uint64_t(gridDim.x) * blockDim.x;
    uint32_t const lane = threadIdx.x & 31;
    for (uint64_t base = uint64_t(blockIdx.x) * blockDim.x + (threadIdx.x & ~31u); base < n; base += stride) {
        uint64_t const i = base + lane;
        uint64_t s = 0;
        bool placed = false;
        if (i < n) {
            KeyWord<KB> const k = KeyWord<KB>(S::key(dense[i]));
            s = t.start(k);
            for (uint32_t probes = 0;;) {
                KeyWord<KB> cur = *t.key(s);
                if (cur == t.empty) cur = atomicCAS(t.key(s), t.empty, k);
                placed = cur == t.empty || cur == k;
                if (placed) break;
                s = t.next(s);
                if (crowded && ++probes == kMaxProbes) {
                    *crowded = 1;
                    break;
                }
            }
        }
        __syncwarp();
        // lanes of one key add together; what is not placed has a number of its own
        uint32_t const peers = __match_any_sync(0xffffffffu, placed ? (unsigned long long)s : ~(unsigned long long)lane);
        uint32_t const first = uint32_t(__ffs(peers) - 1);
        uint32_t rank = 0;
        if (placed && lane == first) rank = atomicAdd(t.count(s), uint32_t(__popc(peers)));
        rank = __shfl_sync(0xffffffffu, rank, first) + __popc(peers & ((1u << lane) - 1u));
        if (i < n) place[i] = placed ? make_uint2(uint32_t(s), rank) : make_uint2(0u, kNoPlace);
    }
}

// The first pair of every key takes its run's place: a block takes the places of
// a tile's keys with one atomic on (runs << 32 | values) -- all of them add to
// one word, so a warp's worth at a time they queue up (395 against 195 us for 16.8 M
// pairs) -- so run numbers and CSR offsets ascend together.  runs[] lists
// (offset, count) in that order.
template <int KB>
__global__ void __launch_bounds__(kThreads) k_run_offsets(RunTable<KB> t, uint2 const* place, uint64_t n,
                                                          unsigned long long* cursor, uint2* runs)
{
    __shared__ unsigned long long base_at;
    for (uint64_t base = uint64_t(blockIdx.x) * kTile; base < n; base += uint64_t(gridDim.x) * kTile) {
        uint2 p[kRounds];
        uint32_t count[kRounds];  // of a first pair's key, else 0
        uint64_t mine = 0;
#pragma unroll
        for (int r = 0; r < kRounds; ++r) {
            uint64_t const i = base + uint64_t(r) * kThreads + threadIdx.x;
            p[r] = i < n ? place[i] : make_uint2(0u, kNoPlace);
        }
#pragma unroll
        for (int r = 0; r < kRounds; ++r) {
            count[r] = p[r].y == 0 ? *t.count(p[r].x) : 0u;
            if (count[r]) mine += (1ull << 32) + count[r];
        }
        uint64_t total;
        uint64_t at = block_excl_scan(mine, &total);
        if (threadIdx.x == 0) base_at = total ? atomicAdd(cursor, (unsigned long long)total) : 0;
        __syncthreads();
        at += base_at;
#pragma unroll
        for (int r = 0; r < kRounds; ++r) {
            if (!count[r]) continue;
            t.count(p[r].x)[1] = uint32_t(at);
            runs[at >> 32] = make_uint2(uint32_t(at), count[r]);
            at += (1ull << 32) + count[r];
        }
        __syncthreads();  // base_at serves the next tile
    }
}

template <int VB>
using ValueWord = typename std::conditional<VB == 4, unsigned int, unsigned long long>::type;

template <int KB, int VB>
__global__ void __launch_bounds__(256) k_run_scatter(RunTable<KB> t, typename SlotT<KB, VB>::Raw const* dense, uint64_t n,
                                                     uint2 const* place, ValueWord<VB>* csr)
{
    using S = SlotT<KB, VB>;
    uint64_t const stride = uint64_t(gridDim.x) * blockDim.x;
    for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) {
        uint2 const p = place[i];
        if (p.y == kNoPlace) continue;
        csr[uint64_t(__ldg(t.count(p.x) + 1)) + p.y] = ValueWord<VB>(S::value(dense[i]));
    }
}

// Survey of a large batch's keys in one pass (55 us for 16.8 M pairs): an estimate of
// how many are distinct (HyperLogLog with 2^11 registers), which sizes the table,
// and the sizes of the partitions by the leading bits of the hash.
constexpr uint32_t kEstimateBits = 11, kEstimateRegs = 1u << kEstimateBits;
constexpr uint32_t kMaxPartBits = 12, kMaxParts = 1u << kMaxPartBits;

struct Survey {  // device; the host reads regs and counts
    unsigned int regs[kEstimateRegs];
    unsigned int counts[kMaxParts];
    unsigned int cursors[kMaxParts];
    unsigned int starts[kMaxParts + 1];
};

template <int KB, int VB>
__global__ void __launch_bounds__(512) k_run_survey(typename SlotT<KB, VB>::Raw const* dense, uint64_t n,
                                                    uint32_t pbits, Survey* out)
{
    using S = SlotT<KB, VB>;
    __shared__ unsigned int sk[kEstimateRegs], hist[kMaxParts];
    uint32_t const parts = 1u << pbits;
    for (uint32_t i = threadIdx.x; i < kEstimateRegs; i += blockDim.x) sk[i] = 0;
    for (uint32_t i = threadIdx.x; i < parts; i += blockDim.x) hist[i] = 0;
    __syncthreads();
    uint64_t const stride = uint64_t(gridDim.x) * blockDim.x;
    for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) {
        uint64_t const key = S::key(dense[i]);
        atomicAdd(hist + uint32_t(run_hash<KB>(KeyWord<KB>(key)) >> (64 - pbits)), 1u);
        uint64_t const h = fmix64(key, 0x2545f4914f6cdd1dull);
        uint32_t const x = uint32_t(h >> (64 - kEstimateBits));
        uint32_t const rank = uint32_t(__clzll((long long)((h << kEstimateBits) | 1ull))) + 1u;
        if (*reinterpret_cast<volatile unsigned int*>(sk + x) < rank) atomicMax(sk + x, rank);
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < kEstimateRegs; i += blockDim.x) {
        uint32_t const w = (i + blockIdx.x * 64) % kEstimateRegs;
        if (sk[w]) atomicMax(out->regs + w, sk[w]);
    }
    for (uint32_t i = threadIdx.x; i < parts; i += blockDim.x) {
        uint32_t const w = (i + blockIdx.x * 64) & (parts - 1);
        if (hist[w]) atomicAdd(out->counts + w, hist[w]);
    }
}

__global__ void __launch_bounds__(kThreads) k_part_starts(Survey* s, uint32_t parts)  // one block
{
    uint32_t const per = (parts + kThreads - 1) / kThreads, p0 = threadIdx.x * per;
    uint64_t sum = 0, total;
    for (uint32_t p = p0; p < p0 + per && p < parts; ++p) sum += s->counts[p];
    uint64_t at = block_excl_scan(sum, &total);
    for (uint32_t p = p0; p < p0 + per && p < parts; ++p) {
        s->starts[p] = s->cursors[p] = uint32_t(at);
        at += s->counts[p];
    }
    if (threadIdx.x == 0) s->starts[parts] = uint32_t(total);
}

// The pairs of a partition come to lie together, in any order: a block ranks a
// tile's pairs in their partitions in shared memory, sorts the tile by partition
// there, takes the tile's places with one atomic a partition and writes run
// after run, so that the pairs of a run leave in whole sectors.  Bound by the
// latency of shared memory within the block's phases (issue slots 22% busy): 16.8 M
// pairs of 16 bytes over 4,096 partitions, 0.49 GB in 187 us.  Storing every pair to
// its place without the sort: 274 us (scattered stores run at about 60 G a second).
constexpr int kRouteThreads = 1024, kRoutePer = 8;
constexpr uint32_t kRouteTile = kRouteThreads * kRoutePer;
template <class Raw>
constexpr size_t kRouteSmem = size_t(kRouteTile) * (sizeof(Raw) + 4) + kMaxParts * 4 * 2;

template <int KB, int VB>
__global__ void __launch_bounds__(kRouteThreads, 1)
    k_part_route(typename SlotT<KB, VB>::Raw const* dense, uint64_t n, uint32_t pbits, Survey* survey,
                 typename SlotT<KB, VB>::Raw* out)
{
    using S = SlotT<KB, VB>;
    using Raw = typename S::Raw;
    constexpr int kWarps = kRouteThreads / 32, kPer = kMaxParts / kRouteThreads;
    extern __shared__ __align__(16) unsigned char route_smem[];
    Raw* const stage = reinterpret_cast<Raw*>(route_smem);
    uint32_t* const stage_at = reinterpret_cast<uint32_t*>(stage + kRouteTile);
    uint32_t* const first = stage_at + kRouteTile;  // a partition's count, then where its run starts in the tile
    uint32_t* const delta = first + kMaxParts;      // its place in `out`, less that
    __shared__ uint32_t warp_tot[kWarps];
    uint32_t const parts = 1u << pbits, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint64_t const stride = uint64_t(gridDim.x) * kRouteTile;
    Raw pr[kRoutePer];
    auto load = [&](uint64_t base) {
#pragma unroll
        for (int r = 0; r < kRoutePer; ++r) {
            uint64_t const i = base + uint64_t(r) * kRouteThreads + threadIdx.x;
            if (i < n) pr[r] = ld_ro(dense + i);
        }
    };
    load(uint64_t(blockIdx.x) * kRouteTile);
    for (uint64_t base = uint64_t(blockIdx.x) * kRouteTile; base < n; base += stride) {
#pragma unroll
        for (int q = 0; q < kPer; ++q) first[threadIdx.x * kPer + q] = 0;
        __syncthreads();
        uint32_t place[kRoutePer];  // partition | rank in the tile's share of it
#pragma unroll
        for (int r = 0; r < kRoutePer; ++r) {
            uint64_t const i = base + uint64_t(r) * kRouteThreads + threadIdx.x;
            if (i < n) {
                uint32_t const p = uint32_t(run_hash<KB>(KeyWord<KB>(S::key(pr[r]))) >> (64 - pbits));
                place[r] = p | (atomicAdd(first + p, 1u) << kMaxPartBits);
            }
        }
        __syncthreads();
        uint32_t c[kPer], at[kPer], sum = 0;
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
            uint32_t const p = threadIdx.x * kPer + q;
            c[q] = first[p];
            at[q] = c[q] && p < parts ? atomicAdd(survey->cursors + p, c[q]) : 0u;
            sum += c[q];
        }
        uint32_t incl = sum;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            uint32_t const o = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= uint32_t(d)) incl += o;
        }
        if (lane == 31) warp_tot[warp] = incl;
        __syncthreads();
        uint32_t run = warp_tot[lane];  // every warp scans the warps' sums for itself
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            uint32_t const o = __shfl_up_sync(0xffffffffu, run, d);
            if (lane >= uint32_t(d)) run += o;
        }
        uint32_t const before = __shfl_sync(0xffffffffu, run, warp ? warp - 1 : 0);
        run = (warp ? before : 0u) + incl - sum;
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
            first[threadIdx.x * kPer + q] = run;
            delta[threadIdx.x * kPer + q] = at[q] - run;
            run += c[q];
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kRoutePer; ++r) {
            uint64_t const i = base + uint64_t(r) * kRouteThreads + threadIdx.x;
            if (i < n) {
                uint32_t const p = place[r] & (kMaxParts - 1), to = first[p] + (place[r] >> kMaxPartBits);
                stage[to] = pr[r];
                stage_at[to] = to + delta[p];
            }
        }
        load(base + stride);  // the next tile, while this one leaves
        __syncthreads();
        uint32_t const total = n - base < kRouteTile ? uint32_t(n - base) : kRouteTile;
        for (uint32_t i = threadIdx.x; i < total; i += kRouteThreads) out[stage_at[i]] = stage[i];
        __syncthreads();
    }
}

// One block builds one partition's region of the table in shared memory: it
// counts the keys, scans the counts (a warp its share of the slots), writes the
// region and the runs, and scatters the values within the partition's stretch
// of the CSR array.  Every access to memory is a stretch read or written whole, or
// lands in one that is in L2, where k_run_count, k_run_offsets and k_run_scatter
// (598, 194 and 821 us for 16.8 M int64 pairs over 4.2 M keys) pay a random access to HBM
// each.  225 us for them, 0.65 GB; bound by the probing in shared memory (L1 82% busy).
constexpr int kPartThreads = 512;
template <int KB, int VB>
__global__ void __launch_bounds__(kPartThreads)
    k_part_build(RunTable<KB> t, typename SlotT<KB, VB>::Raw const* pairs, Survey const* survey, RunCounters* ctr,
                 uint2* runs, ValueWord<VB>* csr)
{
    using S = SlotT<KB, VB>;
    constexpr int kWarps = kPartThreads / 32, kBatch = 4;
    extern __shared__ __align__(16) unsigned char region_smem[];
    __shared__ unsigned long long warp_at[kWarps];
    uint32_t const region = uint32_t(t.region), slots = region + 1;
    KeyWord<KB>* const keys = reinterpret_cast<KeyWord<KB>*>(region_smem);
    uint32_t* const counts = reinterpret_cast<uint32_t*>(keys + slots);
    uint32_t const lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t const begin = survey->starts[blockIdx.x], end = survey->starts[blockIdx.x + 1];
    for (uint32_t i = threadIdx.x; i < slots; i += kPartThreads) keys[i] = t.empty, counts[i] = 0;
    __syncthreads();
    // the slot of a key that is there or finds room; ~0 when the region is crowded
    auto slot_of = [&](KeyWord<KB> k) {
        uint32_t s = uint32_t(t.start(k)) & region;
        for (uint32_t probes = 0; probes < kMaxProbes; ++probes, s = (s + 1) & region) {
            KeyWord<KB> cur = *reinterpret_cast<KeyWord<KB> volatile*>(keys + s);
            if (cur == t.empty) cur = atomicCAS(keys + s, t.empty, k);
            if (cur == t.empty || cur == k) return s;
        }
        return ~0u;
    };
    // f(pair) for every pair of the partition, whole warps at a time
    auto each = [&](auto f) {
        for (uint64_t base = uint64_t(begin) + warp * 32; base < end; base += kBatch * kPartThreads) {
            typename S::Raw pr[kBatch];
#pragma unroll
            for (int b = 0; b < kBatch; ++b)
                if (base + b * kPartThreads + lane < end) pr[b] = ld_ro(pairs + base + b * kPartThreads + lane);
#pragma unroll
            for (int b = 0; b < kBatch; ++b) {
                if (base + b * kPartThreads + lane < end) f(pr[b]);
                __syncwarp();  // lanes that probed on longer rejoin
            }
        }
    };
    each([&](typename S::Raw const& pr) {
        uint32_t const s = slot_of(KeyWord<KB>(S::key(pr)));
        if (s == ~0u) ctr->crowded = 1;
        else atomicAdd(counts + s, 1u);
    });
    __syncthreads();
    uint32_t const share = slots / kWarps, first = warp * share;
    unsigned long long sum = 0;
    for (uint32_t i = lane; i < share; i += 32) {
        uint32_t const c = counts[first + i];
        sum += c ? (1ull << 32) + c : 0;
    }
#pragma unroll
    for (int d = 16; d; d >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
    if (lane == 0) warp_at[warp] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long total = 0;
        for (int w = 0; w < kWarps; ++w) total += warp_at[w];
        unsigned long long at = total ? atomicAdd(&ctr->cursor, total) : 0;
        if (region_crowded(total >> 32, slots)) ctr->crowded = 1;
        for (int w = 0; w < kWarps; ++w) {
            unsigned long long const v = warp_at[w];
            warp_at[w] = at;
            at += v;
        }
    }
    __syncthreads();
    unsigned long long carry = warp_at[warp];
    uint64_t const out = uint64_t(blockIdx.x) * slots;
    // 8-byte keys: with put() the compiler keeps fewer registers, and the kernel takes 266 us, not 225
    RunSlot<KB>* const out8 = reinterpret_cast<RunSlot<KB>*>(t.slots) + out;
    for (uint32_t i = lane; i < share; i += 32) {
        uint32_t const s = first + i, c = counts[s];
        unsigned long long const mine = c ? (1ull << 32) + c : 0;
        unsigned long long incl = mine;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            unsigned long long const o = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= uint32_t(d)) incl += o;
        }
        unsigned long long const at = carry + incl - mine;
        carry += __shfl_sync(0xffffffffu, incl, 31);
        if constexpr (KB == 8) out8[s] = RunSlot<KB>{keys[s], c, c ? uint32_t(at) : 0u};
        else t.put(out + s, keys[s], c, c ? uint32_t(at) : 0u);
        if (c) runs[at >> 32] = make_uint2(uint32_t(at), c);
        counts[s] = uint32_t(at);
    }
    __syncthreads();
    each([&](typename S::Raw const& pr) {
        uint32_t const s = slot_of(KeyWord<KB>(S::key(pr)));
        if (s != ~0u) csr[atomicAdd(counts + s, 1u)] = ValueWord<VB>(S::value(pr));
    });
}

// Upper end of what the registers say (standard error 2.3%, linear counting
// below): four errors above the estimate.
uint64_t estimate_distinct(unsigned int const* regs)
{
    double z = 0;
    uint32_t zeros = 0;
    for (uint32_t i = 0; i < kEstimateRegs; ++i) {
        z += std::ldexp(1.0, -int(regs[i]));
        zeros += regs[i] == 0;
    }
    double const m = kEstimateRegs;
    double e = 0.7213 / (1.0 + 1.079 / m) * m * m / z;
    if (e <= 2.5 * m && zeros) e = m * std::log(m / zeros);
    return uint64_t(1.1 * e) + 64;
}

constexpr int kRunTile = 256;            // runs per block of the tile sort, one a thread
constexpr uint32_t kRunThread = 24;      // longest run that one thread sorts (insertion, in shared memory)
constexpr uint32_t kRunTileValues = 3072;  // values of a tile that fit its shared memory
constexpr uint32_t kRunWarp = 256;       // longest run that one warp sorts (bitonic)
constexpr uint32_t kRunBlock = 4096;     // longest run that one block sorts (bitonic)

// Runs of a tile lie side by side in the CSR array: the tile's values are read
// once, sorted run by run in shared memory and written once.  Longer runs, and
// what passes the tile's shared memory, go on the list of long runs.
template <int VB>
__global__ void __launch_bounds__(kRunTile) k_run_sort_tile(RunCounters* ctr, uint2 const* runs, ValueWord<VB>* csr,
                                                            uint32_t* longs)
{
    using V = ValueWord<VB>;
    __shared__ V vals[kRunTileValues];
    uint32_t const nruns = uint32_t(ctr->cursor >> 32);
    for (uint32_t r0 = blockIdx.x * kRunTile; r0 < nruns; r0 += gridDim.x * kRunTile) {
        uint32_t const r = r0 + threadIdx.x, last = min(r0 + kRunTile, nruns) - 1;
        uint32_t const begin = runs[r0].x;
        uint32_t const total = runs[last].x + runs[last].y - begin;
        uint32_t const kept = min(total, kRunTileValues);
        for (uint32_t i = threadIdx.x; i < kept; i += kRunTile) vals[i] = V(order_bits<VB>(csr[uint64_t(begin) + i]));
        __syncthreads();
        if (r < nruns) {
            uint32_t const at = runs[r].x - begin, count = runs[r].y;
            if (count > kRunThread || at + count > kept) {
                if (count > 1) longs[atomicAdd(&ctr->nlong, 1u)] = r;
            } else {
                for (uint32_t i = 1; i < count; ++i) {
                    V const v = vals[at + i];
                    uint32_t j = i;
                    for (; j > 0 && vals[at + j - 1] > v; --j) vals[at + j] = vals[at + j - 1];
                    vals[at + j] = v;
                }
            }
        }
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < kept; i += kRunTile)
            csr[uint64_t(begin) + i] = V(from_order_bits<VB>(vals[i]));
        __syncthreads();
    }
}

// Bitonic sort of `count` values in `v` (room for `size`, the next power of
// two), by `threads` threads that `sync` joins; thread `t` of them.
template <class V, class Sync>
__device__ __forceinline__ void bitonic_sort(V* v, uint32_t size, uint32_t t, uint32_t threads, Sync sync)
{
    for (uint32_t k = 2; k <= size; k <<= 1) {
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            for (uint32_t p = t; p < size / 2; p += threads) {
                uint32_t const a = 2 * p - (p & (j - 1)), b = a + j;  // j is a power of two
                V const x = v[a], y = v[b];
                bool const up = (a & k) == 0;
                if ((x > y) == up) v[a] = y, v[b] = x;
            }
            sync();
        }
    }
}

__device__ __forceinline__ uint32_t next_pow2(uint32_t n) { return n <= 1 ? 1u : 1u << (32 - __clz(n - 1)); }

template <int VB>
__global__ void __launch_bounds__(256) k_run_sort_long(RunCounters* ctr, uint2 const* runs, ValueWord<VB>* csr,
                                                       uint32_t const* longs, uint32_t* giants)
{
    using V = ValueWord<VB>;
    __shared__ V vals[kRunBlock];  // one run of the block, or one short run of each warp
    uint32_t const nlong = ctr->nlong, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // a warp per run for the shorter ones
    for (uint32_t l = blockIdx.x * 8 + warp; l < nlong; l += gridDim.x * 8) {
        uint2 const run = runs[longs[l]];
        if (run.y > kRunWarp) continue;
        V* const v = vals + warp * kRunWarp;
        uint32_t const size = next_pow2(run.y);
        for (uint32_t i = lane; i < size; i += 32) v[i] = i < run.y ? V(order_bits<VB>(csr[uint64_t(run.x) + i])) : ~V(0);
        __syncwarp();
        bitonic_sort(v, size, lane, 32u, [] { __syncwarp(); });
        for (uint32_t i = lane; i < run.y; i += 32) csr[uint64_t(run.x) + i] = V(from_order_bits<VB>(v[i]));
        __syncwarp();
    }
    __syncthreads();
    // the block together for the others; what does not fit is counted for the radix sort
    for (uint32_t l = blockIdx.x; l < nlong; l += gridDim.x) {
        uint2 const run = runs[longs[l]];
        if (run.y <= kRunWarp) continue;
        if (run.y > kRunBlock) {
            if (threadIdx.x == 0) {
                giants[atomicAdd(&ctr->ngiant, 1u)] = longs[l];
                atomicAdd(&ctr->giant_values, (unsigned long long)run.y);
            }
            continue;
        }
        uint32_t const size = next_pow2(run.y);
        for (uint32_t i = threadIdx.x; i < size; i += blockDim.x)
            vals[i] = i < run.y ? V(order_bits<VB>(csr[uint64_t(run.x) + i])) : ~V(0);
        __syncthreads();
        bitonic_sort(vals, size, threadIdx.x, blockDim.x, [] { __syncthreads(); });
        for (uint32_t i = threadIdx.x; i < run.y; i += blockDim.x)
            csr[uint64_t(run.x) + i] = V(from_order_bits<VB>(vals[i]));
        __syncthreads();
    }
}

// Records of the giant runs: run g of the list is records[at[g], at[g + 1]), and
// back again once they are sorted by (run, value).
template <int VB, bool BACK>
__global__ void __launch_bounds__(256) k_run_giants(uint2 const* runs, uint32_t const* giants, uint64_t const* at,
                                                    uint32_t ngiant, uint64_t total, Record* rec, ValueWord<VB>* csr)
{
    using V = ValueWord<VB>;
    uint64_t const stride = uint64_t(gridDim.x) * blockDim.x;
    for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += stride) {
        uint32_t lo = 0, hi = ngiant;  // at[lo] <= i < at[hi]
        while (hi - lo > 1) {
            uint32_t const mid = (lo + hi) >> 1;
            if (at[mid] <= i) lo = mid;
            else hi = mid;
        }
        V* const v = csr + runs[giants[lo]].x + (i - at[lo]);
        if constexpr (BACK) *v = V(from_order_bits<VB>(rec[i].vbits));
        else rec[i] = Record{order_bits<VB>(*v), lo, 0u};
    }
}

struct GiantLength {
    uint2 const* runs;
    uint32_t const* giants;
    __device__ uint64_t operator()(uint64_t i) const { return runs[giants[i]].y; }
};
struct GiantOffset {
    uint64_t* at;
    __device__ void operator()(uint64_t i, uint64_t, uint64_t prefix) const { at[i] = prefix; }
};
struct HistOf {
    uint64_t* h;
    __device__ uint64_t operator()(uint64_t i) const { return h[i]; }
};
struct HistPrefix {
    uint64_t* h;
    __device__ void operator()(uint64_t i, uint64_t, uint64_t prefix) const { h[i] = prefix; }
};

// mode: 0 contains (u8), 1 find (smallest value or the empty value)
template <int KB, int VB, int MODE>
__global__ void __launch_bounds__(256) k_mmap_query(RunTable<KB> t, void const* csr, KeyWord<KB> const* keys,
                                                    uint8_t const* stencil, void* out, uint64_t n, uint64_t ev)
{
    using V = ValueWord<VB>;
    uint64_t const stride = uint64_t(gridDim.x) * blockDim.x;
    for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) {
        RunSlot<KB> run;
        bool const hit = (!stencil || stencil[i]) && find_run<KB>(t, keys[i], run);
        if constexpr (MODE == 0) static_cast<uint8_t*>(out)[i] = hit;
        else static_cast<V*>(out)[i] = hit ? static_cast<V const*>(csr)[run.offset] : V(ev);
    }
}

// A query's run length; `match`, when given, keeps its place and length for Retrieve.
template <int KB>
struct MmapCount {
    RunTable<KB> t;
    KeyWord<KB> const* keys;
    uint2* match;
    __device__ uint64_t operator()(uint64_t i) const
    {
        RunSlot<KB> run;
        bool const hit = find_run<KB>(t, keys[i], run);
        if (match) match[i] = make_uint2(hit ? run.offset : 0u, run.count);
        return run.count;
    }
};

// Copies the runs of a tile's queries to the output: the block ranks 256 queries
// at a time and its threads then take one output position each (the query found
// by a search in the block's prefixes), so writes are coalesced and a long run
// is copied by the whole block.
template <int KB, int VB>
__global__ void __launch_bounds__(kThreads) k_mmap_retrieve(KeyWord<KB> const* keys, uint2 const* match,
                                                            ValueWord<VB> const* csr, KeyWord<KB>* key_out,
                                                            ValueWord<VB>* value_out, uint64_t n,
                                                            uint64_t const* tile_offsets)
{
    __shared__ uint64_t prefix[kThreads];
    __shared__ uint32_t first[kThreads];
    __shared__ KeyWord<KB> skey[kThreads];
    uint64_t const base = uint64_t(blockIdx.x) * kTile;
    uint64_t carry = tile_offsets[blockIdx.x];
    for (int r = 0; r < kRounds; ++r) {
        uint64_t const i = base + uint64_t(r) * kThreads + threadIdx.x;
        uint2 const m = i < n ? match[i] : make_uint2(0u, 0u);
        uint64_t round_total;
        prefix[threadIdx.x] = block_excl_scan(m.y, &round_total);
        first[threadIdx.x] = m.x;
        skey[threadIdx.x] = i < n && m.y ? keys[i] : KeyWord<KB>(0);
        __syncthreads();
        for (uint64_t p = threadIdx.x; p < round_total; p += kThreads) {
            uint32_t lo = 0;  // the last query whose prefix is not above p (queries without matches share a prefix
                              // with the next one, so the last is the one that owns the position)
#pragma unroll
            for (uint32_t step = kThreads / 2; step; step >>= 1)
                if (prefix[lo + step] <= p) lo += step;
            key_out[carry + p] = skey[lo];
            value_out[carry + p] = csr[uint64_t(first[lo]) + (p - prefix[lo])];
        }
        carry += round_total;
        __syncthreads();  // the arrays are rewritten by the next round
    }
}

template <int KB, int VB>
__global__ void __launch_bounds__(256) k_mmap_export(typename SlotT<KB, VB>::Raw const* dense, uint64_t n,
                                                     KeyWord<KB>* key_out, void* value_out)
{
    using S = SlotT<KB, VB>;
    using V = typename std::conditional<VB == 4, unsigned int, unsigned long long>::type;
    uint64_t const stride = uint64_t(gridDim.x) * blockDim.x;
    for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) {
        typename S::Raw const r = dense[i];
        key_out[i] = KeyWord<KB>(S::key(r));
        static_cast<V*>(value_out)[i] = V(S::value(r));
    }
}

uint32_t blocks_for(uint64_t n) { return uint32_t(std::min<uint64_t>((n + 255) / 256, 148ull * 16)); }

}  // namespace

// ---------------------------------------------------------------------------
// containers
// ---------------------------------------------------------------------------

struct b2co_mset {
    uint64_t capacity = 0, size = 0;
    uint32_t kb = 0;
    uint64_t empty = 0;
    void* ordered = nullptr;
    void* tkeys = nullptr;
    uint32_t* tcounts = nullptr;
    uint64_t tsize = 0;
    Scratch scratch;
    uint64_t* h_word = nullptr;  // pinned

    template <int KB>
    KeyTable<KB> table() const
    {
        return KeyTable<KB>{static_cast<KeyWord<KB>*>(tkeys), tcounts, tsize - 1, KeyWord<KB>(empty)};
    }
};

struct b2co_mmap {
    uint64_t capacity = 0, size = 0;
    uint32_t kb = 0, vb = 0;
    uint64_t ek = 0, ev = 0;
    void* dense = nullptr;
    bool dirty = false;
    // grouped index
    void* tslots = nullptr;  // of a RunTable
    uint64_t tsize = 0, tslots_bytes = 0;
    void* csr = nullptr;
    uint64_t csr_cap = 0;
    Scratch scratch, build, hist, records;
    RunCounters* d_ctr = nullptr;
    RunCounters* h_ctr = nullptr;  // pinned
    uint64_t region = 0;             // slots of a probing region of the table
    Survey* d_survey = nullptr;      // made at the first build that wants one
    Survey* h_survey = nullptr;      // pinned
    unsigned int* d_status = nullptr;
    uint64_t* h_word = nullptr;

    template <int KB>
    RunTable<KB> table() const
    {
        return RunTable<KB>{static_cast<unsigned char*>(tslots), tsize - 1, region - 1,
                            uint32_t(64 - __builtin_ctzll(tsize)), KeyWord<KB>(ek)};
    }
    uint32_t slot_bytes() const { return (kb == 4 && vb == 4) ? 8 : 16; }
};

namespace {

int check_mset(b2co_mset const* s)
{
    if (!s || !s->ordered) return fail(B2CO_ELOGIC, "StaticMultiset: moved-from or destroyed object");
    return B2CO_OK;
}
int check_mmap(b2co_mmap const* m)
{
    if (!m || !m->dense) return fail(B2CO_ELOGIC, "StaticMultimap: moved-from or destroyed object");
    return B2CO_OK;
}

template <int KB>
int mset_clear(b2co_mset* s, cudaStream_t st)
{
    k_table_clear<KB><<<blocks_for(s->tsize), 256, 0, st>>>(s->table<KB>());
    B2CO_CUDA(cudaGetLastError());
    B2CO_CUDA(cudaStreamSynchronize(st));
    s->size = 0;
    return B2CO_OK;
}

template <int KB>
int mset_insert(b2co_mset* s, void const* keys, uint8_t const* stencil, uint64_t n, cudaStream_t st, uint64_t* failed)
{
    if (int e = s->scratch.reserve(scan_scratch_words(n) * 8)) return e;
    uint64_t* sc = s->scratch.as<uint64_t>();
    MsetFlag<KB> f{static_cast<KeyWord<KB> const*>(keys), stencil, KeyWord<KB>(s->empty)};
    if (int e = tile_scan(f, NoAct{}, n, sc, false, st)) return e;
    uint64_t total = 0;
    if (int e = read_word(sc + (n + kTile - 1) / kTile, s->h_word, st, &total)) return e;
    uint64_t const valid = total & 0xffffffffull, invalid = total >> 32;
    uint64_t const accepted = std::min(valid, s->capacity - s->size);
    if (accepted) {
        MsetAppend<KB> act{s->table<KB>(), static_cast<KeyWord<KB> const*>(keys),
                           static_cast<KeyWord<KB>*>(s->ordered), s->size, accepted};
        if (int e = apply_scanned(f, act, n, sc, st)) return e;
        B2CO_CUDA(cudaStreamSynchronize(st));
    }
    s->size += accepted;
    if (failed) *failed = valid - accepted + invalid;
    return B2CO_OK;
}

template <int KB, int MODE>
int mset_query(b2co_mset* s, void const* keys, uint8_t const* stencil, void* out, uint64_t n, cudaStream_t st)
{
    k_mset_query<KB, MODE><<<blocks_for(n), 256, 0, st>>>(s->table<KB>(), static_cast<KeyWord<KB> const*>(keys),
                                                           stencil, out, n);
    B2CO_CUDA(cudaGetLastError());
    B2CO_CUDA(cudaStreamSynchronize(st));
    return B2CO_OK;
}

template <int KB>
int mset_count(b2co_mset* s, void const* keys, uint64_t n, cudaStream_t st, uint64_t* total, bool retrieve,
               void* probe_out, void* match_out, uint64_t cap)
{
    if (int e = s->scratch.reserve(scan_scratch_words(n) * 8)) return e;
    uint64_t* sc = s->scratch.as<uint64_t>();
    MsetCount<KB> f{s->table<KB>(), static_cast<KeyWord<KB> const*>(keys)};
    if (int e = tile_scan(f, NoAct{}, n, sc, false, st)) return e;
    if (int e = read_word(sc + (n + kTile - 1) / kTile, s->h_word, st, total)) return e;
    if (!retrieve || *total == 0) return B2CO_OK;
    if (*total > cap) return fail(B2CO_ERANGE, "StaticMultiset: output capacity too small");
    if (!probe_out || !match_out) return fail(B2CO_EINVAL, "StaticMultiset: null output for a nonempty result");
    MsetRetrieve<KB> act{static_cast<KeyWord<KB> const*>(keys), static_cast<KeyWord<KB>*>(probe_out),
                         static_cast<KeyWord<KB>*>(match_out)};
    if (int e = apply_scanned(f, act, n, sc, st)) return e;
    B2CO_CUDA(cudaStreamSynchronize(st));
    return B2CO_OK;
}

// ---- multimap ------------------------------------------------------------------

template <int KB, int VB>
int mmap_insert(b2co_mmap* m, void const* pairs, uint8_t const* stencil, uint64_t n, cudaStream_t st,
                uint64_t* failed)
{
    using Raw = typename SlotT<KB, VB>::Raw;
    B2CO_CUDA(cudaMemsetAsync(m->d_status, 0, sizeof(unsigned int), st));
    if (!stencil) {
        uint64_t const room = std::min(n, m->capacity - m->size);
        k_mmap_append<KB, VB><<<blocks_for(n), 256, 0, st>>>(static_cast<Raw const*>(pairs), n, m->ek, m->ev,
                                                             static_cast<Raw*>(m->dense) + m->size, room, m->d_status);
        B2CO_CUDA(cudaGetLastError());
        *m->h_word = 0;
        B2CO_CUDA(cudaMemcpyAsync(m->h_word, m->d_status, sizeof(unsigned int), cudaMemcpyDeviceToHost, st));
        B2CO_CUDA(cudaStreamSynchronize(st));
        if (*m->h_word) return fail(B2CO_EINVAL, "StaticMultimap: selected input contains a reserved key or value");
        if (room) m->dirty = true;
        m->size += room;
        if (failed) *failed = n - room;
        return B2CO_OK;
    }
    k_mmap_validate<KB, VB><<<blocks_for(n), 256, 0, st>>>(static_cast<Raw const*>(pairs), stencil, n, m->ek, m->ev,
                                                           m->d_status);
    B2CO_CUDA(cudaGetLastError());
    if (int e = m->scratch.reserve(scan_scratch_words(n) * 8)) return e;
    uint64_t* sc = m->scratch.as<uint64_t>();
    MmapSelect<KB, VB> f{stencil};
    if (int e = tile_scan(f, NoAct{}, n, sc, false, st)) return e;
    unsigned int bad = 0;
    B2CO_CUDA(cudaMemcpyAsync(&bad, m->d_status, sizeof(bad), cudaMemcpyDeviceToHost, st));
    uint64_t selected = 0;
    if (int e = read_word(sc + (n + kTile - 1) / kTile, m->h_word, st, &selected)) return e;
    if (bad) return fail(B2CO_EINVAL, "StaticMultimap: selected input contains a reserved key or value");
    uint64_t const accepted = std::min(selected, m->capacity - m->size);
    if (accepted) {
        MmapAppend<KB, VB> act{static_cast<Raw const*>(pairs), static_cast<Raw*>(m->dense), m->size, accepted};
        if (int e = apply_scanned(f, act, n, sc, st)) return e;
        B2CO_CUDA(cudaStreamSynchronize(st));
        m->dirty = true;
    }
    m->size += accepted;
    if (failed) *failed = selected - accepted;
    return B2CO_OK;
}

int mmap_reserve_index(b2co_mmap* m, uint64_t tsize)
{
    uint64_t const bytes = tsize * (m->kb == 8 ? kSlotBytes<8> : kSlotBytes<4>);
    if (bytes > m->tslots_bytes) {
        cudaFree(m->tslots);
        m->tslots = nullptr;
        m->tslots_bytes = 0;
        B2CO_CUDA(cudaMalloc(&m->tslots, bytes));
        m->tslots_bytes = bytes;
    }
    m->tsize = tsize;
    if (m->size > m->csr_cap) {
        cudaFree(m->csr);
        m->csr = nullptr;
        m->csr_cap = 0;
        B2CO_CUDA(cudaMalloc(&m->csr, m->size * m->vb));
        m->csr_cap = m->size;
    }
    return B2CO_OK;
}

// Runs longer than a block sorts: a stable LSD radix sort of their values as
// (value, run) records, value bytes first, then the bytes of the run's number.
template <int VB>
int mmap_sort_giants(b2co_mmap* m, uint2 const* runs, uint32_t const* giants, uint32_t ngiant, uint64_t total,
                     cudaStream_t st)
{
    uint64_t const ntiles = (total + kSortTile - 1) / kSortTile;
    if (int e = m->records.reserve(2 * total * sizeof(Record) + (uint64_t(ngiant) + 1) * 8)) return e;
    if (int e = m->hist.reserve(256 * ntiles * 8)) return e;
    if (int e = m->scratch.reserve(scan_scratch_words(std::max(uint64_t(ngiant), 256 * ntiles)) * 8)) return e;
    Record* rec[2] = {m->records.as<Record>(), m->records.as<Record>() + total};
    uint64_t* at = reinterpret_cast<uint64_t*>(rec[1] + total);
    uint64_t* sc = m->scratch.as<uint64_t>();
    uint64_t* h = m->hist.as<uint64_t>();
    auto* csr = static_cast<ValueWord<VB>*>(m->csr);
    if (int e = tile_scan(GiantLength{runs, giants}, GiantOffset{at}, ngiant, sc, true, st)) return e;
    k_run_giants<VB, false><<<blocks_for(total), 256, 0, st>>>(runs, giants, at, ngiant, total, rec[0], csr);
    int run_bytes = 0;
    for (uint32_t v = ngiant - 1; v; v >>= 8) ++run_bytes;
    int cur = 0;
    for (int p = 0; p < VB + run_bytes; ++p) {
        k_radix_hist<<<uint32_t(ntiles), kSortThreads, 0, st>>>(rec[cur], total, p, VB, ntiles, h);
        if (int e = tile_scan(HistOf{h}, HistPrefix{h}, 256 * ntiles, sc, true, st)) return e;
        k_radix_scatter<<<uint32_t(ntiles), kSortThreads, 0, st>>>(rec[cur], rec[1 - cur], total, p, VB, ntiles, h);
        cur = 1 - cur;
    }
    k_run_giants<VB, true><<<blocks_for(total), 256, 0, st>>>(runs, giants, at, ngiant, total, rec[cur], csr);
    B2CO_CUDA(cudaGetLastError());
    return B2CO_OK;
}

// Pairs from which the keys are surveyed.  Below, the full-size table is in L2
// anyway and the survey's pass and wait (about 20 us) cost more.
constexpr uint64_t kSurveyPairs = 1ull << 20;
constexpr uint64_t kMinRegion = 512;             // slots; a larger one only for the partitions' size
constexpr uint64_t kMaxRegionBytes = 200 << 10;  // of shared memory

// The table's size, and the bits of the partition number when the index is to be
// built by partitions: when a partition's share of the table fits shared memory
// and no partition is over four times as large as they are on average (one block
// would be at work on it long after the others).  Whole builds, shared table and
// partitions, in us, n pairs over n / 4 and n / 256 int64 keys: n = 2^20: 174, 165 and 248, 243;
// 2^22: 361, 273 and 586, 554; 2^24: 1,907, 655 and 1,959, 1,736; 2^26: 10,260, 2,759 and 8,710, 6,796.
// 2,048 partitions against 4,096, over n / 4 keys: 2^22: 273 and 284; 2^24: 655 and 654 (over n: 865 and
// 797); 2^25: 1,386 and 1,233; 2^26: only the smaller ones fit.
template <int KB, int VB>
int mmap_plan(b2co_mmap* m, cudaStream_t st, uint64_t* tsize, uint32_t* part_bits)
{
    uint64_t const n = m->size;
    *tsize = table_size_for(n);
    *part_bits = 0;
    if (n < kSurveyPairs) return B2CO_OK;
    using Raw = typename SlotT<KB, VB>::Raw;
    if (!m->d_survey) {
        if (!m->h_survey) B2CO_CUDA(cudaMallocHost(reinterpret_cast<void**>(&m->h_survey), sizeof(Survey)));
        B2CO_CUDA(cudaMalloc(reinterpret_cast<void**>(&m->d_survey), sizeof(Survey)));
    }
    uint32_t const pbits = n > (1ull << 23) ? kMaxPartBits : kMaxPartBits - 1, parts = 1u << pbits;
    constexpr size_t kRead = offsetof(Survey, cursors);
    B2CO_CUDA(cudaMemsetAsync(m->d_survey, 0, kRead, st));
    k_run_survey<KB, VB><<<uint32_t(sm_count()) * 4, 512, 0, st>>>(static_cast<Raw const*>(m->dense), n, pbits,
                                                                   m->d_survey);
    B2CO_CUDA(cudaGetLastError());
    B2CO_CUDA(cudaMemcpyAsync(m->h_survey, m->d_survey, kRead, cudaMemcpyDeviceToHost, st));
    B2CO_CUDA(cudaStreamSynchronize(st));
    *tsize = std::min(*tsize, table_size_for(estimate_distinct(m->h_survey->regs)));
    uint64_t const wide = std::max(*tsize, parts * kMinRegion);
    unsigned int const* const counts = m->h_survey->counts;
    if ((wide >> pbits) * (KB + 4) <= kMaxRegionBytes &&
        uint64_t(*std::max_element(counts, counts + parts)) << pbits <= 4 * n) {
        *tsize = wide;
        *part_bits = pbits;
    }
    return B2CO_OK;
}

// The index's table, runs and unsorted values by partitions.
template <int KB, int VB>
int mmap_group_parts(b2co_mmap* m, cudaStream_t st, uint32_t pbits, void* pairs, uint2* runs)
{
    using Raw = typename SlotT<KB, VB>::Raw;
    uint32_t const parts = 1u << pbits;
    size_t const smem = size_t(m->region) * (KB + 4);
    auto* const build = k_part_build<KB, VB>;
    B2CO_CUDA(cudaFuncSetAttribute((void const*)build, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
    k_part_starts<<<1, kThreads, 0, st>>>(m->d_survey, parts);
    auto* const route = k_part_route<KB, VB>;
    B2CO_CUDA(cudaFuncSetAttribute((void const*)route, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kRouteSmem<Raw>)));
    uint64_t const tiles = (m->size + kRouteTile - 1) / kRouteTile;
    route<<<uint32_t(std::min<uint64_t>(tiles, uint64_t(sm_count()))), kRouteThreads, kRouteSmem<Raw>, st>>>(
        static_cast<Raw const*>(m->dense), m->size, pbits, m->d_survey, static_cast<Raw*>(pairs));
    build<<<parts, kPartThreads, smem, st>>>(m->table<KB>(), static_cast<Raw const*>(pairs), m->d_survey, m->d_ctr, runs,
                                             static_cast<ValueWord<VB>*>(m->csr));
    B2CO_CUDA(cudaGetLastError());
    return B2CO_OK;
}

// The same with random accesses to the whole table.  `place` has room for n places.
template <int KB, int VB>
int mmap_group_table(b2co_mmap* m, cudaStream_t st, uint2* place, uint2* runs, bool full)
{
    using Raw = typename SlotT<KB, VB>::Raw;
    auto const* dense = static_cast<Raw const*>(m->dense);
    uint64_t const n = m->size;
    RunTable<KB> const t = m->table<KB>();
    k_run_clear<KB><<<blocks_for(m->tsize), 256, 0, st>>>(t);
    if (n == 0) return B2CO_OK;
    k_run_count<KB, VB><<<blocks_for(n), 256, 0, st>>>(t, dense, n, place, full ? nullptr : &m->d_ctr->crowded);
    k_run_offsets<KB><<<uint32_t(std::min<uint64_t>((n + kTile - 1) / kTile, 148ull * 8)), kThreads, 0, st>>>(
        t, place, n, &m->d_ctr->cursor, runs);
    k_run_scatter<KB, VB><<<blocks_for(n), 256, 0, st>>>(t, dense, n, place, static_cast<ValueWord<VB>*>(m->csr));
    B2CO_CUDA(cudaGetLastError());
    return B2CO_OK;
}

// Builds the grouped index of the stored pairs: the table of distinct keys with
// their runs, and the values of every run ascending.
template <int KB, int VB>
int mmap_build(b2co_mmap* m, cudaStream_t st)
{
    if (!m->dirty) return B2CO_OK;
    using Raw = typename SlotT<KB, VB>::Raw;
    uint64_t const n = m->size, full = table_size_for(n);
    uint64_t tsize = 0;
    uint32_t pbits = 0;
    if (int e = mmap_plan<KB, VB>(m, st, &tsize, &pbits)) return e;
    // a table that turns out too small is built again, full-size and as a whole
    for (;; tsize = full, pbits = 0) {
        if (int e = mmap_reserve_index(m, tsize)) return e;
        m->region = tsize >> pbits;
        // runs[n] (a key may have one pair only), long runs (of two values or more), giants, and
        // the partitioned pairs or the pairs' places
        uint64_t const nlong = n / 2 + 1, ngiant = n / kRunBlock + 1;
        uint64_t const lists = n * 8 + (nlong + ngiant) * 4 + 8;
        if (pbits && m->build.reserve(n * sizeof(Raw) + lists)) {
            cudaGetLastError();  // no room for the partitioned pairs
            pbits = 0;
            m->region = tsize;
        }
        if (int e = m->build.reserve(n * (pbits ? sizeof(Raw) : sizeof(uint2)) + lists)) return e;
        auto* const work = m->build.as<unsigned char>();
        uint2* const runs = reinterpret_cast<uint2*>(work + n * (pbits ? sizeof(Raw) : sizeof(uint2)));
        uint32_t* const longs = reinterpret_cast<uint32_t*>(runs + n);
        uint32_t* const giants = longs + nlong;
        B2CO_CUDA(cudaMemsetAsync(m->d_ctr, 0, sizeof(RunCounters), st));
        if (int e = pbits ? mmap_group_parts<KB, VB>(m, st, pbits, work, runs)
                          : mmap_group_table<KB, VB>(m, st, reinterpret_cast<uint2*>(work), runs, tsize == full))
            return e;
        if (n == 0) {  // an empty table answers every query with a miss
            B2CO_CUDA(cudaStreamSynchronize(st));
            break;
        }
        auto* csr = static_cast<ValueWord<VB>*>(m->csr);
        k_run_sort_tile<VB><<<blocks_for(n), kRunTile, 0, st>>>(m->d_ctr, runs, csr, longs);
        k_run_sort_long<VB><<<uint32_t(std::min<uint64_t>((nlong + 7) / 8, 148 * 4)), 256, 0, st>>>(
            m->d_ctr, runs, csr, longs, giants);
        B2CO_CUDA(cudaGetLastError());
        B2CO_CUDA(cudaMemcpyAsync(m->h_ctr, m->d_ctr, sizeof(RunCounters), cudaMemcpyDeviceToHost, st));
        B2CO_CUDA(cudaStreamSynchronize(st));
        if (m->h_ctr->crowded) continue;
        // a table of full size holds every key that there can be; a smaller one may have been filled up
        if (tsize != full && region_crowded(m->h_ctr->cursor >> 32, tsize)) continue;
        if (m->h_ctr->ngiant) {
            if (int e = mmap_sort_giants<VB>(m, runs, giants, m->h_ctr->ngiant, m->h_ctr->giant_values, st)) return e;
            B2CO_CUDA(cudaStreamSynchronize(st));
        }
        break;
    }
    m->dirty = false;
    return B2CO_OK;
}

template <int KB, int VB, int MODE>
int mmap_query(b2co_mmap* m, void const* keys, uint8_t const* stencil, void* out, uint64_t n, cudaStream_t st)
{
    if (int e = mmap_build<KB, VB>(m, st)) return e;
    k_mmap_query<KB, VB, MODE><<<blocks_for(n), 256, 0, st>>>(m->table<KB>(), m->csr,
                                                               static_cast<KeyWord<KB> const*>(keys), stencil, out, n,
                                                               m->ev);
    B2CO_CUDA(cudaGetLastError());
    B2CO_CUDA(cudaStreamSynchronize(st));
    return B2CO_OK;
}

}  // namespace

// ---------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------

namespace {

template <class F>
int by_kb(uint32_t kb, F f)
{
    return kb == 4 ? f(std::integral_constant<int, 4>{}) : f(std::integral_constant<int, 8>{});
}
template <class F>
int by_kv(uint32_t kb, uint32_t vb, F f)
{
    if (kb == 4) return vb == 4 ? f(std::integral_constant<int, 4>{}, std::integral_constant<int, 4>{})
                                : f(std::integral_constant<int, 4>{}, std::integral_constant<int, 8>{});
    return vb == 4 ? f(std::integral_constant<int, 8>{}, std::integral_constant<int, 4>{})
                   : f(std::integral_constant<int, 8>{}, std::integral_constant<int, 8>{});
}

int check_batch(uint64_t n)
{
    if (n > kMaxBatch) return fail(B2CO_ERANGE, "batch exceeds the 32-bit index range");
    return B2CO_OK;
}

int mset_query_any(b2co_mset* s, void const* keys, uint8_t const* stencil, bool use_stencil, void* out, uint64_t n,
                   b2co_stream st, int mode)
{
    if (int e = check_mset(s)) return e;
    if (n == 0) return B2CO_OK;
    if (!keys || !out) return fail(B2CO_EINVAL, "StaticMultiset: null nonempty buffer");
    if (use_stencil && !stencil) return fail(B2CO_EINVAL, "StaticMultiset: null stencil");
    if (int e = check_batch(n)) return e;
    return by_kb(s->kb, [&](auto k) {
        constexpr int KB = decltype(k)::value;
        switch (mode) {
            case 0: return mset_query<KB, 0>(s, keys, stencil, out, n, cs(st));
            case 1: return mset_query<KB, 1>(s, keys, stencil, out, n, cs(st));
            case 2: return mset_query<KB, 2>(s, keys, stencil, out, n, cs(st));
            default: return mset_query<KB, 3>(s, keys, stencil, out, n, cs(st));
        }
    });
}

int mmap_query_any(b2co_mmap* m, void const* keys, uint8_t const* stencil, bool use_stencil, void* out, uint64_t n,
                   b2co_stream st, int mode)
{
    if (int e = check_mmap(m)) return e;
    if (n == 0) return B2CO_OK;
    if (!keys || !out) return fail(B2CO_EINVAL, "StaticMultimap: null nonempty buffer");
    if (use_stencil && !stencil) return fail(B2CO_EINVAL, "StaticMultimap: null stencil");
    if (int e = check_batch(n)) return e;
    return by_kv(m->kb, m->vb, [&](auto k, auto v) {
        constexpr int KB = decltype(k)::value, VB = decltype(v)::value;
        return mode == 0 ? mmap_query<KB, VB, 0>(m, keys, stencil, out, n, cs(st))
                         : mmap_query<KB, VB, 1>(m, keys, stencil, out, n, cs(st));
    });
}

// The reference's Count / Retrieve guards (static_multimap.h:258-270 CheckCount
// with detail/static_multimap/storage.h:29-35 Bytes; static_multiset.h CountImpl):
// the query array's byte size and n * Size() must be representable.
int count_guard(uint64_t n, uint64_t size, uint32_t key_bytes)
{
    if (n > ~0ull / key_bytes) return fail(B2CO_EOVERFLOW, "buffer byte size overflow");
    if (size && n > ~0ull / size) return fail(B2CO_EOVERFLOW, "potential total count overflow");
    return B2CO_OK;
}

}  // namespace

extern "C" {

// ---- StaticMultiset ---------------------------------------------------------------

int b2co_mset_create(uint64_t capacity, uint32_t key_bytes, uint64_t empty_key_bits, b2co_stream stream,
                     b2co_mset** out)
{
    if (!out) return fail(B2CO_EINVAL, "null output");
    *out = nullptr;
    if (capacity == 0) return fail(B2CO_EINVAL, "StaticMultiset: capacity must be positive");
    if (capacity > kMaxElements) return fail(B2CO_EINVAL, "StaticMultiset: capacity above 2^31");
    if (key_bytes != 4 && key_bytes != 8) return fail(B2CO_EINVAL, "StaticMultiset: keys are 4 or 8 bytes");
    auto* s = new (std::nothrow) b2co_mset;
    if (!s) return fail(B2CO_ENOMEM, "host allocation failed");
    s->capacity = capacity;
    s->kb = key_bytes;
    s->empty = mask_bits(empty_key_bits, key_bytes);
    s->tsize = table_size_for(capacity);
    cudaError_t e = cudaMalloc(&s->ordered, capacity * key_bytes);
    if (e == cudaSuccess) e = cudaMalloc(&s->tkeys, s->tsize * key_bytes);
    if (e == cudaSuccess) e = cudaMalloc(reinterpret_cast<void**>(&s->tcounts), s->tsize * 4);
    if (e == cudaSuccess) e = cudaMallocHost(reinterpret_cast<void**>(&s->h_word), sizeof(uint64_t));
    if (e != cudaSuccess) {
        b2co_mset_destroy(s);
        return e == cudaErrorMemoryAllocation ? fail(B2CO_ENOMEM, "StaticMultiset allocation") : cuda_fail(e, "StaticMultiset");
    }
    if (int st = b2co_mset_clear(s, stream)) {
        b2co_mset_destroy(s);
        return st;
    }
    *out = s;
    return B2CO_OK;
}

int b2co_mset_destroy(b2co_mset* s)
{
    if (!s) return B2CO_OK;
    cudaFree(s->ordered);
    cudaFree(s->tkeys);
    cudaFree(s->tcounts);
    if (s->h_word) cudaFreeHost(s->h_word);
    s->scratch.release();
    delete s;
    return B2CO_OK;
}

int b2co_mset_capacity(b2co_mset const* s, uint64_t* c)
{
    if (int e = check_mset(s)) return e;
    if (!c) return fail(B2CO_EINVAL, "null output");
    *c = s->capacity;
    return B2CO_OK;
}

int b2co_mset_size(b2co_mset const* s, uint64_t* n)
{
    if (int e = check_mset(s)) return e;
    if (!n) return fail(B2CO_EINVAL, "null output");
    *n = s->size;
    return B2CO_OK;
}

int b2co_mset_clear(b2co_mset* s, b2co_stream st)
{
    if (int e = check_mset(s)) return e;
    return by_kb(s->kb, [&](auto k) { return mset_clear<decltype(k)::value>(s, cs(st)); });
}

static int mset_insert_any(b2co_mset* s, void const* keys, uint8_t const* stencil, bool use_stencil, uint64_t n,
                           b2co_stream st, uint64_t* failed)
{
    if (int e = check_mset(s)) return e;
    if (failed) *failed = 0;
    if (n == 0) return B2CO_OK;
    if (use_stencil && !stencil) return fail(B2CO_EINVAL, "StaticMultiset::InsertIf: null stencil");
    if (!keys) {  // static_multiset.h:161: a null key array reports every key failed
        if (failed) *failed = n;
        return B2CO_OK;
    }
    if (int e = check_batch(n)) return e;
    return by_kb(s->kb, [&](auto k) { return mset_insert<decltype(k)::value>(s, keys, stencil, n, cs(st), failed); });
}

int b2co_mset_insert(b2co_mset* s, void const* keys, uint64_t n, b2co_stream st, uint64_t* failed)
{
    return mset_insert_any(s, keys, nullptr, false, n, st, failed);
}

int b2co_mset_insert_if(b2co_mset* s, void const* keys, uint8_t const* stencil, uint64_t n, b2co_stream st,
                        uint64_t* failed)
{
    return mset_insert_any(s, keys, stencil, true, n, st, failed);
}

int b2co_mset_contains(b2co_mset* s, void const* keys, uint8_t* out, uint64_t n, b2co_stream st)
{
    return mset_query_any(s, keys, nullptr, false, out, n, st, 0);
}
int b2co_mset_contains_if(b2co_mset* s, void const* keys, uint8_t const* stencil, uint8_t* out, uint64_t n,
                          b2co_stream st)
{
    return mset_query_any(s, keys, stencil, true, out, n, st, 0);
}
int b2co_mset_find(b2co_mset* s, void const* keys, void* out, uint64_t n, b2co_stream st)
{
    return mset_query_any(s, keys, nullptr, false, out, n, st, 1);
}
int b2co_mset_find_if(b2co_mset* s, void const* keys, uint8_t const* stencil, void* out, uint64_t n, b2co_stream st)
{
    return mset_query_any(s, keys, stencil, true, out, n, st, 1);
}
int b2co_mset_count_each(b2co_mset* s, void const* keys, uint64_t* out, uint64_t n, b2co_stream st)
{
    return mset_query_any(s, keys, nullptr, false, out, n, st, 2);
}
int b2co_mset_count_each_outer(b2co_mset* s, void const* keys, uint64_t* out, uint64_t n, b2co_stream st)
{
    return mset_query_any(s, keys, nullptr, false, out, n, st, 3);
}

int b2co_mset_count(b2co_mset* s, void const* keys, uint64_t n, b2co_stream st, uint64_t* total)
{
    if (int e = check_mset(s)) return e;
    if (!total) return fail(B2CO_EINVAL, "null output");
    *total = 0;
    if (n == 0) return B2CO_OK;
    if (!keys) return fail(B2CO_EINVAL, "StaticMultiset: null nonempty buffer");
    if (int e = count_guard(n, s->size, s->kb)) return e;
    if (int e = check_batch(n)) return e;
    return by_kb(s->kb, [&](auto k) {
        return mset_count<decltype(k)::value>(s, keys, n, cs(st), total, false, nullptr, nullptr, 0);
    });
}

int b2co_mset_retrieve(b2co_mset* s, void const* keys, uint64_t n, void* probe_out, void* match_out,
                       uint64_t cap, b2co_stream st, uint64_t* written)
{
    if (int e = check_mset(s)) return e;
    if (!written) return fail(B2CO_EINVAL, "null output");
    *written = 0;
    if (n == 0) return B2CO_OK;
    if (!keys) return fail(B2CO_EINVAL, "StaticMultiset: null nonempty buffer");
    if (int e = count_guard(n, s->size, s->kb)) return e;
    if (int e = check_batch(n)) return e;
    uint64_t total = 0;
    int r = by_kb(s->kb, [&](auto k) {
        return mset_count<decltype(k)::value>(s, keys, n, cs(st), &total, true, probe_out, match_out, cap);
    });
    if (!r) *written = total;
    return r;
}

int b2co_mset_retrieve_all(b2co_mset* s, void* out, uint64_t cap, b2co_stream st, uint64_t* written)
{
    if (int e = check_mset(s)) return e;
    if (!written) return fail(B2CO_EINVAL, "null output");
    *written = 0;
    if (s->size > cap) return fail(B2CO_ERANGE, "StaticMultiset: output capacity too small");
    if (!s->size) return B2CO_OK;
    if (!out) return fail(B2CO_EINVAL, "StaticMultiset: null nonempty buffer");
    B2CO_CUDA(cudaMemcpyAsync(out, s->ordered, s->size * s->kb, cudaMemcpyDeviceToDevice, cs(st)));
    B2CO_CUDA(cudaStreamSynchronize(cs(st)));
    *written = s->size;
    return B2CO_OK;
}

// ---- StaticMultimap ---------------------------------------------------------------

int b2co_mmap_create(uint64_t capacity, uint32_t key_bytes, uint32_t value_bytes, uint64_t ek, uint64_t ev,
                     b2co_stream stream, b2co_mmap** out)
{
    if (!out) return fail(B2CO_EINVAL, "null output");
    *out = nullptr;
    if (capacity == 0) return fail(B2CO_EINVAL, "StaticMultimap: capacity must be positive");
    if (capacity > kMaxElements) return fail(B2CO_EINVAL, "StaticMultimap: capacity above 2^31");
    if ((key_bytes != 4 && key_bytes != 8) || (value_bytes != 4 && value_bytes != 8))
        return fail(B2CO_EINVAL, "StaticMultimap: keys and values are 4 or 8 bytes");
    auto* m = new (std::nothrow) b2co_mmap;
    if (!m) return fail(B2CO_ENOMEM, "host allocation failed");
    m->capacity = capacity;
    m->kb = key_bytes;
    m->vb = value_bytes;
    m->ek = mask_bits(ek, key_bytes);
    m->ev = mask_bits(ev, value_bytes);
    cudaError_t e = cudaMalloc(&m->dense, capacity * m->slot_bytes());
    if (e == cudaSuccess) e = cudaMalloc(reinterpret_cast<void**>(&m->d_status), sizeof(unsigned int));
    if (e == cudaSuccess) e = cudaMalloc(reinterpret_cast<void**>(&m->d_ctr), sizeof(RunCounters));
    if (e == cudaSuccess) e = cudaMallocHost(reinterpret_cast<void**>(&m->h_word), sizeof(uint64_t));
    if (e == cudaSuccess) e = cudaMallocHost(reinterpret_cast<void**>(&m->h_ctr), sizeof(RunCounters));
    if (e != cudaSuccess) {
        b2co_mmap_destroy(m);
        return e == cudaErrorMemoryAllocation ? fail(B2CO_ENOMEM, "StaticMultimap allocation") : cuda_fail(e, "StaticMultimap");
    }
    if (int st = b2co_mmap_clear(m, stream)) {
        b2co_mmap_destroy(m);
        return st;
    }
    *out = m;
    return B2CO_OK;
}

int b2co_mmap_destroy(b2co_mmap* m)
{
    if (!m) return B2CO_OK;
    cudaFree(m->dense);
    cudaFree(m->tslots);
    cudaFree(m->csr);
    cudaFree(m->d_status);
    cudaFree(m->d_ctr);
    if (m->h_word) cudaFreeHost(m->h_word);
    if (m->h_ctr) cudaFreeHost(m->h_ctr);
    cudaFree(m->d_survey);
    if (m->h_survey) cudaFreeHost(m->h_survey);
    m->scratch.release();
    m->build.release();
    m->hist.release();
    m->records.release();
    delete m;
    return B2CO_OK;
}

int b2co_mmap_capacity(b2co_mmap const* m, uint64_t* c)
{
    if (int e = check_mmap(m)) return e;
    if (!c) return fail(B2CO_EINVAL, "null output");
    *c = m->capacity;
    return B2CO_OK;
}

int b2co_mmap_size(b2co_mmap const* m, uint64_t* n)
{
    if (int e = check_mmap(m)) return e;
    if (!n) return fail(B2CO_EINVAL, "null output");
    *n = m->size;
    return B2CO_OK;
}

int b2co_mmap_clear(b2co_mmap* m, b2co_stream)
{
    if (int e = check_mmap(m)) return e;
    m->size = 0;
    m->dirty = true;  // the next query builds an empty index
    return B2CO_OK;
}

static int mmap_insert_any(b2co_mmap* m, void const* pairs, uint8_t const* stencil, bool use_stencil, uint64_t n,
                           b2co_stream st, uint64_t* failed)
{
    if (int e = check_mmap(m)) return e;
    if (failed) *failed = 0;
    if (n == 0) return B2CO_OK;
    if (!pairs) return fail(B2CO_EINVAL, "StaticMultimap: null nonempty buffer");
    if (use_stencil && !stencil) return fail(B2CO_EINVAL, "StaticMultimap: null nonempty buffer");
    if (int e = check_batch(n)) return e;
    return by_kv(m->kb, m->vb, [&](auto k, auto v) {
        return mmap_insert<decltype(k)::value, decltype(v)::value>(m, pairs, stencil, n, cs(st), failed);
    });
}

int b2co_mmap_insert(b2co_mmap* m, void const* pairs, uint64_t n, b2co_stream st, uint64_t* failed)
{
    return mmap_insert_any(m, pairs, nullptr, false, n, st, failed);
}

int b2co_mmap_insert_if(b2co_mmap* m, void const* pairs, uint8_t const* stencil, uint64_t n, b2co_stream st,
                        uint64_t* failed)
{
    return mmap_insert_any(m, pairs, stencil, true, n, st, failed);
}

int b2co_mmap_contains(b2co_mmap* m, void const* keys, uint8_t* out, uint64_t n, b2co_stream st)
{
    return mmap_query_any(m, keys, nullptr, false, out, n, st, 0);
}
int b2co_mmap_contains_if(b2co_mmap* m, void const* keys, uint8_t const* stencil, uint8_t* out, uint64_t n,
                          b2co_stream st)
{
    return mmap_query_any(m, keys, stencil, true, out, n, st, 0);
}
int b2co_mmap_find(b2co_mmap* m, void const* keys, void* out, uint64_t n, b2co_stream st)
{
    return mmap_query_any(m, keys, nullptr, false, out, n, st, 1);
}
int b2co_mmap_find_if(b2co_mmap* m, void const* keys, uint8_t const* stencil, void* out, uint64_t n, b2co_stream st)
{
    return mmap_query_any(m, keys, stencil, true, out, n, st, 1);
}

static int mmap_count_any(b2co_mmap* m, void const* keys, uint64_t n, b2co_stream st, uint64_t* total, bool retrieve,
                          void* key_out, void* value_out, uint64_t cap)
{
    if (int e = check_mmap(m)) return e;
    *total = 0;
    if (n == 0) return B2CO_OK;
    if (!keys) return fail(B2CO_EINVAL, "StaticMultimap: null nonempty buffer");
    if (int e = count_guard(n, m->size, m->kb)) return e;
    if (int e = check_batch(n)) return e;
    return by_kv(m->kb, m->vb, [&](auto k, auto v) -> int {
        constexpr int KB = decltype(k)::value, VB = decltype(v)::value;
        cudaStream_t s = cs(st);
        if (int e = mmap_build<KB, VB>(m, s)) return e;
        uint64_t const words = scan_scratch_words(n);
        if (int e = m->scratch.reserve((words + (retrieve ? n : 0)) * 8)) return e;
        uint64_t* sc = m->scratch.as<uint64_t>();
        uint2* match = retrieve ? reinterpret_cast<uint2*>(sc + words) : nullptr;
        MmapCount<KB> f{m->table<KB>(), static_cast<KeyWord<KB> const*>(keys), match};
        if (int e = tile_scan(f, NoAct{}, n, sc, false, s)) return e;
        if (int e = read_word(sc + (n + kTile - 1) / kTile, m->h_word, s, total)) return e;
        if (!retrieve || *total == 0) return B2CO_OK;
        if (*total > cap) return fail(B2CO_ERANGE, "StaticMultimap: output capacity is insufficient");
        if (!key_out || !value_out) return fail(B2CO_EINVAL, "StaticMultimap: null nonempty buffer");
        k_mmap_retrieve<KB, VB><<<uint32_t((n + kTile - 1) / kTile), kThreads, 0, s>>>(
            static_cast<KeyWord<KB> const*>(keys), match, static_cast<ValueWord<VB> const*>(m->csr),
            static_cast<KeyWord<KB>*>(key_out), static_cast<ValueWord<VB>*>(value_out), n, sc);
        B2CO_CUDA(cudaGetLastError());
        B2CO_CUDA(cudaStreamSynchronize(s));
        return B2CO_OK;
    });
}

int b2co_mmap_count(b2co_mmap* m, void const* keys, uint64_t n, b2co_stream st, uint64_t* total)
{
    if (!total) return fail(B2CO_EINVAL, "null output");
    return mmap_count_any(m, keys, n, st, total, false, nullptr, nullptr, 0);
}

int b2co_mmap_retrieve(b2co_mmap* m, void const* keys, uint64_t n, void* key_out, void* value_out, uint64_t cap,
                       b2co_stream st, uint64_t* written)
{
    if (!written) return fail(B2CO_EINVAL, "null output");
    uint64_t total = 0;
    *written = 0;
    int r = mmap_count_any(m, keys, n, st, &total, true, key_out, value_out, cap);
    if (!r) *written = total;
    return r;
}

int b2co_mmap_retrieve_all(b2co_mmap* m, void* key_out, void* value_out, uint64_t cap, b2co_stream st,
                           uint64_t* written)
{
    if (int e = check_mmap(m)) return e;
    if (!written) return fail(B2CO_EINVAL, "null output");
    *written = 0;
    if (m->size > cap) return fail(B2CO_ERANGE, "StaticMultimap: output capacity is insufficient");
    if (!m->size) return B2CO_OK;
    if (!key_out || !value_out) return fail(B2CO_EINVAL, "StaticMultimap: null nonempty buffer");
    int r = by_kv(m->kb, m->vb, [&](auto k, auto v) -> int {
        constexpr int KB = decltype(k)::value, VB = decltype(v)::value;
        using Raw = typename SlotT<KB, VB>::Raw;
        k_mmap_export<KB, VB><<<blocks_for(m->size), 256, 0, cs(st)>>>(static_cast<Raw const*>(m->dense), m->size,
                                                                        static_cast<KeyWord<KB>*>(key_out), value_out);
        B2CO_CUDA(cudaGetLastError());
        B2CO_CUDA(cudaStreamSynchronize(cs(st)));
        return B2CO_OK;
    });
    if (!r) *written = m->size;
    return r;
}

}  // extern "C"
