// oa_inst.cuh -- launchers of the open-addressing kernels for one slot layout.
// Each oa_slot_*.cu instantiates this for one layout so the six layouts
// compile in parallel.
#pragma once

#include "b2co_host.h"
#include "group_kernels.cuh"
#include "oa_insert.cuh"
#include "oa_kernels.cuh"

namespace b2co {

// Which kernels a table takes by default (no shape set), by measurement with
// half-full tables and 50% hits on one B200 (both kernels, same box):
//
// Lookups.  The one-lane sector kernel (oa_sector.cuh) asks L2 for a window
// sector by sector.  Where most sectors are in L2 that is the cheapest form, but
// HBM serves about 37 G missed requests a second however many are in flight, so
// on large tables the tiled kernels, which ask for a window in one or two
// requests, win.  16 M queries, sector / 2 lanes / 4 lanes x 2 in Gkeys/s:
//   16-byte slots: 40 MB 70 / 66 / 42, 120 MB 47 / 40 / 33, 220 MB 38 / 34 / 31, 300 MB 26 / 33 / 30
//   8-byte slots:  20 MB 97 / 83 / 51, 160 MB 57 / 50 / 35, 300 MB 36 / 46 / 33
//   4-byte slots:  40 MB 72 / 93 / 59: two lanes read such a window in fewer instructions
// A small batch is bound by the length of its chain of loads, not by requests,
// whatever the table: on a 1 GB table, sector / 4 lanes x 2 take 4.8 / 6.9 us for
// 16,384 keys, 8.9 / 10.1 for 65,536 and 13.6 / 12.1 for 131,072.
constexpr uint64_t kSectorFindBytes = uint64_t(224) << 20;
constexpr uint32_t kSectorFindKeys = 3u << 15;
// Tables inside the line all the same take the tiled lookup in large batches where
// the sector kernel is bound by instructions, sector / tiled in Gkeys/s (16 M queries,
// 16-byte slots): windows of four sectors (eight slots), 24 / 150 / 220 MB 46 / 46 / 39 and
// 56 / 49 / 46; and of three for a Contains, which needs the keys only, with the table
// well inside L2 (five slots), 24 / 60 / 150 MB 72 / 71 / 51 and 80 / 63 / 40.  Smaller
// batches and fuller tables would lose: 1 Mi queries at load 0.95, 24 MB, 69 us and 91.
constexpr uint64_t kTiledContainsBytes = uint64_t(40) << 20;
constexpr uint32_t kTiledFourKeys = 1u << 20, kTiledContainsKeys = 1u << 22;
// Two lanes and one window in flight against four and two: 34 / 31 at 220 MB,
// 33 / 30 at 300 MB, 27 / 29 at 520 MB.
constexpr uint64_t kNarrowFindBytes = uint64_t(320) << 20;
// Writes.  The same trade with a CAS or a store behind every window, sector / 4
// lanes in Gpairs/s: Insert 300 MB 18.9 / 15.8, 400 MB 14.9 / 15.7; InsertOrAssign of
// present keys 220 MB 22.5 / 19.4, 300 MB 17.9 / 18.8.
constexpr uint64_t kSectorInsertBytes = uint64_t(352) << 20;
constexpr uint64_t kSectorAssignBytes = uint64_t(256) << 20;
// A small batch, as with the lookups: on a 1.2 GB table, sector / tiled, InsertOrAssign of 8,192 /
// 32,768 / 65,536 / 131,072 present keys takes 5.4 / 8.2, 6.8 / 8.5, 10.1 / 10.2 and 16.9 / 13.3 us.
constexpr uint32_t kSectorWriteKeys = 1u << 16;
// Threads per block of the sector kernels: a batch that does not fill the GPU is
// spread over more SMs in smaller blocks (an SM takes its windows' requests one
// after the other): 1,000 keys take 3.8 us in blocks of 64 and 4.8 in blocks of 256.
constexpr uint32_t kSpreadKeys = 1u << 17;
inline uint32_t sector_block(uint32_t n) { return n <= kSpreadKeys ? 64 : 256; }

template <class S>
struct OaImpl {
    static constexpr uint32_t kBlock = 256;
    // The integer 4- and 8-byte layouts compile every lookup and write shape;
    // 2-byte and floating-point-key layouts compile the default shapes only
    // (another requested shape runs the default one).
    static constexpr bool kAllShapes = !S::float_key && S::key_bytes >= 4;

    template <class F>
    static int with_b(uint32_t b, F&& f)
    {
        switch (b) {
            case 1: return f(std::integral_constant<int, 1>{});
            case 2: return f(std::integral_constant<int, 2>{});
            case 4: return f(std::integral_constant<int, 4>{});
            case 5: return f(std::integral_constant<int, 5>{});
            case 8: return f(std::integral_constant<int, 8>{});
        }
        return fail(B2CO_EINVAL, "unsupported bucket size");
    }

    static int check_launch(char const* what)
    {
        cudaError_t e = cudaGetLastError();
        return e == cudaSuccess ? B2CO_OK : cuda_fail(e, what);
    }

    static int clear(OaArgs const& a, cudaStream_t s)
    {
        auto k = k_clear<S>;
        k<<<grid_for((void const*)k, kBlock, a.probe.capacity, kBlock * 4), kBlock, 0, s>>>(
            a.slots, a.probe.capacity, a.empty_key, a.empty_value);
        return check_launch("clear kernel");
    }

    static uint64_t table_bytes(OaArgs const& a) { return uint64_t(a.probe.capacity) * S::bytes; }

    // Whether the insert family runs one key per lane (oa_sector.cuh) instead of
    // a tile per window (oa_insert.cuh).
    static bool sector_writes(OaArgs const& a, int B, int mode, uint32_t n)
    {
        uint32_t const lanes = a.write_shape >> 8;
        return B == 1 || lanes == 1 ||
               (lanes == 0 && (n <= kSectorWriteKeys ||
                               table_bytes(a) <= (mode == kInsAssign ? kSectorAssignBytes
                                                  : mode >= kInsMark  ? kSectorFindBytes
                                                                      : kSectorInsertBytes)));
    }

    // A write of one mode.
    template <int B, int MODE>
    static int write(OaArgs const& a, void const* pairs, uint8_t const* stencil, uint32_t n, InsOut const& o,
                     cudaStream_t s)
    {
        if constexpr (B > 1) {
            if (!sector_writes(a, B, MODE, n)) {
                auto k = k_insert_tile<S, B, MODE>;
                uint32_t const block = sector_block(n);
                k<<<grid_for((void const*)k, block, n, block), block, 0, s>>>(a, pairs, stencil, n, o);
                return check_launch("insert kernel");
            }
        }
        auto k = k_insert_sector<S, B, MODE>;
        uint32_t const block = sector_block(n);
        k<<<grid_for((void const*)k, block, n, block), block, 0, s>>>(a, pairs, stencil, n, o);
        return check_launch("insert kernel");
    }

    static int insert(OaArgs const& a, uint32_t b, void const* pairs, uint8_t const* stencil, uint32_t n,
                      bool assign, Counters const& counters, cudaStream_t s)
    {
        return with_b(b, [&](auto bc) {
            constexpr int B = decltype(bc)::value;
            InsOut o{};
            o.counters = counters;
            return assign ? write<B, kInsAssign>(a, pairs, stencil, n, o, s)
                          : write<B, kInsPlain>(a, pairs, stencil, n, o, s);
        });
    }

    static int mark(OaArgs const& a, uint32_t b, void const* pairs, uint32_t n, bool assign, uint8_t* absent,
                    cudaStream_t s)
    {
        if constexpr (S::is_set) {
            return fail(B2CO_ELOGIC, "marking is for maps (DynamicMap's submaps)");
        } else {
            return with_b(b, [&](auto bc) {
                constexpr int B = decltype(bc)::value;
                InsOut o{};
                o.inserted = absent;
                return assign ? write<B, kInsMarkAssign>(a, pairs, nullptr, n, o, s)
                              : write<B, kInsMark>(a, pairs, nullptr, n, o, s);
            });
        }
    }

    static int assign_if(OaArgs const& a, uint32_t b, void const* pairs, uint8_t const* stencil, uint32_t n,
                         cudaStream_t s)
    {
        return with_b(b, [&](auto bc) {
            constexpr int B = decltype(bc)::value;
            auto k = k_assign_if<S, B>;
            k<<<grid_for((void const*)k, kBlock, n, kBlock), kBlock, 0, s>>>(a, pairs, stencil, n);
            return check_launch("assign kernel");
        });
    }

    static int iaf_race(OaArgs const& a, uint32_t b, void const* pairs, void* found, uint8_t* inserted, uint32_t n,
                        cudaStream_t s)
    {
        return with_b(b, [&](auto bc) {
            constexpr int B = decltype(bc)::value;
            InsOut o{};
            o.found = found;
            o.inserted = inserted;
            return write<B, kInsIafRace>(a, pairs, nullptr, n, o, s);
        });
    }

    static int iaf_first(OaArgs const& a, uint32_t b, void const* pairs, void* found, uint8_t* inserted,
                         uint32_t n, uint32_t* pos, uint32_t* newbits, uint32_t* owner, cudaStream_t s)
    {
        return with_b(b, [&](auto bc) {
            constexpr int B = decltype(bc)::value;
            // `newbits` holds two bitmaps of the table's slots: claimed in this
            // batch, then shared with later inputs of the batch (`dup`)
            uint32_t* dup = newbits + (uint64_t(a.probe.capacity) + 31) / 32;
            uint32_t const claim_bit = a.probe.capacity < kClaimBit ? kClaimBit : 0u;  // slot indices below 2^31 - 1
            InsOut o{};
            o.pos = pos;
            o.newbits = newbits;
            o.owner = owner;
            o.claim_bit = claim_bit;
            if (int st = write<B, kInsIafPlace>(a, pairs, nullptr, n, o, s)) return st;
            auto const grid = [&](void const* k) { return grid_for(k, kBlock, (uint64_t(n) + 3) / 4, kBlock); };
            k_iaf_min<S><<<grid((void const*)k_iaf_min<S>), kBlock, 0, s>>>(pos, newbits, dup, owner, n, claim_bit);
            if (claim_bit)
                k_iaf_claim<S><<<grid((void const*)k_iaf_claim<S>), kBlock, 0, s>>>(pos, dup, owner, n, claim_bit);
            auto k3 = k_iaf_final<S>;
            k3<<<grid((void const*)k3), kBlock, 0, s>>>(a, pairs, pos, newbits, dup, owner, found, inserted, n,
                                                        claim_bit);
            if (claim_bit) {
                // owner[] back to all-ones: a batch within 8x of the table's slots
                // clears the whole array (one sequential write) rather than
                // visiting its shared slots at random
                if (uint64_t(a.probe.capacity) <= 8ull * n) {
                    cudaError_t const e = cudaMemsetAsync(owner, 0xff, uint64_t(a.probe.capacity) * 4, s);
                    if (e != cudaSuccess) return cuda_fail(e, "insert_and_find (first wins) owner reset");
                } else {
                    k_iaf_restore<S><<<grid((void const*)k_iaf_restore<S>), kBlock, 0, s>>>(pos, dup, owner, n,
                                                                                             claim_bit);
                }
            }
            return check_launch("insert_and_find (first wins) kernels");
        });
    }

    template <int B, int G, bool C, bool SEG>
    static int find_staged(OaArgs const& a, uint32_t items, void const* keys, void* out, uint32_t n, WaitCtl wc,
                           cudaStream_t s)
    {
        void (*k)(OaArgs, void const*, void*, uint32_t, WaitCtl) = nullptr;
        if (items >= 4 && G >= 4) k = k_find_staged<S, B, G, (G >= 4 ? 4 : 1), C, SEG>;
        else if (items >= 2) k = k_find_staged<S, B, G, 2, C, SEG>;
        else k = k_find_staged<S, B, G, 1, C, SEG>;
        uint64_t chunks = n / kStageKeys;
        uint32_t grid = grid_for((void const*)k, kBlock, chunks ? chunks : 1, 1);
        k<<<grid, kBlock, 0, s>>>(a, keys, out, n, wc);
        return check_launch(C ? "contains kernel" : "find kernel");
    }

    template <int B, int G, bool C>
    static int find_wstaged(OaArgs const& a, uint32_t items, void const* keys, void* out, uint32_t n, WaitCtl wc,
                            cudaStream_t s)
    {
        void (*k)(OaArgs, void const*, void*, uint32_t, WaitCtl) = nullptr;
        if (items >= 4 && G >= 4) k = k_find_wstaged<S, B, G, (G >= 4 ? 4 : 1), C>;
        else if (items >= 2) k = k_find_wstaged<S, B, G, 2, C>;
        else k = k_find_wstaged<S, B, G, 1, C>;
        uint64_t warps = (n + kWarpStageKeys - 1) / kWarpStageKeys;
        uint32_t grid = grid_for((void const*)k, kBlock, warps ? warps : 1, kBlock / 32);
        k<<<grid, kBlock, 0, s>>>(a, keys, out, n, wc);
        return check_launch(C ? "contains kernel" : "find kernel");
    }

    using DeferFn = void (*)(OaArgs, void const*, void*, uint32_t, uint32_t, WaitCtl);

    // Resident warps of a deferred lookup.
    static uint64_t defer_warps(DeferFn k) { return uint64_t(grid_for((void const*)k, kBlock, ~0ull, 1)) * (kBlock / 32); }

    static int launch_wdefer(DeferFn k, bool contains, OaArgs const& a, void const* keys, void* out, uint32_t n,
                             uint64_t chunk, WaitCtl wc, cudaStream_t s)
    {
        k<<<grid_for((void const*)k, kBlock, (n + chunk - 1) / chunk, kBlock / 32), kBlock, 0, s>>>(
            a, keys, out, n, uint32_t(chunk), wc);
        return check_launch(contains ? "contains kernel" : "find kernel");
    }

    // The default deferred lookup.  A batch that does not fill every resident
    // warp's stage is dealt evenly over them (a stage is a chain of dependent
    // passes: 65,536 keys in whole stages ran 16 of them one after the other on 32
    // blocks, 16.1 us against 10.1).
    template <int B, int G, int Q, bool C>
    static int find_defer_auto(OaArgs const& a, void const* keys, void* out, uint32_t n, WaitCtl wc, cudaStream_t s)
    {
        DeferFn even = k_find_wdefer<S, B, G, Q, C, true>;
        if constexpr (!S::is_set)  // DynamicMap's lookups
            if (a.keep_misses) even = k_find_wdefer<S, B, G, Q, C, true, true>;
        uint64_t const share = (n + defer_warps(even) - 1) / defer_warps(even);
        // (the even deal's kernel for windows of four sectors is the slower one: 1 Mi keys, 300 MB, 29 us against 40)
        uint64_t const whole = SectorWindow<S, B>::NS >= 4 ? kWarpStageKeys / 2 : kWarpStageKeys;
        if (share >= whole && !a.keep_misses)
            return launch_wdefer(k_find_wdefer<S, B, G, Q, C>, C, a, keys, out, n, kWarpStageKeys, wc, s);
        uint64_t const rounds = (share + kWarpStageKeys - 1) / kWarpStageKeys;
        return launch_wdefer(even, C, a, keys, out, n, ((share + rounds - 1) / rounds + 31) / 32 * 32, wc, s);
    }

    template <int B, int G, bool C>
    static int find_wdefer(OaArgs const& a, uint32_t items, void const* keys, void* out, uint32_t n, WaitCtl wc,
                           cudaStream_t s)
    {
        DeferFn k = nullptr;
        if (items >= 4 && G >= 4) k = k_find_wdefer<S, B, G, (G >= 4 ? 4 : 1), C>;
        else if (items >= 2) k = k_find_wdefer<S, B, G, 2, C>;
        else k = k_find_wdefer<S, B, G, 1, C>;
        return launch_wdefer(k, C, a, keys, out, n, kWarpStageKeys, wc, s);
    }

    template <int B, bool C>
    static int find_sector(OaArgs const& a, void const* keys, uint8_t const* stencil, void* out, uint32_t n,
                           cudaStream_t s)
    {
        auto k = k_find_sector<S, B, C, false>;
        if constexpr (!S::is_set)  // DynamicMap's lookups
            if (a.keep_misses) k = k_find_sector<S, B, C, true>;
        uint32_t const block = sector_block(n);
        k<<<grid_for((void const*)k, block, n, block), block, 0, s>>>(a, keys, stencil, out, n);
        return check_launch(C ? "contains kernel" : "find kernel");
    }

    // The lookup of a table without a shape of its own (lanes 0); see
    // kSectorFindBytes.
    template <int B, bool C>
    static int find_auto(OaArgs const& a, void const* keys, uint8_t const* stencil, void* out, uint32_t n, WaitCtl wc,
                         cudaStream_t s)
    {
        if constexpr (B > 1) {
            constexpr int kSectors = SectorWindow<S, B>::NS;
            bool const tiled = table_bytes(a) > kSectorFindBytes || S::bytes <= 4 || (kSectors >= 4 && n >= kTiledFourKeys) ||
                               (C && kSectors == 3 && !a.keep_misses && table_bytes(a) <= kTiledContainsBytes &&
                                n >= kTiledContainsKeys);
            if (tiled && n > kSectorFindKeys) {
                bool const narrow = S::bytes <= 4 || table_bytes(a) <= kNarrowFindBytes;
                if (stencil || (reinterpret_cast<uintptr_t>(keys) & 15))  // keys cannot be staged
                    return find_shape<B, C>(a, narrow ? 2 : 4, 1, keys, stencil, out, n, wc, s);
                return narrow ? find_defer_auto<B, 2, 1, C>(a, keys, out, n, wc, s)
                              : find_defer_auto<B, 4, 2, C>(a, keys, out, n, wc, s);
            }
        }
        return find_sector<B, C>(a, keys, stencil, out, n, s);
    }

    template <int B, bool C>
    static int find_bulk(OaArgs const& a, void const* keys, void* out, uint32_t n, WaitCtl wc, cudaStream_t s)
    {
        if constexpr (S::bytes == 16) {
            auto k = k_find_bulk<S, B, C>;
            constexpr uint32_t smem = bulk_window_smem<S, B>();
            // a per-device function attribute: set on every launch (about a microsecond)
            cudaError_t const ea = cudaFuncSetAttribute((void const*)k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                        smem);
            if (ea != cudaSuccess) return cuda_fail(ea, "bulk find attribute");
            int per_sm = 0;
            cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (void const*)k, kBlock, smem);
            if (e != cudaSuccess) return cuda_fail(e, "bulk find occupancy");
            uint64_t chunks = n / kStageKeys;
            uint64_t cap = uint64_t(per_sm < 1 ? 1 : per_sm) * sm_count();
            uint32_t grid = uint32_t(chunks == 0 ? 1 : (chunks < cap ? chunks : cap));
            k<<<grid, kBlock, smem, s>>>(a, keys, out, n, wc);
            return check_launch(C ? "contains kernel" : "find kernel");
        } else {
            return fail(B2CO_EINVAL, "bulk windows need 16-byte slots");
        }
    }

    // The shapes of layouts without kAllShapes: per-warp staging with deferred
    // continuations, 2 or 4 lanes per window, one or two windows in flight; the
    // ballot tile (stencils, unaligned key streams) or one lane per key (bucket
    // size 1) otherwise.
    template <int B, bool C>
    static int find_default(OaArgs const& a, uint32_t lanes, uint32_t items, void const* keys,
                            uint8_t const* stencil, void* out, uint32_t n, WaitCtl wc, cudaStream_t s)
    {
        bool const staged = !stencil && (reinterpret_cast<uintptr_t>(keys) & 15) == 0 && n >= kWarpStageKeys &&
                            B > 1 && lanes >= 2;
        uint32_t const q = (items & ~(kShapeDeferred | kShapeWarpStaged | kShapeSegmented | kShapeBulk)) >= 2 ? 2 : 1;
        if (staged) {
            DeferFn k = nullptr;
            if (lanes == 2) k = q == 2 ? k_find_wdefer<S, B, 2, 2, C> : k_find_wdefer<S, B, 2, 1, C>;
            else k = q == 2 ? k_find_wdefer<S, B, 4, 2, C> : k_find_wdefer<S, B, 4, 1, C>;
            return launch_wdefer(k, C, a, keys, out, n, kWarpStageKeys, wc, s);
        }
        if (B == 1 || lanes <= 1) return find_sector<B, C>(a, keys, stencil, out, n, s);
        uint64_t const per_block = lanes == 2 ? kBlock / 2 : kBlock / 4;
        auto k = lanes == 2 ? k_find_tile<S, B, 2, C> : k_find_tile<S, B, 4, C>;
        k<<<grid_for((void const*)k, kBlock, n, per_block), kBlock, 0, s>>>(a, keys, stencil, out, n);
        return check_launch(C ? "contains kernel" : "find kernel");
    }

    template <int B, bool C>
    static int find_shape(OaArgs const& a, uint32_t lanes, uint32_t items, void const* keys, uint8_t const* stencil,
                          void* out, uint32_t n, WaitCtl wc, cudaStream_t s)
    {
        if constexpr (!kAllShapes) {
            return find_default<B, C>(a, lanes, items, keys, stencil, out, n, wc, s);
        } else {
            return find_any<B, C>(a, lanes, items, keys, stencil, out, n, wc, s);
        }
    }

    template <int B, bool C>
    static int find_any(OaArgs const& a, uint32_t lanes, uint32_t items, void const* keys, uint8_t const* stencil,
                        void* out, uint32_t n, WaitCtl wc, cudaStream_t s)
    {
        bool const stageable = !stencil && (reinterpret_cast<uintptr_t>(keys) & 15) == 0 && n >= kStageKeys && B > 1;
        // bulk-window path: 16-byte slots only
        if constexpr (B == 5) {  // the block-staged, warp-staged and bulk shapes: bucket size 5 only (build time)
            if ((items & kShapeBulk) && stageable && S::bytes == 16) return find_bulk<B, C>(a, keys, out, n, wc, s);
        } else if (stageable && lanes >= 2) {
            items |= kShapeDeferred;  // other bucket sizes stage keys the default way
        }
        items &= ~kShapeBulk;
        // staged path: no stencil, 16-byte aligned key stream, at least one stage of keys
        bool const staged = stageable && lanes >= 2;
        if (staged && (items & kShapeDeferred)) {
            items &= ~(kShapeDeferred | kShapeWarpStaged | kShapeSegmented);
            if (lanes == 2) return find_wdefer<B, 2, C>(a, items, keys, out, n, wc, s);
            if (lanes == 4) return find_wdefer<B, 4, C>(a, items, keys, out, n, wc, s);
            return find_wdefer<B, 8, C>(a, items, keys, out, n, wc, s);
        }
        items &= ~kShapeDeferred;
        if constexpr (B == 5) {
            if (staged && (items & kShapeWarpStaged)) {
                items &= ~(kShapeWarpStaged | kShapeSegmented);
                if (lanes == 2) return find_wstaged<B, 2, C>(a, items, keys, out, n, wc, s);
                if (lanes == 4) return find_wstaged<B, 4, C>(a, items, keys, out, n, wc, s);
                return find_wstaged<B, 8, C>(a, items, keys, out, n, wc, s);
            }
            items &= ~kShapeWarpStaged;
            if (staged) {
                bool const seg = (items & kShapeSegmented) != 0;
                items &= ~kShapeSegmented;
                if (seg) {
                    if (lanes == 2) return find_staged<B, 2, C, true>(a, items, keys, out, n, wc, s);
                    if (lanes == 4) return find_staged<B, 4, C, true>(a, items, keys, out, n, wc, s);
                    return find_staged<B, 8, C, true>(a, items, keys, out, n, wc, s);
                }
                if (lanes == 2) return find_staged<B, 2, C, false>(a, items, keys, out, n, wc, s);
                if (lanes == 4) return find_staged<B, 4, C, false>(a, items, keys, out, n, wc, s);
                return find_staged<B, 8, C, false>(a, items, keys, out, n, wc, s);
            }
        }
        items &= ~kShapeWarpStaged;
        items &= ~kShapeSegmented;
        if (B == 1 || lanes <= 1) return find_sector<B, C>(a, keys, stencil, out, n, s);
        auto k = lanes == 2 ? k_find_tile<S, B, 2, C> : lanes == 4 ? k_find_tile<S, B, 4, C> : k_find_tile<S, B, 8, C>;
        k<<<grid_for((void const*)k, kBlock, n, kBlock / lanes), kBlock, 0, s>>>(a, keys, stencil, out, n);
        return check_launch(C ? "contains kernel" : "find kernel");
    }

    static int find(OaArgs const& a, uint32_t b, uint32_t lanes, uint32_t items, bool contains, void const* keys,
                    uint8_t const* stencil, void* out, uint32_t n, WaitCtl wc, cudaStream_t s)
    {
        return with_b(b, [&](auto bc) {
            constexpr int B = decltype(bc)::value;
            if (lanes == 0)
                return contains ? find_auto<B, true>(a, keys, stencil, out, n, wc, s)
                                : find_auto<B, false>(a, keys, stencil, out, n, wc, s);
            return contains ? find_shape<B, true>(a, lanes, items, keys, stencil, out, n, wc, s)
                            : find_shape<B, false>(a, lanes, items, keys, stencil, out, n, wc, s);
        });
    }

    static int erase(OaArgs const& a, uint32_t b, void const* keys, uint32_t n, unsigned long long* counters,
                     cudaStream_t s)
    {
        return with_b(b, [&](auto bc) {
            constexpr int B = decltype(bc)::value;
            auto k = k_erase<S, B>;
            k<<<grid_for((void const*)k, kBlock, n, kBlock), kBlock, 0, s>>>(a, keys, n, counters);
            return check_launch("erase kernel");
        });
    }

    static int count(OaArgs const& a, uint32_t b, void const* keys, uint32_t n, unsigned long long* counter,
                     cudaStream_t s)
    {
        return with_b(b, [&](auto bc) {
            constexpr int B = decltype(bc)::value;
            auto k = k_count<S, B>;
            k<<<grid_for((void const*)k, kBlock, n, kBlock), kBlock, 0, s>>>(a, keys, n, counter);
            return check_launch("count kernel");
        });
    }

    static constexpr OaOps ops{&clear, &insert, &mark, &assign_if, &iaf_race, &iaf_first, &find, &erase, &count};
};

template <class S>
struct GroupImpl {
    static constexpr uint32_t kBlock = 256;

    // `shape` packs lanes per window (bits 0-7), keys in flight per lane group
    // (bits 8-15; 1 = one key per tile, resolved at once) and threads per block
    // (bits 16-31; 0 = 256).  Keys per tile above 1 run the deferred kernel;
    // its 2-, 4- and 8-lane variants other than 4x2 exist for bucket size 5.
    template <int B, bool C>
    static int find_b(GroupArgs const& g, uint32_t shape, void const* keys, void* out, uint64_t n, cudaStream_t s)
    {
        uint32_t const lanes = shape & 0xffu, items = (shape >> 8) & 0xffu;
        uint32_t const block = (shape >> 16) ? (shape >> 16) : kBlock;
        void (*k)(GroupArgs, void const*, void*, uint64_t, uint32_t) = nullptr;
        if (lanes >= 2 && items >= 2) {
            if constexpr (B == 5) {
                if (lanes == 2) k = k_group_find_q<S, B, 2, 2, C>;
                else if (lanes == 4 && items >= 4) k = k_group_find_q<S, B, 4, 4, C>;
                else if (lanes == 8) k = items >= 4 ? k_group_find_q<S, B, 8, 4, C> : k_group_find_q<S, B, 8, 2, C>;
            }
            if (!k) k = k_group_find_q<S, B, 4, 2, C>;
        } else if (lanes <= 1) {
            k = k_group_find_lane<S, B, C>;
        } else if (lanes == 2) {
            k = k_group_find<S, B, 2, C>;
        } else if (lanes == 4) {
            k = k_group_find<S, B, 4, C>;
        } else {
            k = k_group_find<S, B, 8, C>;
        }
        // persistent: every resident block, at least 32 items a warp
        uint32_t const grid = grid_for((void const*)k, block, n, block);
        k<<<grid, block, 0, s>>>(g, keys, out, n, group_chunk(n, uint64_t(grid) * block / 32));
        return OaImpl<S>::check_launch(C ? "group contains kernel" : "group find kernel");
    }

    static int find(GroupArgs const& g, uint32_t b, uint32_t shape, bool contains, void const* keys, void* out,
                    uint64_t n, cudaStream_t s)
    {
        return OaImpl<S>::with_b(b, [&](auto bc) {
            constexpr int B = decltype(bc)::value;
            return contains ? find_b<B, true>(g, shape, keys, out, n, s) : find_b<B, false>(g, shape, keys, out, n, s);
        });
    }

    static int insert(GroupArgs const& g, uint32_t b, bool tiled, void const* pairs, uint64_t n,
                      unsigned long long* failed, cudaStream_t s)
    {
        return OaImpl<S>::with_b(b, [&](auto bc) {
            constexpr int B = decltype(bc)::value;
            auto k = k_group_insert<S, B, false>;
            if constexpr (B > 1)
                if (tiled) k = k_group_insert<S, B, true>;
            uint32_t const grid = grid_for((void const*)k, kBlock, n, kBlock);
            k<<<grid, kBlock, 0, s>>>(g, pairs, n, group_chunk(n, uint64_t(grid) * kBlock / 32), failed);
            return OaImpl<S>::check_launch("group insert kernel");
        });
    }

    static constexpr GroupOps ops{&find, &insert};
};

}  // namespace b2co

#define B2CO_DEFINE_OA_OPS(NAME, GNAME, KB, VB)            \
    namespace b2co {                                       \
    OaOps const NAME = OaImpl<SlotT<KB, VB>>::ops;         \
    GroupOps const GNAME = GroupImpl<SlotT<KB, VB>>::ops;  \
    }

// Layouts served by single tables only (no table-group kernels): 2-byte keys
// and floating-point keys (FK = true).
#define B2CO_DEFINE_OA_OPS_ONLY(NAME, KB, VB, FK)          \
    namespace b2co {                                       \
    OaOps const NAME = OaImpl<SlotT<KB, VB, FK>>::ops;     \
    }
