// oa_insert.cuh -- the write kernel of large tables: Insert / InsertIf,
// InsertOrAssign, InsertAndFind (race), the placement pass of first-wins
// InsertAndFind, and the marking passes of DynamicMap.
//
// Per-key algorithm (InsertVerdict, open_addressing_ref_impl.h:489-532): walk
// the key's probe sequence bucket window by bucket window; in a window the
// first slot, in scan order, that is empty (bitwise sentinel test) or holds an
// equal key decides -- an equal key is DUPLICATE (InsertOrAssign overwrites its
// payload), an empty slot is claimed by a compare-and-swap of the whole slot
// (SUCCESS), and a lost CAS continues the scan after that slot unless the
// winner holds an equal key (DUPLICATE).  A whole cycle without a decision, or
// the empty key itself, is FAILED.
//
// As in the sector kernels (oa_sector.cuh) a lane owns a key, hashes it, issues
// its CAS and queues it.  Between, the warp reads its 32 windows in G sub-passes
// of 32/G windows: the G lanes of a tile read one sector each, so a window is
// one load instruction and one or two requests, all sub-passes in flight
// together.  HBM answers a missed request, not a byte, at a time, which is why
// large tables want a window in as few requests as it takes.  A tile agrees by
// one ballot (the lowest lane holding a deciding slot), and the owner gets the
// slot's place by one shuffle.
//
// InsertAndFind (race) of slots up to 8 bytes takes the present slot from the tile
// by one more shuffle; reading it again is an access to HBM (16 M pairs, 1.1 GB of
// 8-byte slots: 884 to 519 us).  A wider slot is read again.
//
// The window is a snapshot, and that is safe: during these kernels slots only
// go from empty to occupied, so a slot seen occupied by another key stays so,
// and a slot seen empty is re-checked by the CAS itself.
//
// Bound by HBM's random accesses, a read of the window and the write-back of a
// slot per key.  134 M pairs into a half-full 4.3 GB table: 17.4 Gpairs/s, against
// 15.2 with one key per four lanes (a slot a lane, two loads a window, 8 keys in
// flight a warp and not 32).
// Every loop is bounded by the probe cycle, so no kernel can spin.
#pragma once

#include "oa_sector.cuh"

namespace b2co {

template <class S, int B>
constexpr int kTileLanes = SectorWindow<S, B>::NS <= 1 ? 1 : SectorWindow<S, B>::NS <= 2 ? 2 : 4;

#ifndef B2CO_TILE_WRITE_MINB
#define B2CO_TILE_WRITE_MINB(G) ((G) >= 4 ? 3 : 4)
#endif

template <class S, int B, int MODE>
__global__ void __launch_bounds__(256, B2CO_TILE_WRITE_MINB((kTileLanes<S, B>)))
    k_insert_tile(__grid_constant__ const OaArgs a, void const* pairs, uint8_t const* stencil, uint32_t n,
                  __grid_constant__ const InsOut o)
{
    using Raw = typename S::Raw;
    constexpr int G = kTileLanes<S, B>;
    constexpr bool kCarry = MODE == kInsIafRace && S::bytes <= 8;  // the owner gets the slot itself
    static_assert(SectorWindow<S, B>::NS <= G && G * (32 / S::bytes) <= 32, "tile shape");
    constexpr uint32_t TILES = 32 / G, TM = (1u << G) - 1u, N = 32 / S::bytes;
    constexpr uint32_t RING = kSectorRing - 1;
    __shared__ Raw qpair[8][kSectorRing];
    __shared__ uint32_t qinit[8][kSectorRing], qidx[8][kSectorRing], qpos[8][kSectorRing];

    uint32_t const lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t const r = lane % G, tile = lane / G;
    uint32_t const own_q = lane / TILES, own_shift = (lane % TILES) * G;  // who reads this lane's window
    uint32_t const stride = gridDim.x * blockDim.x;
    uint32_t base = blockIdx.x * blockDim.x + (threadIdx.x & ~31u);
    uint32_t head = 0, count = 0;
    Raw* const slots = reinterpret_cast<Raw*>(a.slots);
    InsRecord<S, MODE> record;

    bool next_in = base + lane < n && (!stencil || stencil[base + lane]);
    Raw next_pair = next_in ? Io<S>::load_pair(pairs, base + lane) : Raw{};
    for (;;) {
        Raw pr;
        uint32_t init, idx, pos;
        bool live;
        if (count >= 32 || base >= n) {
            if (base >= n && count <= 32) break;
            __syncwarp();
            uint32_t const take = count < 32 ? count : 32;
            live = lane < take;
            uint32_t const e = (head + (live ? lane : 0u)) & RING;
            pr = qpair[warp][e];
            init = qinit[warp][e];
            idx = qidx[warp][e];
            pos = qpos[warp][e];
            __syncwarp();
            head = (head + take) & RING;
            count -= take;
            idx = probe_next(idx, probe_step<S::key_bytes, B>(a.probe, S::key(pr)), a.probe.capacity);
            if (live && idx == init) {
                record(a, o, pos, kFailed, 0, 0);
                live = false;
            }
        } else {
            pos = base + lane;
            pr = next_pair;
            live = next_in;
            if (live && S::key(pr) == a.empty_key) {
                record(a, o, pos, kFailed, 0, 0);
                live = false;
            }
            init = idx = probe_init<S::key_bytes, B>(a.probe, S::key(pr));
            base += stride;
            next_in = base < n && base + lane < n && (!stencil || stencil[base + lane]);
            next_pair = next_in ? Io<S>::load_pair(pairs, base + lane) : Raw{};
        }
        uint64_t const key = S::key(pr);
        uint32_t const live_mask = __ballot_sync(0xffffffffu, live);
        Sector w[G];
        uint64_t k[G];
        uint32_t valid[G];  // the slots of this lane's sector that lie in the window
#pragma unroll
        for (int q = 0; q < G; ++q) {
            uint32_t const src = q * TILES + tile;
            k[q] = S::key_bytes <= 4 ? uint64_t(__shfl_sync(0xffffffffu, uint32_t(key), src))
                                     : __shfl_sync(0xffffffffu, (unsigned long long)key, src);
            uint32_t const ix = __shfl_sync(0xffffffffu, idx, src);
            uintptr_t const addr = reinterpret_cast<uintptr_t>(slots + ix);
            valid[q] = ((((1u << B) - 1u) << (uint32_t(addr & 31) / S::bytes)) >> (r * N)) & ((1u << N) - 1u);
            if (!((live_mask >> src) & 1u)) valid[q] = 0;
            if (valid[q]) w[q] = ld_sector<true, false>(reinterpret_cast<void const*>((addr & ~uintptr_t(31)) + r * 32));
        }
        // each owner learns where its window's first deciding slot is and whether it is empty
        uint32_t mine = 0;  // slot among the window's sectors | 32: empty | 64: found
        Raw carried{};
#pragma unroll
        for (int q = 0; q < G; ++q) {
            uint32_t info = 0;
            Raw stop{};
            if (valid[q]) {
                uint32_t stops = 0, empties = 0;
#pragma unroll
                for (int i = 0; i < int(N); ++i) {
                    uint64_t const sk = S::key(sector_slot<S>(w[q], i));
                    if (sk == a.empty_key) empties |= 1u << i;
                    else if (S::key_eq(sk, k[q])) stops |= 1u << i;
                }
                stops = (stops | empties) & valid[q];
                if (stops) {
                    uint32_t const i = uint32_t(__ffs(stops) - 1);
                    info = i | (((empties >> i) & 1u) ? 96u : 64u);
                    if constexpr (kCarry) {
#pragma unroll
                        for (int j = 0; j < int(N); ++j)
                            if (i == uint32_t(j)) stop = sector_slot<S>(w[q], j);
                    }
                }
            }
            uint32_t const m = (__ballot_sync(0xffffffffu, info != 0) >> own_shift) & TM;
            uint32_t const first = m ? uint32_t(__ffs(m) - 1) : 0u;
            uint32_t const got = __shfl_sync(0xffffffffu, info, own_shift + first);
            if (uint32_t(q) == own_q && m) mine = got + first * N;
            if constexpr (kCarry) {
                using Word = typename std::conditional<S::bytes == 8, unsigned long long, uint32_t>::type;
                Raw const at = Raw(__shfl_sync(0xffffffffu, Word(stop), own_shift + first));
                if (uint32_t(q) == own_q) carried = at;
            }
        }
        int verdict = kOpen;
        if (live && mine) {
            Raw* const win = slots + idx;
            int j = int(mine & 31u) - int(uint32_t(reinterpret_cast<uintptr_t>(win) & 31) / S::bytes);
            // a 16-byte slot stayed with the tile: a present one is read again where its payload is wanted
            Raw cur = S::make(a.empty_key, a.empty_value);
            if (!(mine & 32u)) cur = kCarry ? carried : MODE == kInsIafRace ? ld_rw(win + j) : S::make(~a.empty_key, 0);
            uint64_t found = 0;
            verdict = sector_decide<S, B, MODE>(a, win, j, cur, key, S::value(pr), found);
            if (verdict != kOpen) record(a, o, pos, verdict, idx + uint32_t(j), found);
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
    // out of line: the loop above runs 5% longer on large batches with it in the kernel
    insert_rest<S, B, MODE, true>(a, o, record, slots, qpair[warp], qinit[warp], qidx[warp], qpos[warp], head, count);
    record.finish(o);
}

}  // namespace b2co
