// Reverse permutations: a B-tree, BST, mvEB or standard-vEB layout back to
// sorted order, in place.  The reference converts only from sorted order to the
// layouts; this is the other direction of the same index maps.
//
// The forward schedule run backwards.  Forward, sorted tile z stores a key
// straight into layout tile u when u was read before z, and through scratch
// otherwise.  Here the tiles go in the opposite order: tile z reads the first
// kind of keys straight from the layout (u is overwritten after z has read it),
// and the second kind from a scratch that a save pass filled first, the mirror
// of the forward second pass.  So a reverse permutation is
//
//  1. init: per tile, the keys that other tiles (and the tile itself) have yet
//     to read from it (its length less what the save pass takes whole);
//  2. save: the scratch keys copied out of the layout;
//  3. unstream: tiles by ticket, in the forward order backwards.  A tile
//     gathers its keys into shared memory, takes what it read off the counts of
//     the tiles it read from, waits for its own count to reach zero and is
//     stored in sorted order.  A wait is only for tiles with earlier tickets,
//     which take off their reads before they wait themselves, so every wait
//     ends; each is bounded.
//
// Traffic is 2 n w (1 + f), f the forward scratch fraction, where a copy of the
// layout and a gather from the copy take 4 n w.  Measured on B200, copy and gather
// as it was (one load a thread at a time) against this: B-tree b = 8 over 6e7 u64
// keys 371 -> 220 us, b = 16 over 5e8 2.97 -> 1.41 ms (5.66 TB/s of 2 n w), mvEB
// over 3e8 u32 keys 969 -> 468 us, over 2^30 - 1 3.37 -> 1.70 ms, standard vEB
// over 3e8 984 -> 517 us, BST over 2^28 - 1 u64 1.87 -> 1.13 ms.  Smaller arrays,
// which stay in L2, go back from a copy in two launches without waits
// (reverse_form).
#include <algorithm>
#include <mutex>
#include <vector>

#include "internal.h"
#include "unpermute.h"

namespace tl {

constexpr int kGatherThreads = 256;
constexpr int kGatherBlocksPerSM = 6;

// ---------------------------------------------------------------- init and save
// Position ranges the save pass takes whole (B-tree).
struct SavedRanges {
    int nr;
    uint64_t lo[kMaxBulkRanges], hi[kMaxBulkRanges];
};

__global__ void btree_reverse_init_kernel(unsigned int *__restrict__ rem, uint64_t n, uint32_t tile_shift,
                                          const __grid_constant__ SavedRanges sr, Ctrl *ctrl) {
    const uint64_t u = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (u == 0) *ctrl = Ctrl{};
    const uint64_t p0 = u << tile_shift;
    if (p0 >= n) return;
    const uint64_t p1 = min(n, p0 + ((uint64_t)1 << tile_shift));
    uint64_t left = p1 - p0;
    for (int r = 0; r < sr.nr; ++r) {
        const uint64_t a = max(p0, sr.lo[r]), e = min(p1, sr.hi[r]);
        if (a < e) left -= e - a;
    }
    rem[u] = (unsigned int)left;
}

// The save pass's whole ranges, through the bulk-copy engine.
template <typename K>
__global__ void __launch_bounds__(32)
btree_save_kernel(K *__restrict__ scr, const K *__restrict__ A, const __grid_constant__ BulkPlan P, Ctrl *ctrl) {
    extern __shared__ __align__(128) unsigned char stage[];
    __shared__ __align__(8) uint64_t bars[kBulkStages];
    bulk_copy_plan(scr, A, P, stage, bars, ctrl);
}

// Plan O's other scratch keys: the host-listed copies backwards, a warp per copy.
template <typename K>
__global__ void __launch_bounds__(kScatterThreads)
btree_fix_save_kernel(K *__restrict__ scr, const K *__restrict__ A, const FixSeg *__restrict__ segs, uint64_t nsegs,
                      uint32_t tile_shift, unsigned int *__restrict__ rem) {
    const uint64_t w = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t i = w; i < nsegs; i += nw) {
        const uint64_t dl = __ldg(reinterpret_cast<const unsigned long long *>(&segs[i].dst_len));
        const uint64_t src = __ldg(reinterpret_cast<const unsigned long long *>(&segs[i].src));
        const uint64_t a = dl & kSegDstMask, e = a + (dl >> 48);
        warp_copy_keys(scr + src, A + a, 0, (uint32_t)(dl >> 48));
        for (uint64_t u = (a >> tile_shift) + (threadIdx.x & 31); u <= (e - 1) >> tile_shift; u += 32)
            atomicSub(&rem[u], (unsigned int)(min(e, (u + 1) << tile_shift) - max(a, u << tile_shift)));
    }
}

__global__ void mveb_reverse_init_kernel(unsigned int *__restrict__ rem, const __grid_constant__ MvebParams prm,
                                         Ctrl *ctrl) {
    const uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k == 0) *ctrl = Ctrl{};
    if (k >= prm.plan.total_tiles) return;
    int ri;
    uint64_t p0, p1;
    mveb_tile(prm.plan, k, ri, p0, p1);
    rem[k] = (unsigned int)(p1 - p0);
}

// Every scratch slot's key (the units' separators and the regions without
// units) from its place in the layout.
template <typename K>
__global__ void __launch_bounds__(kScatterThreads)
mveb_save_kernel(K *__restrict__ scr, const K *__restrict__ A, const __grid_constant__ MvebParams prm,
                 unsigned int *__restrict__ rem) {
    const MvebPlan &P = prm.plan;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t s = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; s < P.total_slots; s += stride) {
        const uint64_t rank = mveb_slot_rank(P, s);
        if (rank == ~0ull) continue;
        const uint64_t p = veb_pos(P.n, rank, P.modified != 0);
        scr[s] = A[p];
        atomicSub(&rem[mveb_tile_of(P, p)], 1u);
    }
}

// ---------------------------------------------------------------- unstream
// Starts copying src[0, len) to shared memory at dst; both are at the same
// offset within 16 bytes.  Vectors by cp.async (wait with load_tile_wait), the
// ragged ends by plain loads.
template <typename K>
__device__ __forceinline__ void stage_run(const K *__restrict__ src, uint32_t len, K *dst, uint32_t tid, uint32_t nt) {
    constexpr uint32_t V = 16 / sizeof(K);
    const uint32_t head = min(len, ((16u - (uint32_t)(reinterpret_cast<uintptr_t>(src) & 15)) & 15u) / (uint32_t)sizeof(K));
    const uint32_t nvec = (len - head) / V, tail = head + nvec * V;
    if (tid < head) dst[tid] = src[tid];
    const char *g = reinterpret_cast<const char *>(src + head);
    const uint32_t s = (uint32_t)__cvta_generic_to_shared(dst + head);
    for (uint32_t v = tid; v < nvec; v += nt)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s + v * 16), "l"(g + (size_t)v * 16) : "memory");
    if (tid < len - tail) dst[tail + tid] = src[tail + tid];
}

// The bulk keys of a kind-1 or kind-3 tile: indices [dbase + j0, dbase + j0 + nb).
TL_HD void btree_bulk_indices(const BtreeStream &S, const Regime &R, uint32_t cnt, uint32_t &j0, uint32_t &nb) {
    const uint32_t d = S.fd32.d;
    uint32_t v0 = R.r0, v1 = R.r0 + cnt;  // [v0, v1) of r0 + offset
    uint32_t q0 = S.fd32.div(v0), q1 = S.fd32.div(v1 - 1);
    if (v0 - q0 * d == R.skip) q0 = S.fd32.div(++v0);
    j0 = v0 - q0;
    nb = 0;
    if (v0 >= v1) return;
    if (v1 - 1 - q1 * d == R.skip) --v1;
    if (v0 >= v1) return;
    nb = v1 - 1 - S.fd32.div(v1 - 1) - j0 + 1;
}

// The part of a run that is read straight from the layout, by tile: c0 keys of
// tile u, c1 of tile u + 1.
TL_HD void btree_run_reads(const BtreeStream &S, const TopRun &run, uint64_t &u, uint32_t &c0, uint32_t &c1) {
    const uint32_t e0 = (run.direct & 1u) ? 0 : run.nlo, e1 = (run.direct & 2u) ? run.cnt : run.nlo;
    c0 = c1 = 0;
    u = 0;
    if (e0 >= e1) return;
    u = (run.dest0 + e0) >> S.tile_shift;
    const uint64_t split = ((u + 1) << S.tile_shift) - run.dest0;
    c0 = (uint32_t)(split < e1 ? split : e1) - e0;
    c1 = e1 - e0 - c0;
}

struct ReadPart {  // c0 keys read from tile u, c1 from tile u + 1
    uint32_t u;
    uint16_t c0, c1;
};

struct GatherShared {
    StoreRun runs[kMaxTopRuns];
    ReadPart reads[kMaxTopRuns];
    uint32_t cum[kMaxTopRuns + 1];
    uint32_t nslots;
    int ok, ok1;  // warp 0's and warps 1..'s (no schedule error, no expired wait)
    Regime reg;
    ReadPart bulk;
};

// Warp 0: the tile's runs of top keys, one lane per slot: where each part is
// read from, and what it takes off the tiles it reads.  (Out of line: see
// btree_tile_runs_warp.)
static __device__ __noinline__ void btree_gather_runs_warp(const BtreeStream &S, uint64_t p0, uint64_t p1, uintptr_t ab,
                                                           uintptr_t sb, uint32_t kb, Ctrl *ctrl, GatherShared &gs) {
    const uint32_t lane = threadIdx.x;
    const uint64_t own = p0 >> S.tile_shift;
    TopGroup G0{}, G1{};
    const int ng = btree_stream_groups(S, p0, p1, G0, G1);
    const uint32_t h = S.g.h, nslots = (uint32_t)ng * h;
    uint32_t carry = 0;
    for (uint32_t s0 = 0; s0 < nslots; s0 += 32) {
        const uint32_t sl = s0 + lane;
        TopRun run{};
        if (sl < nslots) run = btree_group_run(S, sl < h ? G0 : G1, sl < h ? sl : sl - h, own);
        uint32_t incl = run.cnt;
#pragma unroll
        for (int dd = 1; dd < 32; dd <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, dd);
            if (lane >= (uint32_t)dd) incl += y;
        }
        if (S.plan == PLAN_O && run.cnt &&
            ((run.nlo && !(run.direct & 1u) && run.slo == kNoScratch) ||
             (run.nlo < run.cnt && !(run.direct & 2u) && run.shi == kNoScratch))) {
            btree_o_bad(ctrl);
            gs.ok = 0;
        }
        if (sl < nslots) {
            StoreRun sr;
            const uintptr_t d0 = (uintptr_t)run.dest0 * kb;
            sr.blo = (run.direct & 1u) ? ab + d0 : sb + d0 + (uintptr_t)run.slo * kb;
            sr.bhi = (run.direct & 2u) ? ab + d0 : sb + d0 + (uintptr_t)run.shi * kb;
            sr.off0 = run.off0;
            sr.mult = run.mult;
            sr.rb = run.rb;
            sr.nlo = run.nlo;
            gs.runs[sl] = sr;
            gs.cum[sl] = carry + incl - run.cnt;
            uint64_t u;
            uint32_t c0, c1;
            btree_run_reads(S, run, u, c0, c1);
            gs.reads[sl] = ReadPart{(uint32_t)u, (uint16_t)c0, (uint16_t)c1};
        }
        carry += __shfl_sync(0xFFFFFFFFu, incl, 31);
    }
    if (lane == 0) {
        gs.cum[nslots] = carry;
        gs.nslots = nslots;
    }
}

// A shared-memory slot with one padding key after every 32, so that keys
// placed at power-of-two strides (a BST's levels) spread over the banks.
__device__ __forceinline__ uint32_t gskew(uint32_t o) { return o + (o >> 5); }

// Keys of the tile buffer: the staged bulk keys (with up to a line of offset)
// and one slot per top key, or the whole tile in order.
static inline uint64_t btree_gather_keys(uint64_t tile_keys, uint64_t b, uint32_t key_bytes, uint32_t *top_at) {
    const uint64_t tops = tile_keys / (b + 1) + 2, bulk = tile_keys - tile_keys / (b + 1) + 2 + 128 / key_bytes;
    *top_at = (uint32_t)bulk;
    return std::max(bulk + tops + tops / 32 + 2, tile_keys + tile_keys / 32 + 2);
}

// The bulk keys of a boundary tile into the tile buffer, by warps 1..: four a
// thread at a time; a load has returned once its key is in shared memory, and a
// warp then takes off the layout keys it read, a subtraction a tile.  The lanes
// meet in between: the one that subtracts does so for keys that others loaded.
// (Out of line: its state would spill the common path's registers; 1.41 -> 1.67 ms
// on the 5e8-key B-tree.)
template <typename K, bool kCopy>
static __device__ __noinline__ void gather_boundary(const BtreeStream &S, const K *src, const K *scr, K *sm, uint64_t p0,
                                                    uint32_t cnt, Ctrl *ctrl, unsigned int *rem, int *ok) {
    const uint32_t tb = threadIdx.x - 32, nb = blockDim.x - 32, lane = tb & 31u;
    constexpr uint32_t kNone = 0xFFFFFFFFu;
    for (uint32_t b0 = tb & ~31u; b0 < cnt; b0 += 4 * nb) {
        K v[4];
        uint32_t from[4];  // the tile a layout key was read from
        uint32_t have = 0;
#pragma unroll
        for (int x = 0; x < 4; ++x) {
            const uint32_t o = b0 + x * nb + lane;
            from[x] = kNone;
            if (o >= cnt || btree_is_top(S, p0 + o)) continue;
            if (kCopy) {
                have |= 1u << x;
                v[x] = src[btree_pos(S.g, S.fd, p0 + o)];
            } else {
                uint64_t idx;
                const bool direct = btree_place(S, p0 + o, idx);
                if (!direct && idx >= S.nscratch) {
                    btree_o_bad(ctrl);
                    *ok = 0;
                    continue;
                }
                have |= 1u << x;
                v[x] = (direct ? src : scr)[idx];
                if (direct) from[x] = (uint32_t)(idx >> S.tile_shift);
            }
        }
#pragma unroll
        for (int x = 0; x < 4; ++x)
            if ((have >> x) & 1u) sm[gskew(b0 + x * nb + lane)] = v[x];
        if (kCopy) continue;
        __syncwarp();  // every lane's keys are in shared memory before any is taken off a count
#pragma unroll
        for (int x = 0; x < 4; ++x) {
            const uint32_t u = from[x];
            const unsigned act = __ballot_sync(0xFFFFFFFFu, u != kNone);
            if (u != kNone) {
                const unsigned same = __match_any_sync(act, u);
                if ((int)lane == __ffs(same) - 1) atomicSub(&rem[u], (unsigned)__popc(same));
            }
        }
    }
}

// The tile loop: tickets, or (kCopy) a grid stride.
template <bool kCopy>
__device__ __forceinline__ unsigned long long first_tile(Ctrl *ctrl, unsigned long long *s_ticket) {
    if constexpr (kCopy) return blockIdx.x;
    return ticket_first(ctrl, s_ticket);
}
template <bool kCopy>
__device__ __forceinline__ unsigned long long next_tile(unsigned long long t, const TicketPipe &tp,
                                                        unsigned long long *s_ticket) {
    if constexpr (kCopy) {
        __syncthreads();  // the block is done with the tile
        return t + gridDim.x;
    }
    return ticket_advance(tp, s_ticket);
}

// Named barrier among the threads of warps 1.. of the block.
__device__ __forceinline__ void bar_sync_tail() {
    asm volatile("bar.sync 1, %0;" ::"r"(blockDim.x - 32) : "memory");
}

// Sorted tile z of a B-tree or BST.  In most tiles (kinds 1 and 3) the bulk
// keys are one stretch of the layout (or of scratch, split at a tile boundary):
// cp.async copies it as it lies, at its own offset within a 128-byte line,
// while the top keys come run by run into slots of their own; the tile is put
// together as it is written, 16 bytes a thread.  Boundary tiles and the tail
// under the right-to-left schedule are gathered in order, key by key.
// kCopy: every key comes from a copy of the layout (scr, under the
// left-to-right schedule with every scratch slot at its final position), in any
// tile order, with nothing to count or wait for.
// kTops: top keys a thread loads at a time.  Where they are a ninth of the keys or
// more (b <= 8), four at 5 blocks an SM (48 registers): b = 8 over 6e7 u64 keys 220
// us against 226 with one at 6 blocks, b = 3 over 2^27 509 / 528, BST over 2^28 - 1
// 1126 / 1214; above, one at 6 blocks: b = 16 over 5e8 1403 against 1491 us.  From a
// copy two at a time (one call, four / one / two / eight: BST over 1.7e7 u32 keys 98 /
// 104 / 92 / 108, over 4e7 184 / 184 / 171 / 202, b = 8 over 3.4e7 133 / - / 128 / -).
template <typename K, bool kCopy, int kTops>
__global__ void __launch_bounds__(kGatherThreads, kTops == 1 ? kGatherBlocksPerSM : kGatherBlocksPerSM - 1)
btree_unstream_kernel(K *__restrict__ A, const K *__restrict__ scr, const __grid_constant__ BtreeStream S,
                      uint32_t top_at, Ctrl *ctrl, WaitCfg wc, unsigned int *rem) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    K *sm = tile_smem<K>(smem_raw);
    K *top = sm + top_at;
    const K *src = kCopy ? scr : A;  // where the layout is read
    __shared__ unsigned long long s_ticket;
    __shared__ GatherShared gs;
    __shared__ uint32_t s_stage[2];  // the staged stretch: its offset in the buffer, its first index - dbase
    TicketPipe tp;
    for (unsigned long long t = first_tile<kCopy>(ctrl, &s_ticket); t < S.ntiles;
         t = next_tile<kCopy>(t, tp, &s_ticket)) {
        if (!kCopy) ticket_claim(ctrl, tp);
        const uint64_t k = kCopy ? t : btree_tile_of_ticket(S, S.ntiles - 1 - t);
        uint64_t p0, p1;
        btree_tile(S, k, p0, p1);
        const uint32_t cnt = (uint32_t)(p1 - p0);
        uint32_t ph = 0, j0 = 0;
        if (threadIdx.x < 32) {
            if (threadIdx.x == 0) gs.ok = 1;  // the previous tile's readers are past the ticket barrier
            __syncwarp();
            btree_gather_runs_warp(S, p0, p1, reinterpret_cast<uintptr_t>(src), reinterpret_cast<uintptr_t>(scr),
                                   (uint32_t)sizeof(K), ctrl, gs);
        } else {
            const uint32_t tb = threadIdx.x - 32, nb = blockDim.x - 32;
            if (tb == 0) {
                gs.ok1 = 1;
                gs.reg = btree_stream_regime(S, p0, p1);
            }
            bar_sync_tail();
            const Regime &R = gs.reg;
            if (R.kind == 1 || R.kind == 3) {
                uint32_t len;
                btree_bulk_indices(S, R, cnt, j0, len);
                const uint64_t i0 = R.dbase + j0;
                // indices below lo_len of the stretch, and the rest
                const uint32_t lo_len =
                    R.kind == 1 || R.dsplit >= i0 + len ? len : R.dsplit <= i0 ? 0u : (uint32_t)(R.dsplit - i0);
                const bool lo_A = R.to_A, hi_A = R.kind == 3 && R.hi_A;
                const bool bad = R.kind == 3 && !btree_regime_ok(S, R, cnt);
                if (!bad) {
                    const K *lo = (lo_A ? src : scr) + i0 + (R.kind == 3 ? (uint64_t)R.slo : 0ull);
                    ph = (uint32_t)(reinterpret_cast<uintptr_t>(lo) & 127) / (uint32_t)sizeof(K);
                    const K *hi = (hi_A ? src : scr) + i0 + lo_len + (R.kind == 3 ? (uint64_t)R.shi : 0ull);
                    if (lo_len == 0) ph = (uint32_t)(reinterpret_cast<uintptr_t>(hi) & 127) / (uint32_t)sizeof(K);
                    if (lo_len) stage_run(lo, lo_len, sm + ph, tb, nb);
                    if (lo_len < len) stage_run(hi, len - lo_len, sm + ph + lo_len, tb, nb);
                }
                if (tb == 0) {
                    if (bad) {
                        btree_o_bad(ctrl);
                        gs.ok1 = 0;
                    }
                    // what was read straight from the layout, by tile
                    uint64_t a = i0, e = i0 + len;
                    if (!lo_A) a = i0 + lo_len;
                    if (R.kind == 3 && !hi_A) e = i0 + lo_len;
                    gs.bulk = ReadPart{0, 0, 0};
                    if (a < e) {
                        const uint64_t u = a >> S.tile_shift, m = min(e, (u + 1) << S.tile_shift);
                        gs.bulk = ReadPart{(uint32_t)u, (uint16_t)(m - a), (uint16_t)(e - m)};
                    }
                }
            } else {
                if (tb == 0) gs.bulk = ReadPart{0, 0, 0};
                if (R.kind == 0) gather_boundary<K, kCopy>(S, src, scr, sm, p0, cnt, ctrl, rem, &gs.ok1);
            }
        }
        __syncthreads();  // the runs and the regime are known
        const Regime &R = gs.reg;
        const bool staged = R.kind == 1 || R.kind == 3;
        const uint32_t d = S.fd32.d, r0 = R.r0, skip = R.skip;
        if (gs.ok && gs.ok1) {
            const uint32_t total = gs.cum[gs.nslots];
            uint32_t r = 0;  // the run of gi only moves forward as gi grows
            for (uint32_t g0 = threadIdx.x; g0 < total; g0 += kTops * kGatherThreads) {
                K v[kTops];
                uint32_t at[kTops];
#pragma unroll
                for (int x = 0; x < kTops; ++x) {
                    const uint32_t gi = g0 + x * kGatherThreads;
                    if (gi < total) {
                        while (gi >= gs.cum[r + 1]) ++r;
                        const StoreRun &run = gs.runs[r];
                        const uint32_t e = gi - gs.cum[r];
                        v[x] = reinterpret_cast<const K *>(e < run.nlo ? run.blo : run.bhi)[e];
                        const uint32_t off = btree_top_item_off(S, run, e);
                        at[x] = staged ? top_at + gskew(S.fd32.div(r0 + off)) : gskew(off);
                    }
                }
#pragma unroll
                for (int x = 0; x < kTops; ++x)
                    if (g0 + x * kGatherThreads < total) sm[at[x]] = v[x];
            }
        }
        load_tile_wait();
        if (threadIdx.x == 32) {
            s_stage[0] = ph;
            s_stage[1] = j0;
        }
        __syncthreads();  // every key has been read
        if (!kCopy && threadIdx.x < 32) {
            if (gs.ok && gs.ok1) {
                const uint32_t lane = threadIdx.x;
                for (uint32_t s0 = 0; s0 < gs.nslots; s0 += 32) {
                    const ReadPart rp = s0 + lane < gs.nslots ? gs.reads[s0 + lane] : ReadPart{0, 0, 0};
                    // the upper levels share tiles: one subtraction a tile
                    const unsigned act = __ballot_sync(0xFFFFFFFFu, rp.c0 != 0);
                    if (rp.c0) {
                        const unsigned same = __match_any_sync(act, rp.u);
                        const unsigned sum = __reduce_add_sync(same, (unsigned)rp.c0);
                        if ((int)lane == __ffs(same) - 1) atomicSub(&rem[rp.u], sum);
                    }
                    if (rp.c1) atomicSub(&rem[rp.u + 1], (unsigned)rp.c1);
                }
                if (lane == 0 && gs.bulk.c0) atomicSub(&rem[gs.bulk.u], (unsigned)gs.bulk.c0);
                if (lane == 1 && gs.bulk.c1) atomicSub(&rem[gs.bulk.u + 1], (unsigned)gs.bulk.c1);
                __syncwarp();
                if (lane == 0 && !wait_flag(&rem[k], wc.wait_value, ctrl, wc)) gs.ok = 0;
            }
        }
        if (!kCopy) __syncthreads();
        if (!gs.ok || !gs.ok1) continue;
        K *out = A + p0;
        if (staged) {
            constexpr uint32_t V = 16 / sizeof(K);
            const K *bulk = sm + s_stage[0] - (int64_t)s_stage[1];  // bulk[v - ql]
            const uint32_t vecs = (reinterpret_cast<uintptr_t>(out) & 15) == 0 ? cnt / V : 0;
            for (uint32_t w = threadIdx.x; w < vecs; w += kGatherThreads) {
                uint32_t v = r0 + w * V;
                uint32_t ql = S.fd32.div(v), m = v - ql * d;
                uint4 x;
                K *kx = reinterpret_cast<K *>(&x);
#pragma unroll
                for (uint32_t e = 0; e < V; ++e) {
                    kx[e] = m == skip ? top[gskew(ql)] : bulk[v - ql];
                    ++v;
                    if (++m == d) {
                        m = 0;
                        ++ql;
                    }
                }
                reinterpret_cast<uint4 *>(out)[w] = x;
            }
            for (uint32_t o = vecs * V + threadIdx.x; o < cnt; o += kGatherThreads) {
                const uint32_t v = r0 + o, ql = S.fd32.div(v);
                out[o] = v - ql * d == skip ? top[gskew(ql)] : bulk[v - ql];
            }
        } else {
            for (uint32_t o = threadIdx.x; o < cnt; o += kGatherThreads) out[o] = sm[gskew(o)];
        }
    }
}

// Sorted tile k of an mvEB or standard vEB.  Units that follow one another in
// the tile mostly follow one another in the layout, so a tile's bodies are a few
// stretches of it: each is copied by cp.async as it lies, and a thread then
// writes the same rank of every unit (unit sizes divide the block), its slot in
// the unit looked up once per unit height.  Tiles with more stretches or units
// than the tables hold are gathered key by key.
constexpr uint32_t kGatherUnits = 256, kGatherStretches = 24;

template <typename K>
static inline uint64_t mveb_gather_keys(uint64_t tile_keys) {
    return tile_keys + (kGatherStretches + 1) * (128 / sizeof(K)) / 4 + 128 / sizeof(K);
}

template <typename K, bool kCopy>
__global__ void __launch_bounds__(kGatherThreads, kGatherBlocksPerSM)
mveb_unstream_kernel(K *__restrict__ A, const K *__restrict__ scr, const __grid_constant__ MvebParams prm, Ctrl *ctrl,
                     WaitCfg wc, unsigned int *rem) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    K *sm = tile_smem<K>(smem_raw);
    const K *src = kCopy ? scr : A;  // where the layout is read
    __shared__ unsigned long long s_ticket;
    __shared__ unsigned long long s_from[kGatherStretches];
    __shared__ uint32_t s_at[kGatherStretches], s_len[kGatherStretches], s_n;
    __shared__ uint16_t s_unit[kGatherUnits];  // where each unit starts in the buffer
    __shared__ K s_sep[kGatherUnits];
    __shared__ unsigned char s_slot[256];  // sorted rank in a unit -> its slot
    __shared__ int s_ok;
    const MvebPlan &P = prm.plan;
    constexpr uint32_t V = 16 / sizeof(K), kMany = 0xFFFFFFFFu;
    uint32_t U = 0, slot = 0;
    TicketPipe tp;
    for (unsigned long long t = first_tile<kCopy>(ctrl, &s_ticket); t < P.total_tiles;
         t = next_tile<kCopy>(t, tp, &s_ticket)) {
        if (!kCopy) ticket_claim(ctrl, tp);
        const uint64_t k = t;  // the forward pass takes the tiles from the last
        int ri;
        uint64_t p0, p1;
        mveb_tile(P, k, ri, p0, p1);
        const MvebRegion &R = P.reg[ri];
        const uint32_t cnt = (uint32_t)(p1 - p0);
        if (R.U && R.U != U) {  // block-uniform
            U = R.U;
            const uint32_t u = (1u << U) - 1;
            if (threadIdx.x < u) s_slot[prm.inv[unit_table_off(U) + threadIdx.x]] = (unsigned char)threadIdx.x;
            __syncthreads();
            slot = (threadIdx.x & u) < u ? s_slot[threadIdx.x & u] : u;  // the last of a unit: its separator
        }
        const uint32_t u = (1u << U) - 1;
        uint64_t g0 = 0, g1 = 0;
        if (R.U) mveb_tile_groups(R, p0, p1, g0, g1);
        const uint32_t ng = (uint32_t)(g1 - g0);
        const uint32_t seps = R.U ? (uint32_t)min((uint64_t)ng, (R.len - (g0 << U)) >> U) : 0;
        if (threadIdx.x < 32) {  // warp 0: the stretches
            const uint32_t lane = threadIdx.x;
            uint32_t ns = 0, at = 0, first = 0;  // stretches so far; the buffer's end; the current stretch's first unit
            uint64_t next = ~0ull;               // where the last unit's stretch goes on
            if (ng > kGatherUnits) ns = kMany;
            for (uint32_t j0 = 0; j0 < ng && ns != kMany; j0 += 32) {
                const uint32_t j = j0 + lane, m = min(32u, ng - j0);
                const uint64_t dst = j < ng ? mveb_unit_dst(R, g0 + j) : 0;
                uint64_t prev = __shfl_up_sync(0xFFFFFFFFu, dst, 1) + u;
                if (lane == 0) prev = next;
                unsigned starts = __ballot_sync(0xFFFFFFFFu, j < ng && dst != prev);
                uint32_t done = 0;  // units of this batch placed
                while (starts) {
                    const uint32_t b = __ffs(starts) - 1;
                    starts &= starts - 1;
                    at += (b - done) * u;  // the units before it go on with their stretch
                    if (lane >= done && lane < b) s_unit[j0 + lane] = (uint16_t)(at - (b - lane) * u);
                    if (ns == kGatherStretches) {
                        ns = kMany;
                        break;
                    }
                    if (lane == 0 && ns) s_len[ns - 1] = (j0 + b - first) * u;
                    const uint64_t d0 = __shfl_sync(0xFFFFFFFFu, dst, b);
                    // the first stretch keeps its offset within a line, the others within 16 bytes
                    const uint32_t ph = (uint32_t)(reinterpret_cast<uintptr_t>(src + d0) / sizeof(K)) & (ns ? V - 1 : 128 / (uint32_t)sizeof(K) - 1);
                    at = (at + V - 1) / V * V + ph;
                    if (lane == 0) {
                        s_from[ns] = d0;
                        s_at[ns] = at;
                    }
                    first = j0 + b;
                    ++ns;
                    done = b;
                }
                if (ns == kMany) break;
                at += (m - done) * u;
                if (lane >= done && lane < m) s_unit[j0 + lane] = (uint16_t)(at - (m - lane) * u);
                next = __shfl_sync(0xFFFFFFFFu, dst, m - 1) + u;
            }
            if (lane == 0) {
                if (ns && ns != kMany) s_len[ns - 1] = (ng - first) * u;
                s_n = ns;
                s_ok = 1;
            }
        }
        __syncthreads();
        const uint32_t ns = s_n;
        if (ns != kMany) {
            for (uint32_t s = 0; s < ns; ++s) stage_run(src + s_from[s], s_len[s], sm + s_at[s], threadIdx.x, kGatherThreads);
            if (threadIdx.x < seps)
                s_sep[threadIdx.x] = kCopy ? src[veb_pos(P.n, p0 + (((uint64_t)threadIdx.x << U) + u), P.modified != 0)]
                                           : scr[R.slot_base + g0 + threadIdx.x];
            if (R.U == 0)
                for (uint32_t o = threadIdx.x; o < cnt; o += kGatherThreads)
                    sm[o] = kCopy ? src[veb_pos(P.n, p0 + o, P.modified != 0)] : scr[R.slot_base + (p0 - R.src) + o];
        } else {
            for (uint32_t o = threadIdx.x; o < cnt; o += kGatherThreads) {
                const uint32_t j = o >> U, q = o & u;
                if (kCopy)
                    sm[o] = src[veb_pos(P.n, p0 + o, P.modified != 0)];
                else
                    sm[o] = q == u ? scr[R.slot_base + g0 + j] : src[mveb_unit_dst(R, g0 + j) + s_slot[q]];
            }
        }
        load_tile_wait();
        __syncthreads();  // every key has been read
        if (!kCopy && threadIdx.x < 32) {
            const uint32_t parts = ns == kMany ? ng : ns;
            for (uint32_t s = threadIdx.x; s < parts; s += 32) {
                uint64_t a = ns == kMany ? mveb_unit_dst(R, g0 + s) : s_from[s];
                uint64_t left = ns == kMany ? u : s_len[s];
                while (left) {
                    const uint64_t f = mveb_tile_of(P, a);
                    int fi;
                    uint64_t f0, f1;
                    mveb_tile(P, f, fi, f0, f1);
                    const uint64_t c = min(left, f1 - a);
                    atomicSub(&rem[f], (unsigned int)c);
                    a += c;
                    left -= c;
                }
            }
            __syncwarp();
            if (threadIdx.x == 0 && !wait_flag(&rem[k], wc.wait_value, ctrl, wc)) s_ok = 0;
        }
        if (!kCopy) __syncthreads();
        if (!s_ok) continue;
        K *out = A + p0;
        if (R.U && ns != kMany) {
            const uint32_t q = threadIdx.x & u, step = kGatherThreads >> U;
            out += threadIdx.x & ((1u << U) - 1);
            if (q < u) {
#pragma unroll 4
                for (uint32_t j = threadIdx.x >> U; j < ng; j += step) out[j << U] = sm[s_unit[j] + slot];
            } else {
                for (uint32_t j = threadIdx.x >> U; j < seps; j += step) out[j << U] = s_sep[j];
            }
        } else {
            for (uint32_t o = threadIdx.x; o < cnt; o += kGatherThreads) out[o] = sm[o];
        }
    }
}

// B-trees and BSTs of a few megabytes: a thread a key from the copy.
template <typename K>
__global__ void __launch_bounds__(kGatherThreads)
btree_gather_keys_kernel(K *__restrict__ A, const K *__restrict__ C, uint64_t n, const __grid_constant__ KeysGeometry kg) {
    const uint64_t x = (uint64_t)blockIdx.x * kGatherThreads + threadIdx.x;
    if (x < n) A[x] = __ldg(C + btree_pos(kg.g, kg.fd, x));
}

// ---------------------------------------------------------------- host side
static inline uint64_t align256(uint64_t x) { return (x + 255) / 256 * 256; }

// How an array of `bytes` goes back: key by key from a copy of the layout,
// tile by tile from a copy, or in place.  Measured on B200 (us, key by key / from
// a copy / in place): B-tree b = 16 u64 of 8 MB 18 / 24 / 45, 16 MB 22 / 26 / 48,
// 64 MB 72 / 60 / 66, 128 MB 136 / 107 / 102, 256 MB 260 / 192 / 162; b = 2 u32 of
// 8 MB 29 / 29 / 56, 256 MB 610 / 256 / 272; BST u64 of 16 MB 23 / 24 / 34, 256 MB
// 252 / 214 / 219 on the fixed directions (39 % of its keys take scratch), 2 GB
// on the ordered schedule 1129 in place; one call's wall time of an
// mvEB from a copy / in place: u64 of 32 MB 43 / 57, 48 MB 53 / 59, 64 MB 70 / 67,
// 96 MB 91 / 83, u32 of 48 MB 57 / 61, 64 MB 76 / 71; standard vEB u32 of 48 MB 63 /
// 81, 64 MB 81 / 85.
// (Key by key: permute_by_keys, decided before there is a plan.)
enum ReverseForm { REVERSE_KEYS, REVERSE_COPY, REVERSE_IN_PLACE };
// Workspace of the in-place form: the scratch (starting at the array's own offset
// within a line), the tiles' counts, the control block.
struct ReverseSpace {
    uint64_t off_rem, off_ctrl, bytes;
};
static ReverseSpace reverse_space(const PermutePlan &pl) {
    ReverseSpace r;
    r.off_rem = align256(pl.scratch_keys * pl.key_bytes + 128);
    r.off_ctrl = r.off_rem + align256(pl.ntiles * sizeof(unsigned int));
    r.bytes = r.off_ctrl + align256(sizeof(Ctrl));
    return r;
}

// Decided before there is a plan: the copy form takes the fixed-direction one,
// whose geometry is all that it reads.  (The ordered plan's tables would take a
// first call 0.2 to 0.5 ms, where the copy of 16 to 192 MB takes 0.05 to 0.3, and
// a place in the library's cache of them.)
static bool reverse_copies(int layout, uint64_t n, uint64_t b, uint32_t key_bytes) {
    const uint64_t bytes = n * key_bytes;
    if (is_veb_layout(layout)) return bytes <= (56ull << 20);
    if (layout == TL_LAYOUT_BTREE && b > 1) return bytes <= (192ull << 20);
    return !permute_takes_order(layout, n, b, key_bytes);
}

static ReverseForm reverse_form(const PermutePlan &pl) {
    // a BST whose tables could not be had; a schedule whose scratch is about as large as the array gains nothing
    if (pl.b == 1 && !is_veb_layout(pl.layout) && !pl.ordered) return REVERSE_COPY;
    return reverse_space(pl).bytes <= align256(pl.n * pl.key_bytes) ? REVERSE_IN_PLACE : REVERSE_COPY;
}

// A copy of the array, whatever the form takes of it.
int unpermute_workspace_bytes(int layout, uint64_t n, uint64_t b, uint32_t key_bytes, uint64_t *bytes) {
    if (!bytes) return TL_ERROR_INVALID_VALUE;
    uint64_t fixed = 0;
    const int rc = permute_workspace_bytes_fixed(layout, n, b, key_bytes, &fixed);  // the arguments' checks
    if (rc) return rc;
    *bytes = align256(n * key_bytes);
    return TL_SUCCESS;
}

static int g_gather_sms = 0;
static std::once_flag g_gather_once;
static int gather_sms() {
    std::call_once(g_gather_once, [] {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&g_gather_sms, cudaDevAttrMultiProcessorCount, dev);
        if (g_gather_sms <= 0) g_gather_sms = 148;
    });
    return g_gather_sms;
}

// Blocks of a persistent launch over the tiles.  The limit is the same for every
// call: one thread's smaller need (another b) must not lower it under another's launch.
constexpr size_t kGatherSmemMax = 40 * 1024;
template <typename Kern>
static int gather_grid(Kern kern, size_t smem, uint64_t ntiles, unsigned *grid) {
    if (smem > kGatherSmemMax) return TL_ERROR_UNSUPPORTED;  // (a 32 KB tile and its padding: never)
    TL_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGatherSmemMax));
    int per_sm = 0;
    TL_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kGatherThreads, smem));
    *grid = (unsigned)std::min<uint64_t>((uint64_t)std::max(per_sm, 1) * gather_sms(), ntiles);
    return TL_SUCCESS;
}

template <typename K>
static int launch_from_copy(const PermutePlan &pl, const KeysGeometry &kg, ReverseForm form, uint64_t n, K *A,
                            char *ws, cudaStream_t st) {
    K *C = reinterpret_cast<K *>(ws);
    TL_CUDA_TRY(cudaMemcpyAsync(C, A, n * sizeof(K), cudaMemcpyDeviceToDevice, st));
    unsigned grid = 1;
    int rc = TL_SUCCESS;
    if (form == REVERSE_KEYS) {
        grid = (unsigned)((n + kGatherThreads - 1) / kGatherThreads);
        btree_gather_keys_kernel<K><<<grid, kGatherThreads, 0, st>>>(A, C, n, kg);
    } else if (is_veb_layout(pl.layout)) {
        auto kern = mveb_unstream_kernel<K, true>;
        const size_t smem = mveb_gather_keys<K>(pl.tile_keys) * sizeof(K) + 128;
        rc = gather_grid(kern, smem, pl.ntiles, &grid);
        if (rc) return rc;
        kern<<<grid, kGatherThreads, smem, st>>>(A, C, pl.mp, nullptr, WaitCfg{}, nullptr);
    } else {
        uint32_t top_at = 0;
        const size_t smem = btree_gather_keys(pl.tile_keys, pl.b, sizeof(K), &top_at) * sizeof(K) + 128;
        auto kern = pl.b <= 8 ? btree_unstream_kernel<K, true, 2> : btree_unstream_kernel<K, true, 1>;
        rc = gather_grid(kern, smem, pl.ntiles, &grid);
        if (rc) return rc;
        BtreeStream S = pl.bs;  // left to right with slots at their positions: last-level and tail tiles are staged
        S.plan = PLAN_L;
        S.seg1 = S.g.ni;
        S.nscratch = pl.n;
        kern<<<grid, kGatherThreads, smem, st>>>(A, C, S, top_at, nullptr, WaitCfg{}, nullptr);
    }
    TL_CUDA_TRY(cudaGetLastError());
    return TL_SUCCESS;
}

template <typename K>
static int launch_in_place(const PermutePlan &pl, K *A, char *ws, cudaStream_t st) {
    const ReverseSpace sp = reverse_space(pl);
    K *scr = reinterpret_cast<K *>(ws + (reinterpret_cast<uintptr_t>(A) & 127));
    unsigned int *rem = reinterpret_cast<unsigned int *>(ws + sp.off_rem);
    Ctrl *ctrl = reinterpret_cast<Ctrl *>(ws + sp.off_ctrl);
    WaitCfg wc;
    wc.flag_value = 0;
    wc.wait_value = debug_force_timeout() ? 0xFFFFFFFFu : 0u;  // forced: no count ever gets there
    wc.spin_limit = debug_spin_limit();
    const int smx = gather_sms();
    const unsigned ig = (unsigned)((pl.ntiles + 255) / 256);
    unsigned grid = 1;
    if (is_veb_layout(pl.layout)) {
        mveb_reverse_init_kernel<<<ig, 256, 0, st>>>(rem, pl.mp, ctrl);
        if (pl.scratch_keys) {
            const unsigned sg = (unsigned)std::min<uint64_t>((pl.scratch_keys + kScatterThreads - 1) / kScatterThreads,
                                                             (uint64_t)smx * 8);
            mveb_save_kernel<K><<<sg, kScatterThreads, 0, st>>>(scr, A, pl.mp, rem);
        }
        auto kern = mveb_unstream_kernel<K, false>;
        const size_t smem = mveb_gather_keys<K>(pl.tile_keys) * sizeof(K) + 128;
        const int rc = gather_grid(kern, smem, pl.ntiles, &grid);
        if (rc) return rc;
        kern<<<grid, kGatherThreads, smem, st>>>(A, scr, pl.mp, ctrl, wc, rem);
    } else {
        BulkPlan bp;
        int rc = make_bulk_plan(pl.bs, pl.ot, A, scr, bp);
        if (rc) return rc;
        SavedRanges sr;
        sr.nr = bp.nr;
        for (int r = 0; r < bp.nr; ++r) {
            sr.lo[r] = bp.r[r].key_dst;
            sr.hi[r] = bp.r[r].key_dst + bp.r[r].len;
            std::swap(bp.r[r].dst, bp.r[r].src);  // saved: from the array to the scratch
            std::swap(bp.r[r].key_dst, bp.r[r].key_src);
        }
        btree_reverse_init_kernel<<<ig, 256, 0, st>>>(rem, pl.n, pl.bs.tile_shift, sr, ctrl);
        if (pl.ordered && pl.ot.nsegs) {
            const unsigned fg = (unsigned)std::min<uint64_t>((pl.ot.nsegs * 32 + kScatterThreads - 1) / kScatterThreads,
                                                             (uint64_t)smx * 8);
            btree_fix_save_kernel<K><<<fg, kScatterThreads, 0, st>>>(scr, A, pl.ot.segs, pl.ot.nsegs, pl.bs.tile_shift,
                                                                   rem);
        }
        if (bp.nr) {
            const size_t smem = (size_t)kBulkStages * kBulkChunk;
            auto ck = btree_save_kernel<K>;
            TL_CUDA_TRY(cudaFuncSetAttribute(ck, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            int cper = 0;
            TL_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&cper, ck, 32, smem));
            const uint64_t cg = std::max<uint64_t>(1, std::min<uint64_t>(bp.nchunks, (uint64_t)std::max(cper, 1) * smx));
            ck<<<(unsigned)cg, 32, smem, st>>>(scr, A, bp, ctrl);
        }
        uint32_t top_at = 0;
        const size_t smem = btree_gather_keys(pl.tile_keys, pl.b, sizeof(K), &top_at) * sizeof(K) + 128;
        auto kern = pl.b <= 8 ? btree_unstream_kernel<K, false, 4> : btree_unstream_kernel<K, false, 1>;
        rc = gather_grid(kern, smem, pl.ntiles, &grid);
        if (rc) return rc;
        kern<<<grid, kGatherThreads, smem, st>>>(A, scr, pl.bs, top_at, ctrl, wc, rem);
    }
    TL_CUDA_TRY(cudaGetLastError());
    return TL_SUCCESS;
}

int unpermute(int layout, void *dev_A, uint64_t n, uint64_t b, uint32_t key_bytes, void *dev_ws, uint64_t ws_bytes,
              cudaStream_t st, float *ms) {
    if (n > 0 && !dev_A) return TL_ERROR_INVALID_VALUE;
    if (reinterpret_cast<uintptr_t>(dev_A) % (key_bytes ? key_bytes : 1)) return TL_ERROR_INVALID_VALUE;
    if (dev_ws && reinterpret_cast<uintptr_t>(dev_ws) % 256) return TL_ERROR_INVALID_VALUE;
    KeysGeometry kg;
    const bool by_keys = permute_by_keys(layout, n, b, key_bytes, kg);
    PermutePlan pl;
    const bool copies = by_keys || reverse_copies(layout, n, b, key_bytes);
    int rc = by_keys  ? TL_SUCCESS
             : copies ? permute_plan_fixed(layout, n, b, key_bytes, pl)
                      : permute_plan_device(layout, n, b, key_bytes, st, pl);
    if (rc) return rc;
    if (n <= 1) {
        if (ms) *ms = 0.f;
        return TL_SUCCESS;
    }
    const ReverseForm form = by_keys ? REVERSE_KEYS : copies ? REVERSE_COPY : reverse_form(pl);
    const bool in_place = form == REVERSE_IN_PLACE;
    if (dev_ws && ws_bytes < align256(n * key_bytes)) return TL_ERROR_WORKSPACE_TOO_SMALL;
    const uint64_t need = in_place ? reverse_space(pl).bytes : align256(n * key_bytes);
    EventTimer timer(ms != nullptr, st);
    char *ws = static_cast<char *>(dev_ws);
    bool owned = false;
    bool pooled = false;
    if (!ws) {
        ws = static_cast<char *>(workspace_acquire(need));
        if (ws) {
            owned = true;
        } else {  // the cache could not help: a stream-ordered allocation
            keep_pool_memory();
            if (cudaMallocAsync(reinterpret_cast<void **>(&ws), need, st) != cudaSuccess) {
                record_cuda_error(cudaGetLastError());
                return TL_ERROR_OUT_OF_MEMORY;
            }
            owned = pooled = true;
        }
    }
    timer.start();
    if (!in_place)
        rc = key_bytes == 8 ? launch_from_copy<uint64_t>(pl, kg, form, n, static_cast<uint64_t *>(dev_A), ws, st)
                            : launch_from_copy<uint32_t>(pl, kg, form, n, static_cast<uint32_t *>(dev_A), ws, st);
    else
        rc = key_bytes == 8 ? launch_in_place<uint64_t>(pl, static_cast<uint64_t *>(dev_A), ws, st)
                            : launch_in_place<uint32_t>(pl, static_cast<uint32_t *>(dev_A), ws, st);
    timer.stop();
    unsigned int err = 0;
    if (rc == TL_SUCCESS && in_place)
        rc = read_ctrl(reinterpret_cast<const Ctrl *>(ws + reverse_space(pl).off_ctrl), &err, st);
    if (owned && pooled) cudaFreeAsync(ws, st);
    if (rc == TL_SUCCESS) rc = sync_and_check(st);
    if (owned && !pooled) {
        if (rc != TL_SUCCESS) cudaStreamSynchronize(st);  // nothing of this call may still use it
        workspace_release(ws);
    }
    // a bounded wait expired, or (never expected) the schedule was inconsistent
    if (rc == TL_SUCCESS && err) rc = (err & (1u << TL_ERROR_TIMEOUT)) ? TL_ERROR_TIMEOUT : TL_ERROR_UNSUPPORTED;
    if (rc == TL_SUCCESS && ms) *ms = timer.elapsed();
    return rc;
}

// Host replay of the save pass and the tiles in ticket order, with the kernels'
// per-tile helpers, at one schedule.  False on any violation: a tile that reads
// an overwritten position or an unsaved slot, counts that do not come out at
// zero when the tile is stored, a position written other than once.
static bool replay_reverse(const PermutePlan &pl, std::vector<uint64_t> &A) {
    const uint64_t n = pl.n;
    std::vector<uint64_t> scr(pl.scratch_keys, 0);
    std::vector<uint8_t> saved(pl.scratch_keys, 0), over(n, 0);
    std::vector<int64_t> rem(pl.ntiles, 0);
    bool ok = true;
    const bool veb = is_veb_layout(pl.layout);
    const MvebPlan &P = pl.mp.plan;
    const BtreeStream &S = pl.bs;
    auto tile_of = [&](uint64_t p) { return veb ? mveb_tile_of(P, p) : p >> S.tile_shift; };
    for (uint64_t k = 0; k < pl.ntiles; ++k) {
        int ri;
        uint64_t p0, p1;
        if (veb) mveb_tile(P, k, ri, p0, p1); else btree_tile(S, k, p0, p1);
        rem[k] = (int64_t)(p1 - p0);
    }
    auto save = [&](uint64_t s, uint64_t p) {
        if (s >= scr.size() || p >= n || saved[s]) { ok = false; return; }
        scr[s] = A[p];
        saved[s] = 1;
        --rem[tile_of(p)];
    };
    if (veb) {
        for (uint64_t s = 0; s < P.total_slots; ++s) {
            const uint64_t rank = mveb_slot_rank(P, s);
            if (rank != ~0ull) save(s, veb_pos(n, rank, P.modified != 0));
        }
    } else if (pl.ordered) {
        for (uint64_t i = 0; i < pl.ot.nranges; ++i)
            for (uint64_t p = (uint64_t)pl.ot.ranges[i].x << S.tile_shift, s = (uint64_t)pl.ot.ranges[i].z << S.tile_shift;
                 p < std::min<uint64_t>((uint64_t)pl.ot.ranges[i].y << S.tile_shift, n); ++p, ++s)
                save(s, p);
        for (uint64_t i = 0; i < pl.ot.nsegs; ++i)
            for (uint64_t e = 0; e < pl.ot.segs[i].dst_len >> 48; ++e)
                save(pl.ot.segs[i].src + e, (pl.ot.segs[i].dst_len & kSegDstMask) + e);
    } else {
        for (int j = 0; j < btree_copy_range_count(S); ++j) {
            CopyRange r;
            if (!btree_copy_range(S, j, r)) continue;
            for (uint64_t e = 0; e < r.len; ++e) save(r.src + e, r.dst + e);
        }
    }
    std::vector<uint64_t> tile(pl.tile_keys);
    std::vector<uint8_t> got(pl.tile_keys);
    for (uint64_t t = 0; t < pl.ntiles && ok; ++t) {
        const uint64_t k = veb ? t : btree_tile_of_ticket(S, pl.ntiles - 1 - t);
        int ri = 0;
        uint64_t p0, p1;
        if (veb) mveb_tile(P, k, ri, p0, p1); else btree_tile(S, k, p0, p1);
        const uint32_t cnt = (uint32_t)(p1 - p0);
        std::fill(got.begin(), got.end(), 0);
        auto put = [&](uint64_t o, uint64_t v) {
            if (o >= cnt || got[o]) { ok = false; return; }
            tile[o] = v;
            got[o] = 1;
        };
        auto direct = [&](uint64_t o, uint64_t p) {
            if (p >= n || over[p]) { ok = false; return; }
            put(o, A[p]);
            --rem[tile_of(p)];
        };
        auto from_scratch = [&](uint64_t o, uint64_t s) {
            if (s >= scr.size() || !saved[s]) { ok = false; return; }
            put(o, scr[s]);
        };
        if (veb) {
            const MvebRegion &R = P.reg[ri];
            if (R.U == 0) {
                for (uint32_t o = 0; o < cnt; ++o) from_scratch(o, R.slot_base + (p0 - R.src) + o);
            } else {
                const unsigned char *inv = pl.mp.inv + unit_table_off(R.U);
                const uint64_t u = (1ull << R.U) - 1;
                uint64_t g0, g1;
                mveb_tile_groups(R, p0, p1, g0, g1);
                for (uint64_t g = g0; g < g1; ++g) {
                    const uint64_t o = (g - g0) << R.U;
                    for (uint64_t q = 0; q < u; ++q) direct(o + inv[q], mveb_unit_dst(R, g) + q);
                    if (g - g0 < std::min<uint64_t>(g1 - g0, (R.len - (g0 << R.U)) >> R.U))
                        from_scratch(o + u, R.slot_base + g);
                }
            }
        } else {
            const Regime RG = btree_stream_regime(S, p0, p1);
            if (RG.kind == 0) {
                for (uint64_t x = p0; x < p1; ++x) {
                    uint64_t idx;
                    if (btree_is_top(S, x)) continue;
                    if (btree_place(S, x, idx)) direct(x - p0, idx); else from_scratch(x - p0, idx);
                }
            } else if (RG.kind != 2) {
                uint32_t j0, len;
                btree_bulk_indices(S, RG, cnt, j0, len);
                uint32_t seen = 0;
                for (uint32_t o = 0; o < cnt; ++o) {
                    uint64_t idx;
                    if (!btree_regime_bulk(S, RG, o, idx)) continue;
                    if (idx != RG.dbase + j0 + seen++) ok = false;  // one stretch
                    const bool hi = RG.kind == 3 && idx >= RG.dsplit;
                    if (hi ? RG.hi_A : RG.to_A) direct(o, idx);
                    else from_scratch(o, RG.kind == 3 ? idx + (uint64_t)(hi ? RG.shi : RG.slo) : idx);
                }
                if (seen != len) ok = false;
            }
            TopGroup G0{}, G1{};
            const int ng = btree_stream_groups(S, p0, p1, G0, G1);
            for (int gq = 0; gq < ng; ++gq)
                for (uint32_t lv = 0; lv < S.g.h; ++lv) {
                    const TopRun run = btree_group_run(S, gq ? G1 : G0, lv, k);
                    std::vector<int64_t> before(rem);
                    for (uint32_t e = 0; e < run.cnt; ++e) {
                        const uint64_t o = btree_top_item_off(S, run, e), p = run.dest0 + e;
                        if (btree_run_direct(S, run, e)) direct(o, p);
                        else from_scratch(o, S.plan == PLAN_O ? p + (uint64_t)(e < run.nlo ? run.slo : run.shi) : p);
                    }
                    uint64_t u;
                    uint32_t c0, c1;
                    btree_run_reads(S, run, u, c0, c1);  // as the kernel counts them
                    if (c0 && before[u] - rem[u] != c0) ok = false;
                    if (c1 && before[u + 1] - rem[u + 1] != c1) ok = false;
                    if (!c0 && before != rem) ok = false;
                }
        }
        if (rem[k] != 0) ok = false;  // some reader of this tile comes later
        for (uint32_t o = 0; o < cnt; ++o) {
            if (!got[o] || over[p0 + o]) ok = false;
            A[p0 + o] = tile[o];
            over[p0 + o] = 1;
        }
    }
    return ok;
}

// The reverse replayed at both key widths under the ordered schedule (wherever
// there is one) and at 8 bytes under the fixed directions (test hook).
int emulate_unpermute(int layout, uint64_t n, uint64_t b, uint64_t *A) {
    if (n > 0 && !A) return TL_ERROR_INVALID_VALUE;
    PermutePlan pl;
    OrderVectors ov;
    int rc = permute_plan_replay(layout, n, b, 8, false, ov, pl);
    if (rc) return rc;
    if (n <= 1) return TL_SUCCESS;
    const std::vector<uint64_t> in(A, A + n);
    std::vector<uint64_t> out(in);
    if (!replay_reverse(pl, out)) return TL_ERROR_UNSUPPORTED;
    for (uint32_t kb : {8u, 4u}) {
        PermutePlan po;
        OrderVectors vo;
        rc = permute_plan_replay(layout, n, b, kb, true, vo, po);
        if (rc) return rc;
        std::vector<uint64_t> again(in);
        if (!replay_reverse(po, again) || again != out) return TL_ERROR_UNSUPPORTED;
    }
    std::copy(out.begin(), out.end(), A);
    return TL_SUCCESS;
}

}  // namespace tl
