// In-place permutations sorted -> {B-tree, BST, mvEB} for sm_100a.
//
// Every layout is a pure index permutation with the same two-part structure:
// most keys belong to "bulk" runs (the leaf level of a B-tree, the bottom-level
// subtrees of an mvEB) that land at a position >= their source position, and a
// minority (the separators above them) land further left.  The permutation is
// therefore done in two kernels instead of the reference's chain of cycle-leader
// and reversal launches:
//
//  1. stream: one pass over the array, one tile per ticket.  A tile is read
//     into shared memory, flagged as read, and its bulk keys are stored
//     straight to their final positions once the tiles under those positions
//     have been read.  The other keys go to a scratch buffer.
//  2. B-tree: a copy of the scratch (indexed by final position) into place,
//     or under the ordered-tile schedule the fix pass over the tiles that
//     received scratch keys; mvEB: a scatter of the scratch slots to their
//     final positions.  Every destination is free by then.
//
// DRAM traffic is 2*n*w for the stream plus 2*w per scratch key: 6-20 % of the
// keys of a B-tree or BST under the ordered schedule, about n/2^8 for an mvEB.
#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <vector>

#include "btree_order.h"
#include "btree_plan.cuh"
#include "bulk.cuh"
#include "geometry.cuh"
#include "internal.h"
#include "mveb_plan.cuh"
#include "unpermute.h"
#include "stream.cuh"

namespace tl {

constexpr uint32_t kUnitMaxLevels = 8;
// mveb_stream_kernel: 32 KB stages a block, blocks per SM (the shared memory of
// six tiles an SM), store warps a block (after the loader, publisher and waiter).
constexpr uint32_t kMvebStages = 3;
constexpr int kMvebBlocksPerSM = 2;
constexpr uint32_t kMvebStoreWarps = 8;
constexpr int kMvebThreads = 32 * (3 + (int)kMvebStoreWarps);
constexpr size_t kMvebStageBytes = 32768 + 128;

template <typename K>
constexpr uint64_t stream_tile_keys() {
    return 32768 / sizeof(K);
}

static inline uint64_t align_up(uint64_t x, uint64_t a) { return (x + a - 1) / a * a; }

constexpr int kBtreeStages = 3, kBtreeBlocksPerSM = 2, kBtreeStoreWarps = 8;
constexpr int kBtreeThreads = 32 * (2 * kBtreeStages + kBtreeStoreWarps);

struct BtreeStage {
    TileShared ts;
    uint64_t ticket, p0, p1, base;
    int last;  // no tile is left
};

// A ring of three 32 KB stages a block.  A stage's first warp claims a tile, loads
// it, publishes it as read and waits for the tiles under its bulk keys; its second
// warp works out the tile's runs of top keys (one lane per level, with their table
// lookups) and waits for the tiles under their direct parts; the store warps take
// the stages in turn and meet at no barrier.  Stages claim in turn, so a block
// stores in ticket order, and every wait is on a tile with an earlier ticket: the
// smallest tile not yet stored is its block's next and always progresses.  With
// `ahead` (kClaimAheadItems tiles a stage or more) a stage claims its next tile
// while its present one is stored.  The bound is the copy rate: with a block
// holding one tile at a time (load, publish, wait, store; six blocks an SM) the
// phases overlapped only between blocks.  Measured on B200, device time of the
// whole permutation: b = 16, 5e8 u64 keys 1361 -> 1287 us (1313 not ahead), u32
// 928 -> 832; b = 8, 2^24 u32 82 -> 71; BST of 2^27 - 1 u64 536 -> 494.  With 4
// store warps 1334, 1049, 85 and 577, with 16 (spills) 1462, 895, 72 and 546.
// kBst: the instance for b = 1 (see btree_store_top's kRunRegs).
template <typename K, bool kBst = false>
__global__ void __launch_bounds__(kBtreeThreads, kBtreeBlocksPerSM)
btree_stream_kernel(K *__restrict__ A, K *__restrict__ scr, const __grid_constant__ BtreeStream S, Ctrl *ctrl,
                    WaitCfg wc, unsigned int *flags, uint32_t ring, uint32_t stage_keys, bool ahead) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ BtreeStage s_st[kBtreeStages];
    __shared__ uint64_t s_claimed[kBtreeStages], s_tile[kBtreeStages], s_ready[kBtreeStages], s_empty[kBtreeStages];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < ring; ++s) {
            mbar_init(&s_claimed[s], 1);
            mbar_init(&s_tile[s], 1);
            mbar_init(&s_ready[s], 2);
            mbar_init(&s_empty[s], kBtreeStoreWarps);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    auto wait_bar = [&](uint64_t *bar, uint32_t parity) {
        const bool ok = __all_sync(0xFFFFFFFFu, mbar_wait_long(bar, parity));
        if (!ok && lane == 0) atomicOr(&ctrl->error, 1u << TL_ERROR_TIMEOUT);
        return ok;
    };
    uint32_t phase = 0;
    if (warp < kBtreeStages) {  // a stage's first warp
        const uint32_t s = warp;
        if (s >= ring) return;
        BtreeStage &T = s_st[s];
        K *sm = tile_smem<K>(smem_raw) + (size_t)s * stage_keys;
        while (true) {
            if (!ahead && !wait_bar(&s_empty[s], phase ^ 1)) return;
            if (!wait_bar(&s_claimed[s ? s - 1 : ring - 1], s ? phase : phase ^ 1)) return;
            unsigned long long t = 0;
            if (lane == 0) {
                t = atomicAdd(&ctrl->ticket, 1ull);
                T.ticket = t;  // and so has its value before the next stage claims
                mbar_arrive(&s_claimed[s]);
            }
            t = __shfl_sync(0xFFFFFFFFu, t, 0);
            const uint64_t k = t < S.ntiles ? btree_tile_of_ticket(S, t) : 0;
            if (!wait_bar(&s_empty[s], phase ^ 1)) return;
            if (t >= S.ntiles) {
                if (lane == 0) {
                    T.last = 1;
                    mbar_arrive(&s_tile[s]);
                    mbar_arrive(&s_ready[s]);
                }
                return;
            }
            uint64_t p0, p1, w_lo, w_hi;
            btree_tile(S, k, p0, p1);
            const uint64_t base = tile_base(A, p0);
            if (lane == 0) {
                T.last = 0;
                T.p0 = p0, T.p1 = p1, T.base = base;
                T.ts.ok0 = T.ts.ok1 = 1;
                mbar_arrive(&s_tile[s]);
            }
            load_tile_issue(A, p0, p1, sm, lane, 32);
            if (lane == 0) T.ts.reg = btree_stream_regime(S, p0, p1);
            // a look at the flags while the copies are in flight mostly finds them set
            bool pending = false;
            if (btree_tile_wait(S, p0, p1, w_lo, w_hi))
                for (uint64_t f = w_lo + lane; f <= w_hi; f += 32)
                    if (f != k && !(S.plan == PLAN_O && !btree_o_direct(S, k, f)))  // else its keys go to scratch
                        pending |= ld_acquire(&flags[f]) != wc.wait_value;
            load_tile_wait();
            __syncwarp();
            if (lane == 0) st_relaxed(&flags[k], wc.flag_value);  // published: every copy has landed
            if (pending)
                for (uint64_t f = w_lo + lane; f <= w_hi; f += 32)
                    if (f != k && !(S.plan == PLAN_O && !btree_o_direct(S, k, f)))
                        if (!wait_flag(&flags[f], wc.wait_value, ctrl, wc)) T.ts.ok1 = 0;
            __syncwarp();
            if (lane == 0) mbar_arrive(&s_ready[s]);
            phase ^= 1;
        }
    } else if (warp < 2 * kBtreeStages) {  // a stage's second warp
        const uint32_t s = warp - kBtreeStages;
        if (s >= ring) return;
        BtreeStage &T = s_st[s];
        while (wait_bar(&s_tile[s], phase)) {
            const int last = T.last;
            if (!last)
                btree_tile_runs_warp(S, T.p0, T.p1, reinterpret_cast<uintptr_t>(A), reinterpret_cast<uintptr_t>(scr),
                                     (uint32_t)sizeof(K), flags, ctrl, wc, T.ts);
            __syncwarp();
            if (lane == 0) mbar_arrive(&s_ready[s]);
            if (last) break;
            phase ^= 1;
        }
    } else {  // store warps
        const uint32_t tb = threadIdx.x - 64 * kBtreeStages, nb = 32 * kBtreeStoreWarps;
        uint32_t s = 0;
        while (wait_bar(&s_ready[s], phase)) {
            const BtreeStage &T = s_st[s];
            if (T.last) break;
            if (T.ts.ok0 && T.ts.ok1) {
                const K *tl = tile_smem<K>(smem_raw) + (size_t)s * stage_keys + (T.p0 - T.base);
                btree_store_bulk(S, A, scr, ctrl, T.p0, T.p1, tl, T.ts, tb, nb);
                btree_store_top<K, kBst>(S, tl, T.ts, tb, nb);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&s_empty[s]);
            if (++s == ring) {
                s = 0;
                phase ^= 1;
            }
        }
    }
}

// Second pass of a B-tree permutation: the scratch ranges to their final
// positions, a plain copy (scratch is indexed by final position) through the
// bulk-copy engine.
template <typename K>
__global__ void __launch_bounds__(32)
btree_copy_kernel(K *__restrict__ A, const K *__restrict__ scr, const __grid_constant__ BulkPlan P, Ctrl *ctrl) {
    extern __shared__ __align__(128) unsigned char stage[];
    __shared__ __align__(8) uint64_t bars[kBulkStages];
    bulk_copy_plan(A, scr, P, stage, bars, ctrl);
}

// Second pass of a plan-O B-tree permutation for the scratch keys outside the
// whole-tile ranges: the host-listed copies, a warp per copy.
template <typename K>
__global__ void __launch_bounds__(kScatterThreads)
btree_fix_kernel(K *__restrict__ A, const K *__restrict__ scr, const FixSeg *__restrict__ segs, uint64_t nsegs) {
    const uint64_t w = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t i = w; i < nsegs; i += nw) {
        const uint64_t dl = __ldg(reinterpret_cast<const unsigned long long *>(&segs[i].dst_len));
        const uint64_t src = __ldg(reinterpret_cast<const unsigned long long *>(&segs[i].src));
        warp_copy_keys(A + (dl & kSegDstMask), scr + src, 0, (uint32_t)(dl >> 48));
    }
}

// Small arrays (permute_by_keys): every key of the copy C to its position.
template <typename K>
__global__ void __launch_bounds__(256)
btree_scatter_keys_kernel(K *__restrict__ A, const K *__restrict__ C, uint64_t n, const __grid_constant__ KeysGeometry kg) {
    const uint64_t x = (uint64_t)blockIdx.x * 256 + threadIdx.x;
    if (x < n) A[btree_pos(kg.g, kg.fd, x)] = C[x];
}

// ---------------------------------------------------------------- mvEB stream
// A tile's stage of the ring: the loader warp fills in the tile, the waiter
// warp clears ok when a wait of the tile ran out.
struct MvebStage {
    uint64_t k, p0, p1, base;  // tile, its source ranks, and the rank at sm[0] of the stage
    int ri;                    // its region; -1: no tile is left
    int ok;
};

// The bound is the copy rate once no store waits: with a tile a block at a time
// (load, publish, wait, store; 6 blocks an SM) every tile met flags that had
// only just been claimed, and those waits were a sixth of the pass.  Here the
// loader keeps a ring of stages filled by the bulk-copy engine, the publisher
// flags each tile the moment its copy lands, while earlier tiles of the block
// are still being stored, and the waiter has a tile's flags checked before the
// store warps, which meet at no barrier, come to it.  A block claims tickets in
// order and a tile is published when its stage is free, that is when tiles with
// smaller tickets are stored: the smallest unpublished tile always progresses.
// Measured on B200, 3e8 keys: u32 500 -> 414 us (5.8 TB/s), u64 948 -> 789; two
// stages in three blocks 442 / 860, six in one 520 / 959 (24 store warps: one
// loader's tickets and copies come too slowly), 12 and 16 store warps 413 / 818
// and 419 / 806.
template <typename K>
__global__ void __launch_bounds__(kMvebThreads, kMvebBlocksPerSM)
mveb_stream_kernel(K *__restrict__ A, K *__restrict__ scr, const __grid_constant__ MvebParams prm,
                   Ctrl *ctrl, WaitCfg wc, unsigned int *flags, uint32_t ring) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ uint64_t s_full[kMvebStages], s_ready[kMvebStages], s_empty[kMvebStages];
    __shared__ MvebStage s_st[kMvebStages];
    const MvebPlan &P = prm.plan;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < ring; ++s) {
            mbar_init(&s_full[s], 32);
            mbar_init(&s_ready[s], 1);
            mbar_init(&s_empty[s], kMvebStoreWarps + 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    uint32_t s = 0, phase = 0;  // stage of this warp's next tile, and the parity of its round
    auto stage_keys = [&](uint32_t i) { return reinterpret_cast<K *>(smem_raw + (size_t)i * kMvebStageBytes); };
    auto advance = [&] {
        if (++s == ring) {
            s = 0;
            phase ^= 1;
        }
    };
    auto wait_bar = [&](uint64_t *bar, uint32_t parity) {
        const bool ok = __all_sync(0xFFFFFFFFu, mbar_wait_long(bar, parity));
        if (!ok && lane == 0) atomicOr(&ctrl->error, 1u << TL_ERROR_TIMEOUT);
        return ok;
    };
    if (warp == 0) {  // loader
        uint32_t issued = 0;
        while (true) {
            // the first round finds the stages empty: waiting for the parity before the first passes at once
            if (!wait_bar(&s_empty[s], phase ^ 1)) break;
            unsigned long long t = 0;
            if (lane == 0) t = atomicAdd(&ctrl->ticket, 1ull);
            t = __shfl_sync(0xFFFFFFFFu, t, 0);
            MvebStage &T = s_st[s];
            if (t >= P.total_tiles) {
                if (lane == 0) T.ri = -1;
                __syncwarp();
                mbar_arrive(&s_full[s]);
                return;  // its loads complete before the publisher leaves
            }
            const uint64_t k = P.total_tiles - 1 - t;
            int ri;
            uint64_t p0, p1;
            mveb_tile(P, k, ri, p0, p1);
            K *sm = stage_keys(s);
            constexpr uint32_t V = 16 / sizeof(K);
            const uint64_t base = tile_base<16>(A, p0);
            uint64_t a0 = base != p0 ? base + V : p0;  // first aligned key (base may lie below 0 and wrap)
            if (a0 > p1) a0 = p1;
            const uint64_t a1 = a0 + (p1 - a0) / V * V;
            if (lane < a0 - p0) sm[p0 + lane - base] = A[p0 + lane];
            if (lane < p1 - a1) sm[a1 + lane - base] = A[a1 + lane];
            if (lane == 0) {
                T.k = k, T.p0 = p0, T.p1 = p1, T.base = base;
                T.ri = ri, T.ok = 1;
                const uint32_t bytes = (uint32_t)((a1 - a0) * sizeof(K));
                // the ragged ends of the tile before were stored to where this copy lands
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                mbar_expect_tx(&s_full[s], bytes);
                if (bytes) bulk_load(sm + (a0 - base), A + a0, bytes, &s_full[s]);
            } else {
                mbar_arrive(&s_full[s]);
            }
            if (issued < ring) ++issued;
            advance();
        }
        for (uint32_t i = 0; i < issued; ++i) {  // a wait ran out: its copies in flight land first
            if (s-- == 0) s = ring - 1, phase ^= 1;
            mbar_wait(&s_full[s], phase);
        }
    } else if (warp == 1) {  // publisher: "tile read" as soon as its copy has landed
        while (wait_bar(&s_full[s], phase)) {
            const int ri = s_st[s].ri;
            __syncwarp();
            if (lane == 0 && ri >= 0) {
                st_relaxed(&flags[s_st[s].k], wc.flag_value);
                mbar_arrive(&s_empty[s]);
            }
            if (ri < 0) break;
            advance();
        }
    } else if (warp == 2) {  // waiter: the tiles under this tile's destinations have been read
        while (wait_bar(&s_full[s], phase)) {
            MvebStage &T = s_st[s];
            const int ri = T.ri;
            uint64_t k_lo, k_hi;
            bool ok = true;
            if (ri >= 0 && mveb_tile_wait(P, P.reg[ri], T.p0, T.p1, k_lo, k_hi))
                for (uint64_t f = k_lo + lane; f <= k_hi; f += 32)
                    if (!wait_flag(&flags[f], wc.wait_value, ctrl, wc)) ok = false;
            if (!ok) T.ok = 0;
            __syncwarp();
            if (lane == 0) mbar_arrive(&s_ready[s]);
            if (ri < 0) break;
            advance();
        }
    } else {  // store warps
        const uint32_t w = warp - 3;
        int loaded_U = -1;
        uint32_t inv_pk[2] = {0, 0};  // this lane's entries q = lane + 32 j (j < 8) of the unit table, four a register
        while (wait_bar(&s_full[s], phase) && wait_bar(&s_ready[s], phase)) {
            const MvebStage &T = s_st[s];
            if (T.ri < 0) break;
            const MvebRegion &R = P.reg[T.ri];
            const uint64_t p0 = T.p0, p1 = T.p1, base = T.base;
            const K *sm = stage_keys(s);
            if (R.U == 0) {
                for (uint64_t x = p0 + w * 32 + lane; x < p1; x += 32 * kMvebStoreWarps)
                    scr[R.slot_base + (x - R.src)] = sm[x - base];
            } else if (T.ok) {
                const uint32_t U = R.U;
                const uint64_t u = (1ull << U) - 1;
                if ((int)U != loaded_U) {
                    const unsigned char *src = prm.inv + unit_table_off(U);
                    inv_pk[0] = inv_pk[1] = 0;
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const uint32_t q = lane + 32u * j;
                        if (q < (uint32_t)u) inv_pk[j >> 2] |= (uint32_t)src[q] << (8 * (j & 3));
                    }
                    loaded_U = (int)U;
                }
                uint64_t g0, g1;
                mveb_tile_groups(R, p0, p1, g0, g1);
                // a warp's units in batches of 32: their destinations lane-parallel, one
                // unit per lane, then each unit's keys by the whole warp
                for (uint64_t gb = g0 + w; gb < g1; gb += 32ull * kMvebStoreWarps) {
                    const uint64_t gl = gb + (uint64_t)lane * kMvebStoreWarps;
                    const uint64_t my_dst = gl < g1 ? mveb_unit_dst(R, gl) : 0;
                    const uint32_t nb = (uint32_t)std::min<uint64_t>(32, (g1 - gb + kMvebStoreWarps - 1) / kMvebStoreWarps);
                    for (uint32_t j = 0; j < nb; ++j) {
                        const uint64_t gi = gb + (uint64_t)j * kMvebStoreWarps;
                        const uint64_t dst = __shfl_sync(0xFFFFFFFFu, my_dst, j);
                        const uint32_t gsrc = (uint32_t)(R.src + (gi << U) - base);
                        K *d = A + dst + lane;
                        const K *g = sm + gsrc;
#pragma unroll
                        for (int jj = 0; jj < 8; ++jj)
                            if (lane + 32u * jj < (uint32_t)u) d[32 * jj] = g[(inv_pk[jj >> 2] >> (8 * (jj & 3))) & 0xFFu];
                        if (lane == 0 && R.src + (gi << U) + u < R.src + R.len)
                            scr[R.slot_base + gi] = sm[gsrc + u];
                    }
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&s_empty[s]);
            advance();
        }
    }
}

template <typename K>
__global__ void __launch_bounds__(kScatterThreads)
mveb_scatter_kernel(K *__restrict__ A, const K *__restrict__ scr, const __grid_constant__ MvebParams prm) {
    const MvebPlan &P = prm.plan;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    uint64_t s = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (; s + 3 * stride < P.total_slots; s += 4 * stride) {
        K v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = __ldcs(scr + s + u * stride);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const uint64_t rank = mveb_slot_rank(P, s + u * stride);
            if (rank != ~0ull) A[veb_pos(P.n, rank, P.modified != 0)] = v[u];
        }
    }
    for (; s < P.total_slots; s += stride) {
        const uint64_t rank = mveb_slot_rank(P, s);
        if (rank != ~0ull) A[veb_pos(P.n, rank, P.modified != 0)] = scr[s];
    }
}

// ---------------------------------------------------------------- host side
// When a B-tree permutation takes plan O: ORDER_AUTO from kOrderMinTiles tiles
// up (below that a tile order has too few tiles to pay for its second pass),
// for a BST from kOrderMinTilesBst (measured on B200, u64 keys: at 2^20 - 1
// the fixed schedule takes 34 us against 42, its second pass one launch
// instead of two; at 2^26 - 1 they tie, 0.289 against 0.290 ms), ORDER_ALWAYS
// whenever there is a top tree and more than one tile (host replay).
enum OrderMode { ORDER_NEVER = 0, ORDER_AUTO = 1, ORDER_ALWAYS = 2 };
constexpr uint64_t kOrderMinTiles = 64;
constexpr uint64_t kOrderMinTilesBst = 16384;
// tl_debug_set_schedule: 1 = ORDER_AUTO acts as ORDER_NEVER; 2 = batched plans
// order every instance that can take the ordered schedule
static std::atomic<int> g_schedule_mode{0};

void set_schedule_mode(int mode) { g_schedule_mode = mode; }
bool fixed_schedule_only() { return g_schedule_mode == 1; }
bool ordered_schedule_forced() { return g_schedule_mode == 2; }

// Plan O's tables come from the library's cache unless `tables` are given.
// Whether a B-tree / BST plan takes the ordered-tile schedule in order_mode.
static bool order_wanted(const PermutePlan &pl, int order_mode) {
    return pl.bs.g.h >= 1 && pl.ntiles >= 2 &&
           (order_mode == ORDER_ALWAYS ||
            (order_mode == ORDER_AUTO && pl.ntiles >= (pl.b == 1 ? kOrderMinTilesBst : kOrderMinTiles) &&
             !fixed_schedule_only()));
}

static int make_plan(int layout, uint64_t n, uint64_t b, uint32_t key_bytes, PermutePlan &pl,
                     int order_mode = ORDER_AUTO, const OrderTables *tables = nullptr) {
    if (key_bytes != 4 && key_bytes != 8) return TL_ERROR_INVALID_VALUE;
    if (layout == TL_LAYOUT_BST) b = 1;
    if (layout == TL_LAYOUT_BTREE && b == 0) return TL_ERROR_INVALID_VALUE;
    if (layout < TL_LAYOUT_BST || layout > TL_LAYOUT_VEB) return TL_ERROR_INVALID_VALUE;
    pl.layout = layout;
    pl.key_bytes = key_bytes;
    pl.n = n;
    pl.b = b;
    pl.tile_keys = 32768 / key_bytes;
    if (is_veb_layout(layout)) {
        if (n >= (1ull << 62)) return TL_ERROR_UNSUPPORTED;
        pl.mp.plan = make_mveb_plan(n, kUnitMaxLevels, pl.tile_keys, layout == TL_LAYOUT_MVEB);
        fill_unit_tables(pl.mp);
        pl.ntiles = pl.mp.plan.total_tiles;
        pl.scratch_keys = pl.mp.plan.total_slots;
    } else {
        if (b >= (1ull << 31)) return TL_ERROR_UNSUPPORTED;
        pl.bs.g = make_btree_geom(n, b);
        // per-level tables and 32-bit tile indices of the wait lists
        if (pl.bs.g.h > (uint32_t)kMaxTopLevels || n / pl.tile_keys >= (1ull << 32)) return TL_ERROR_UNSUPPORTED;
        pl.bs.fd = FastDiv64(b + 1);
        pl.bs.fd32 = FastDiv32((uint32_t)(b + 1));
        if (b >= 2) {
            pl.bs.fd32b = FastDiv32((uint32_t)b);
            pl.bs.fdb = FastDiv64(b);
        }
        pl.bs.tile_keys = pl.tile_keys;
        pl.bs.tile_shift = (uint32_t)__builtin_ctzll(pl.tile_keys);
        btree_set_pow_divs(pl.bs, make_pow_divs(b));
        pl.ntiles = (n + pl.tile_keys - 1) / pl.tile_keys;
        pl.bs.ntiles = pl.ntiles;
        btree_choose_plan(pl.bs, key_bytes);
        if (order_wanted(pl, order_mode)) {
            if (tables) pl.ot = *tables;
            if (tables || btree_order_host(pl.bs, pl.ot)) {
                btree_set_ordered(pl.bs, pl.ot.tab, pl.ot.order, pl.ot.scratch_tiles);
                pl.ordered = true;
            }
        }
        pl.scratch_keys = pl.bs.nscratch;
    }
    // + 16 bytes: the scratch starts at the array's own offset within 16 bytes
    pl.off_flags = align_up(pl.scratch_keys * key_bytes + 16, 256);
    pl.off_ctrl = pl.off_flags + align_up(pl.ntiles * sizeof(unsigned int), 256);
    pl.bytes = pl.off_ctrl + align_up(sizeof(Ctrl), 256);
    return TL_SUCCESS;
}

static int g_sm_count = 0;
static std::once_flag g_props_once;
static int sm_count() {
    std::call_once(g_props_once, [] {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&g_sm_count, cudaDevAttrMultiProcessorCount, dev);
        if (g_sm_count <= 0) g_sm_count = 148;
    });
    return g_sm_count;
}

static std::atomic<int> g_last_launches{0};  // kernels the last permutation launched (profiling hook)

int last_permute_launches() { return g_last_launches; }

template <typename K>
static int launch_permute_k(const PermutePlan &pl, K *A, char *ws, cudaStream_t st, EventTimer &timer, int &nl);

template <typename K>
static int launch_permute(const PermutePlan &pl, K *A, char *ws, cudaStream_t st, EventTimer &timer) {
    int nl = 0;
    const int rc = launch_permute_k(pl, A, ws, st, timer, nl);
    g_last_launches = nl;
    return rc;
}

template <typename K>
static int launch_permute_k(const PermutePlan &pl, K *A, char *ws, cudaStream_t st, EventTimer &timer, int &nl) {
    // the scratch shares A's offset within 16 bytes, so the copy pass vectorises
    K *scr = reinterpret_cast<K *>(ws + (reinterpret_cast<uintptr_t>(A) & 15));
    unsigned int *flags = reinterpret_cast<unsigned int *>(ws + pl.off_flags);
    Ctrl *ctrl = reinterpret_cast<Ctrl *>(ws + pl.off_ctrl);
    WaitCfg wc;
    wc.flag_value = 1;
    wc.wait_value = debug_force_timeout() ? 0xFFFFFFFFu : 1u;  // forced: no tile ever publishes it
    wc.spin_limit = debug_spin_limit();
    // flags and control block are contiguous: one stream-ordered memset clears both
    TL_CUDA_TRY(cudaMemsetAsync(flags, 0, pl.bytes - pl.off_flags, st));
    const int smx = sm_count();
    if (is_veb_layout(pl.layout)) {
        auto kern = mveb_stream_kernel<K>;
        constexpr size_t ring_bytes = kMvebStages * kMvebStageBytes;
        TL_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ring_bytes));
        int per_sm = 0;
        TL_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kMvebThreads, ring_bytes));
        uint64_t grid = std::min<uint64_t>((uint64_t)std::max(per_sm, 1) * smx, std::max<uint64_t>(pl.ntiles, 1));
        const uint32_t ring = (uint32_t)std::min<uint64_t>(kMvebStages, (pl.ntiles + grid - 1) / grid);
        if (pl.ntiles) kern<<<(unsigned)grid, kMvebThreads, ring_bytes, st>>>(A, scr, pl.mp, ctrl, wc, flags, ring), ++nl;
        TL_CUDA_TRY(cudaGetLastError());
        timer.mid();
        if (pl.scratch_keys) {
            int sper = 0;
            TL_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&sper, mveb_scatter_kernel<K>,
                                                                      kScatterThreads, 0));
            uint64_t sg = std::min<uint64_t>((pl.scratch_keys + kScatterThreads - 1) / kScatterThreads,
                                             (uint64_t)std::max(sper, 1) * smx);
            mveb_scatter_kernel<K><<<(unsigned)sg, kScatterThreads, 0, st>>>(A, scr, pl.mp);
            ++nl;
            TL_CUDA_TRY(cudaGetLastError());
        }
    } else {
        auto kern = pl.bs.g.b == 1 ? btree_stream_kernel<K, true> : btree_stream_kernel<K, false>;
        const size_t stage = (size_t)pl.tile_keys * sizeof(K) + 128, ring_bytes = kBtreeStages * stage + 128;
        TL_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ring_bytes));
        int per_sm = 0;
        TL_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kBtreeThreads, ring_bytes));
        uint64_t grid = std::min<uint64_t>((uint64_t)std::max(per_sm, 1) * smx, std::max<uint64_t>(pl.ntiles, 1));
        const uint32_t ring = (uint32_t)std::min<uint64_t>(kBtreeStages, (pl.ntiles + grid - 1) / grid);
        if (pl.ntiles)
            kern<<<(unsigned)grid, kBtreeThreads, ring_bytes, st>>>(A, scr, pl.bs, ctrl, wc, flags, ring,
                                                                    (uint32_t)(stage / sizeof(K)),
                                                                    pl.ntiles >= kClaimAheadItems * grid * ring), ++nl;
        TL_CUDA_TRY(cudaGetLastError());
        timer.mid();
        if (pl.ordered && pl.ot.nsegs) {
            int fper = 0;
            TL_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fper, btree_fix_kernel<K>, kScatterThreads, 0));
            const uint64_t fg = std::min<uint64_t>((pl.ot.nsegs * 32 + kScatterThreads - 1) / kScatterThreads,
                                                   (uint64_t)std::max(fper, 1) * smx);
            btree_fix_kernel<K><<<(unsigned)fg, kScatterThreads, 0, st>>>(A, scr, pl.ot.segs, pl.ot.nsegs);
            ++nl;
            TL_CUDA_TRY(cudaGetLastError());
        }
        BulkPlan bp;
        int rc = make_bulk_plan(pl.bs, pl.ot, A, scr, bp);
        if (rc) return rc;
        if (bp.nr) {
            // one warp per CTA, as many CTAs per SM as the stages' shared memory allows
            const size_t smem = (size_t)kBulkStages * kBulkChunk;
            auto ck = btree_copy_kernel<K>;
            TL_CUDA_TRY(cudaFuncSetAttribute(ck, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            int cper = 0;
            TL_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&cper, ck, 32, smem));
            const uint64_t cg = std::max<uint64_t>(1, std::min<uint64_t>(bp.nchunks, (uint64_t)std::max(cper, 1) * smx));
            ck<<<(unsigned)cg, 32, smem, st>>>(A, scr, bp, ctrl);
            ++nl;
            TL_CUDA_TRY(cudaGetLastError());
        }
    }
    return TL_SUCCESS;
}

int btree_plan_of(uint64_t n, uint64_t b) {
    PermutePlan pl;
    if (make_plan(TL_LAYOUT_BTREE, n, b, 8, pl, ORDER_NEVER)) return -1;
    return pl.bs.plan;
}

template <typename Kern>
static int blocks_per_sm_of(Kern kern, size_t smem, int threads) {
    int per_sm = 0;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem) != cudaSuccess)
        return -1;
    return per_sm;
}

// Resident blocks per SM of the stream kernel instance launch_permute_k picks
// for the layout (the BST has its own instance), at the 32 KB tile.
int stream_blocks_per_sm(int layout, uint32_t key_bytes) {
    const size_t btree_ring = kBtreeStages * (size_t)(32768 + 128) + 128;
    const bool w8 = key_bytes == 8;
    if (is_veb_layout(layout))
        return w8 ? blocks_per_sm_of(mveb_stream_kernel<uint64_t>, kMvebStages * kMvebStageBytes, kMvebThreads)
                  : blocks_per_sm_of(mveb_stream_kernel<uint32_t>, kMvebStages * kMvebStageBytes, kMvebThreads);
    if (layout == TL_LAYOUT_BST)
        return w8 ? blocks_per_sm_of(btree_stream_kernel<uint64_t, true>, btree_ring, kBtreeThreads)
                  : blocks_per_sm_of(btree_stream_kernel<uint32_t, true>, btree_ring, kBtreeThreads);
    return w8 ? blocks_per_sm_of(btree_stream_kernel<uint64_t, false>, btree_ring, kBtreeThreads)
              : blocks_per_sm_of(btree_stream_kernel<uint32_t, false>, btree_ring, kBtreeThreads);
}

int permute_plan_of(int layout, uint64_t n, uint64_t b, uint32_t key_bytes) {
    PermutePlan pl;
    const int rc = make_plan(layout, n, b, key_bytes, pl);
    if (rc) return -rc;
    return is_veb_layout(layout) ? 3 : pl.bs.plan;
}

int permute_scratch_keys(int layout, uint64_t n, uint64_t b, uint32_t key_bytes, uint64_t *keys) {
    if (!keys) return TL_ERROR_INVALID_VALUE;
    PermutePlan pl;
    int rc = make_plan(layout, n, b, key_bytes, pl);
    if (rc) return rc;
    if (is_veb_layout(layout)) {
        *keys = pl.mp.plan.total_slots;
    } else if (pl.ordered) {
        uint64_t c = 0;
        for (uint64_t i = 0; i < pl.ot.nranges; ++i)
            c += std::min<uint64_t>((uint64_t)pl.ot.ranges[i].y << pl.bs.tile_shift, n) -
                 ((uint64_t)pl.ot.ranges[i].x << pl.bs.tile_shift);
        for (uint64_t i = 0; i < pl.ot.nsegs; ++i) c += pl.ot.segs[i].dst_len >> 48;
        *keys = c;
    } else {
        *keys = 0;
        CopyRange r;
        for (int j = 0; j < btree_copy_range_count(pl.bs); ++j)
            if (btree_copy_range(pl.bs, j, r)) *keys += r.len;
    }
    return TL_SUCCESS;
}

// Enough for whichever schedule the call ends up on: the ordered schedule when
// its tables reach the device, else the fixed-direction one (permute() falls
// back to it when the table upload fails), so a workspace of this size is never
// refused.
int permute_workspace_bytes(int layout, uint64_t n, uint64_t b, uint32_t key_bytes, uint64_t *bytes) {
    if (!bytes) return TL_ERROR_INVALID_VALUE;
    PermutePlan pl, fx;
    int rc = make_plan(layout, n, b, key_bytes, pl);
    if (rc) return rc;
    rc = make_plan(layout, n, b, key_bytes, fx, ORDER_NEVER);
    if (rc) return rc;
    *bytes = std::max(pl.bytes, fx.bytes);
    return TL_SUCCESS;
}

int permute_workspace_bytes_fixed(int layout, uint64_t n, uint64_t b, uint32_t key_bytes, uint64_t *bytes) {
    if (!bytes) return TL_ERROR_INVALID_VALUE;
    PermutePlan pl;
    int rc = make_plan(layout, n, b, key_bytes, pl, ORDER_NEVER);
    if (rc) return rc;
    *bytes = pl.bytes;
    return TL_SUCCESS;
}

int permute_plan_fixed(int layout, uint64_t n, uint64_t b, uint32_t key_bytes, PermutePlan &pl) {
    return make_plan(layout, n, b, key_bytes, pl, ORDER_NEVER);
}

bool permute_takes_order(int layout, uint64_t n, uint64_t b, uint32_t key_bytes) {
    PermutePlan fx;
    return !is_veb_layout(layout) && n > 1 && make_plan(layout, n, b, key_bytes, fx, ORDER_NEVER) == TL_SUCCESS &&
           order_wanted(fx, ORDER_AUTO);
}

int permute_plan_device(int layout, uint64_t n, uint64_t b, uint32_t key_bytes, cudaStream_t st, PermutePlan &pl) {
    if (n > 1 && !is_veb_layout(layout)) {
        // a geometry not seen before: its ordered-tile tables with kernels on
        // st (make_plan below finds them cached; if this cannot be done it
        // computes them on the host)
        PermutePlan fx;
        if (make_plan(layout, n, b, key_bytes, fx, ORDER_NEVER) == TL_SUCCESS && order_wanted(fx, ORDER_AUTO))
            btree_order_prepare(fx.bs, st);
    }
    const int rc = make_plan(layout, n, b, key_bytes, pl, ORDER_AUTO);
    if (rc || n <= 1 || !pl.ordered) return rc;
    // plan O needs its tile tables on the device; without them, the
    // fixed-direction plan
    OrderTables dt;
    if (!btree_order_device(pl.bs, st, dt)) {
        pl = PermutePlan{};
        return make_plan(layout, n, b, key_bytes, pl, ORDER_NEVER);
    }
    pl.ot = dt;
    pl.bs.tab = dt.tab;
    pl.bs.order = dt.order;
    return TL_SUCCESS;
}

int permute_plan_replay(int layout, uint64_t n, uint64_t b, uint32_t key_bytes, bool ordered, OrderVectors &ov,
                        PermutePlan &pl) {
    const int rc = make_plan(layout, n, b, key_bytes, pl, ORDER_NEVER);
    if (rc || !ordered || is_veb_layout(layout)) return rc;
    btree_compute_order(pl.bs, ov);  // computed here, not taken from the library's cache
    const OrderTables ot = ov.tables();
    return make_plan(layout, n, b, key_bytes, pl, ORDER_ALWAYS, &ot);
}

bool permute_by_keys(int layout, uint64_t n, uint64_t b, uint32_t key_bytes, KeysGeometry &kg) {
    if (layout == TL_LAYOUT_BST) b = 1;
    else if (layout != TL_LAYOUT_BTREE) return false;
    if ((key_bytes != 4 && key_bytes != 8) || b == 0 || b >= (1ull << 31)) return false;  // make_plan's refusals
    if (n <= 1 || n > kKeysBytes / key_bytes) return false;
    kg.g = make_btree_geom(n, b);
    kg.fd = FastDiv64(b + 1);
    return true;
}

template <typename K>
static int launch_by_keys(const KeysGeometry &kg, K *A, char *ws, uint64_t n, cudaStream_t st, EventTimer &timer) {
    K *C = reinterpret_cast<K *>(ws);
    TL_CUDA_TRY(cudaMemcpyAsync(C, A, n * sizeof(K), cudaMemcpyDeviceToDevice, st));
    timer.mid();
    btree_scatter_keys_kernel<K><<<(unsigned)((n + 255) / 256), 256, 0, st>>>(A, C, n, kg);
    TL_CUDA_TRY(cudaGetLastError());
    g_last_launches = 1;
    return TL_SUCCESS;
}

int permute(int layout, void *dev_A, uint64_t n, uint64_t b, uint32_t key_bytes, void *dev_ws,
            uint64_t ws_bytes, cudaStream_t st, float *ms, float *phase_ms, bool allow_ordered) {
    if (n > 0 && !dev_A) return TL_ERROR_INVALID_VALUE;
    if (reinterpret_cast<uintptr_t>(dev_A) % (key_bytes ? key_bytes : 1)) return TL_ERROR_INVALID_VALUE;
    if (dev_ws && reinterpret_cast<uintptr_t>(dev_ws) % 256) return TL_ERROR_INVALID_VALUE;
    KeysGeometry kg;
    const bool by_keys = permute_by_keys(layout, n, b, key_bytes, kg) && (!dev_ws || ws_bytes >= n * key_bytes);
    PermutePlan pl;
    int rc = by_keys         ? TL_SUCCESS
             : allow_ordered ? permute_plan_device(layout, n, b, key_bytes, st, pl)
                             : make_plan(layout, n, b, key_bytes, pl, ORDER_NEVER);
    if (rc) return rc;
    if (n <= 1) {
        if (ms) *ms = 0.f;
        return TL_SUCCESS;
    }
    if (pl.ordered && dev_ws && ws_bytes < pl.bytes) {  // the fixed-direction plan may fit
        pl = PermutePlan{};
        rc = make_plan(layout, n, b, key_bytes, pl, ORDER_NEVER);
        if (rc) return rc;
    }
    const uint64_t need = by_keys ? n * key_bytes : pl.bytes;
    if (dev_ws && ws_bytes < need) return TL_ERROR_WORKSPACE_TOO_SMALL;
    EventTimer timer(ms != nullptr || phase_ms != nullptr, st);
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
    if (by_keys)
        rc = key_bytes == 8 ? launch_by_keys(kg, static_cast<uint64_t *>(dev_A), ws, n, st, timer)
                            : launch_by_keys(kg, static_cast<uint32_t *>(dev_A), ws, n, st, timer);
    else
        rc = key_bytes == 8 ? launch_permute<uint64_t>(pl, static_cast<uint64_t *>(dev_A), ws, st, timer)
                            : launch_permute<uint32_t>(pl, static_cast<uint32_t *>(dev_A), ws, st, timer);
    timer.stop();
    unsigned int err = 0;
    if (rc == TL_SUCCESS)
        rc = read_ctrl(by_keys ? nullptr : reinterpret_cast<const Ctrl *>(ws + pl.off_ctrl), &err, st);
    if (owned && pooled) cudaFreeAsync(ws, st);
    if (rc == TL_SUCCESS) rc = sync_and_check(st);
    if (owned && !pooled) {
        if (rc != TL_SUCCESS) cudaStreamSynchronize(st);  // nothing of this call may still use it
        workspace_release(ws);
    }
    // a bounded wait expired, or (never expected) the ordered schedule found a
    // scratch store without scratch and skipped it
    if (rc == TL_SUCCESS && err) rc = (err & (1u << TL_ERROR_TIMEOUT)) ? TL_ERROR_TIMEOUT : TL_ERROR_UNSUPPORTED;
    if (rc == TL_SUCCESS && ms) *ms = timer.elapsed();
    if (rc == TL_SUCCESS && phase_ms) timer.elapsed_split(&phase_ms[0], &phase_ms[1]);
    return rc;
}

// Test hook: the ordered-tile tables of a geometry computed on the host and
// with the per-tile kernels on st, uncached, compared entry by entry.  1 equal,
// 0 different, < 0 a status (the geometry takes no ordered tables, or the
// kernels could not run).
int debug_order_tables_match(int layout, uint64_t n, uint64_t b, uint32_t key_bytes, cudaStream_t st) {
    PermutePlan fx;
    int rc = make_plan(layout, n, b, key_bytes, fx, ORDER_NEVER);
    if (rc) return -rc;
    if (is_veb_layout(layout) || !order_wanted(fx, ORDER_ALWAYS)) return -TL_ERROR_UNSUPPORTED;
    OrderVectors h, g;
    btree_compute_order(fx.bs, h);
    if (!btree_compute_order_device(fx.bs, st, g)) return -TL_ERROR_CUDA;
    auto eq2 = [](const std::vector<uint2> &x, const std::vector<uint2> &y) {
        if (x.size() != y.size()) return false;
        for (size_t i = 0; i < x.size(); ++i)
            if (x[i].x != y[i].x || x[i].y != y[i].y) return false;
        return true;
    };
    auto eq4 = [](const std::vector<uint4> &x, const std::vector<uint4> &y) {
        if (x.size() != y.size()) return false;
        for (size_t i = 0; i < x.size(); ++i)
            if (x[i].x != y[i].x || x[i].y != y[i].y || x[i].z != y[i].z || x[i].w != y[i].w) return false;
        return true;
    };
    bool same = eq2(h.tab, g.tab) && h.order == g.order && eq4(h.ranges, g.ranges) &&
                h.scratch_tiles == g.scratch_tiles && h.segs.size() == g.segs.size();
    for (size_t i = 0; same && i < h.segs.size(); ++i)
        same = h.segs[i].dst_len == g.segs[i].dst_len && h.segs[i].src == g.segs[i].src;
    return same ? 1 : 0;
}

// Host replay of the stream + scatter passes on a host array, one tile at a time
// in ticket order, using the same index helpers as the kernels.  Besides the
// result it counts protocol violations: a tile reading a position that was
// already overwritten, a store outside the tile's own source that is not covered
// by the tiles it waits for, a wait on a tile with a later ticket, and a final
// position or scratch slot written other than exactly once.  Test hook only.
static int emulate_permute_kb(int layout, uint64_t n, uint64_t b, uint32_t key_bytes, uint64_t *A,
                              uint64_t *violations, int order_mode) {
    PermutePlan pl;
    OrderVectors ov;
    const int rc = permute_plan_replay(layout, n, b, key_bytes, order_mode != ORDER_NEVER, ov, pl);
    if (rc) return rc;
    // tile kk's ticket precedes (or is) tile k's
    auto earlier = [&](uint64_t kk, uint64_t k) {
        if (pl.ordered) return btree_o_rank(pl.bs, kk) <= btree_o_rank(pl.bs, k);
        return pl.bs.plan == PLAN_R ? kk >= k : kk <= k;
    };
    uint64_t viol = 0;
    if (n > 1) {
        std::vector<uint64_t> scr(pl.scratch_keys, 0), tile(pl.tile_keys + 1);
        std::vector<uint8_t> readk(pl.ntiles, 0), written(n, 0);
        std::vector<uint32_t> slot_writes(pl.scratch_keys, 0), pos_writes(n, 0);
        const bool mv = is_veb_layout(pl.layout);
        const MvebPlan &P = pl.mp.plan;
        auto tile_of = [&](uint64_t d) { return mv ? mveb_tile_of(P, d) : d / pl.tile_keys; };
        for (uint64_t t = 0; t < pl.ntiles; ++t) {
            const uint64_t k = mv ? pl.ntiles - 1 - t : btree_tile_of_ticket(pl.bs, t);
            uint64_t p0, p1, k_lo = 0, k_hi = 0;
            int ri = 0;
            if (mv) mveb_tile(P, k, ri, p0, p1); else btree_tile(pl.bs, k, p0, p1);
            for (uint64_t x = p0; x < p1; ++x) {
                if (written[x]) ++viol;
                tile[x - p0] = A[x];
            }
            readk[k] = 1;
            const bool wait = mv ? mveb_tile_wait(P, P.reg[ri], p0, p1, k_lo, k_hi)
                                 : btree_tile_wait(pl.bs, p0, p1, k_lo, k_hi);
            if (wait)
                for (uint64_t kk = k_lo; kk <= k_hi; ++kk) {
                    if (pl.ordered && !btree_o_direct(pl.bs, k, kk)) continue;  // not waited for
                    const bool ok = mv ? kk > k : pl.ordered ? earlier(kk, k) : pl.bs.plan == PLAN_R ? kk > k : kk < k;
                    if (!ok || !readk[kk]) ++viol;
                }
            auto W = [&](uint64_t d, uint64_t v) {
                if (d >= n) { ++viol; return; }
                const uint64_t kd = tile_of(d);
                if (kd != k && !(wait && kd >= k_lo && kd <= k_hi)) ++viol;
                if (!readk[kd]) ++viol;
                A[d] = v;
                written[d] = 1;
                ++pos_writes[d];
            };
            auto SC = [&](uint64_t s, uint64_t v) {
                if (s >= scr.size()) { ++viol; return; }
                scr[s] = v;
                ++slot_writes[s];
            };
            if (!mv) {
                const BtreeStream &S = pl.bs;
                const Regime RG = btree_stream_regime(S, p0, p1);
                const uint32_t cnt = (uint32_t)(p1 - p0);
                // the runs in slot order, as warp 0 computes them, and the wait list
                TopGroup G0{}, G1{};
                const int ng = btree_stream_groups(S, p0, p1, G0, G1);
                const uint32_t nr = (uint32_t)ng * kMaxTopLevels;
                TopRun runs[kMaxTopRuns];
                uint32_t cum[kMaxTopRuns + 1], wlo[kMaxTopRuns + 1], whi[kMaxTopRuns + 1], nw = 0;
                cum[0] = 0;
                for (uint32_t sl = 0; sl < nr; ++sl) {
                    runs[sl] = btree_group_run(S, sl < kMaxTopLevels ? G0 : G1, sl % kMaxTopLevels, k);
                    cum[sl + 1] = cum[sl] + runs[sl].cnt;
                }
                uint64_t a, bq;
                std::vector<uint64_t> wl;  // plan O: the tiles the bulk stores wait for
                if (btree_tile_wait(S, p0, p1, a, bq)) {
                    if (pl.ordered) {
                        for (uint64_t kk = a; kk <= bq; ++kk) {
                            if (btree_o_direct(S, k, kk)) wl.push_back(kk);
                        }
                    } else {
                        wlo[nw] = (uint32_t)a;
                        whi[nw++] = (uint32_t)bq;
                    }
                }
                for (uint32_t sl = 0; sl < nr; ++sl)
                    if (runs[sl].cnt && btree_run_wait(S, runs[sl], a, bq)) {
                        wlo[nw] = (uint32_t)a;
                        whi[nw++] = (uint32_t)bq;
                    }
                for (uint32_t w = 0; w < nw; ++w)
                    for (uint64_t kk = wlo[w]; kk <= whi[w]; ++kk)
                        if (!earlier(kk, k) || !readk[kk]) ++viol;
                for (uint64_t kk : wl)
                    if (!earlier(kk, k) || !readk[kk]) ++viol;
                auto covered_tile = [&](uint64_t kd) {
                    if (kd == k) return true;
                    for (uint32_t w = 0; w < nw; ++w)
                        if (kd >= wlo[w] && kd <= whi[w]) return true;
                    for (uint64_t kk : wl)
                        if (kd == kk) return true;
                    return false;
                };
                auto WD = [&](uint64_t d, uint64_t v) {  // direct store, checked against the wait list
                    if (d >= n) { ++viol; return; }
                    if (!covered_tile(tile_of(d))) ++viol;
                    if (!readk[tile_of(d)]) ++viol;
                    A[d] = v;
                    written[d] = 1;
                    ++pos_writes[d];
                };
                std::vector<uint8_t> covered(cnt, 0);
                for (uint32_t o = 0; o < cnt; ++o) {
                    const uint64_t x = p0 + o;
                    uint64_t idx, ref;
                    if (RG.kind == 0) {
                        if (btree_is_top(S, x)) continue;
                        if (btree_place(S, x, idx)) WD(idx, tile[o]); else SC(idx, tile[o]);
                    } else {
                        if (RG.kind == 2 || !btree_regime_bulk(S, RG, o, idx)) continue;
                        const bool hi = RG.kind == 3 && idx >= RG.dsplit;
                        const bool to_A = hi ? RG.hi_A : RG.to_A;
                        if (RG.kind == 3 && !to_A) idx += (uint64_t)(hi ? RG.shi : RG.slo);
                        const bool direct = btree_place(S, x, ref);  // fast path == reference form
                        if (direct != to_A || ref != idx) ++viol;
                        if (to_A) WD(idx, tile[o]); else SC(idx, tile[o]);
                    }
                    covered[o] = 1;
                }
                if (cum[nr] > cnt) ++viol;
                for (uint32_t r = 0; r < nr; ++r) {
                    if (cum[r + 1] - cum[r] != runs[r].cnt) ++viol;
                    for (uint32_t e = 0; e < runs[r].cnt; ++e) {
                        const uint64_t off = btree_top_item_off(S, runs[r], e);
                        if (off >= cnt || covered[off]) { ++viol; continue; }
                        const uint64_t p = runs[r].dest0 + e;
                        const bool kdirect = btree_run_direct(S, runs[r], e);
                        const uint64_t kidx =  // the kernel's store index
                            kdirect || !pl.ordered ? p : p + (uint64_t)(e < runs[r].nlo ? runs[r].slo : runs[r].shi);
                        uint64_t ref;
                        const bool direct = btree_place(S, p0 + off, ref);
                        if (direct != kdirect || ref != kidx) ++viol;
                        if (direct) WD(kidx, tile[off]); else SC(kidx, tile[off]);
                        covered[off] = 1;
                    }
                }
                for (uint32_t o = 0; o < cnt; ++o)
                    if (!covered[o]) ++viol;
            } else {
                const MvebRegion &R = P.reg[ri];
                if (R.U == 0) {
                    for (uint64_t x = p0; x < p1; ++x) SC(R.slot_base + (x - R.src), tile[x - p0]);
                } else {
                    const unsigned char *inv = pl.mp.inv + unit_table_off(R.U);
                    const uint64_t u = (1ull << R.U) - 1;
                    uint64_t g0, g1;
                    mveb_tile_groups(R, p0, p1, g0, g1);
                    for (uint64_t gi = g0; gi < g1; ++gi) {
                        const uint64_t gsrc = R.src + (gi << R.U) - p0;
                        const uint64_t dst = mveb_unit_dst(R, gi);
                        for (uint64_t q = 0; q < u; ++q) {
                            if (gsrc + inv[q] >= p1 - p0) { ++viol; continue; }
                            W(dst + q, tile[gsrc + inv[q]]);
                        }
                        if (R.src + (gi << R.U) + u < R.src + R.len) SC(R.slot_base + gi, tile[gsrc + u]);
                    }
                }
            }
        }
        if (!mv) {
            if (pl.ordered) {  // the bulk ranges and the fix pass; every slot they read written once
                std::vector<uint8_t> read_slot(pl.bs.nscratch, 0);
                for (uint64_t i = 0; i < pl.ot.nranges; ++i) {
                    const uint64_t u0 = pl.ot.ranges[i].x;
                    const uint64_t d0 = u0 * pl.tile_keys, d1 = std::min<uint64_t>(pl.ot.ranges[i].y * pl.tile_keys, n);
                    for (uint64_t d = d0; d < d1; ++d) {
                        const uint64_t sl = d + (uint64_t)btree_o_soff(pl.bs, d / pl.tile_keys);
                        if (sl >= pl.bs.nscratch || slot_writes[sl] != 1 || read_slot[sl]) { ++viol; continue; }
                        A[d] = scr[sl];
                        ++pos_writes[d];
                        read_slot[sl] = 1;
                    }
                }
                for (uint64_t i = 0; i < pl.ot.nsegs; ++i) {
                    const uint64_t d0 = pl.ot.segs[i].dst_len & kSegDstMask, len = pl.ot.segs[i].dst_len >> 48;
                    for (uint64_t e = 0; e < len; ++e) {
                        const uint64_t d = d0 + e, sl = pl.ot.segs[i].src + e;
                        // a copy takes the slot of its own position
                        if (d >= n || sl >= pl.bs.nscratch || slot_writes[sl] != 1 || read_slot[sl] ||
                            sl != d + (uint64_t)btree_o_soff(pl.bs, d / pl.tile_keys)) {
                            ++viol;
                            continue;
                        }
                        A[d] = scr[sl];
                        ++pos_writes[d];
                        read_slot[sl] = 1;
                    }
                }
                for (uint64_t c = 0; c < pl.bs.nscratch; ++c)
                    if (slot_writes[c] != read_slot[c]) ++viol;
            } else {
                for (uint64_t c = 0; c < pl.bs.nscratch; ++c)
                    if (slot_writes[c] != (btree_slot_used(pl.bs, c) ? 1u : 0u)) ++viol;
            }
            for (int j = 0; j < btree_copy_range_count(pl.bs); ++j) {
                CopyRange cr;
                if (!btree_copy_range(pl.bs, j, cr)) continue;
                for (uint64_t e = 0; e < cr.len; ++e) {
                    const uint64_t d = cr.dst + e, s1 = cr.src + e;
                    if (d >= n || s1 >= pl.bs.nscratch || !btree_slot_used(pl.bs, s1)) { ++viol; continue; }
                    A[d] = scr[s1];
                    ++pos_writes[d];
                }
            }
        } else {
            for (uint64_t s2 = 0; s2 < P.total_slots; ++s2) {
                const uint64_t rank = mveb_slot_rank(P, s2);
                if (rank == ~0ull) { if (slot_writes[s2]) ++viol; continue; }
                if (slot_writes[s2] != 1) ++viol;
                const uint64_t d = veb_pos(n, rank, P.modified != 0);
                A[d] = scr[s2];
                ++pos_writes[d];
            }
        }
        for (uint64_t d = 0; d < n; ++d)
            if (pos_writes[d] != 1) ++viol;
    }
    if (violations) *violations = viol;
    return TL_SUCCESS;
}

// Replays the ordered schedule (plan O wherever it applies) at both key widths
// (their tile sizes and scratch alignment differ) and the fixed-direction
// schedule; the results must agree.
int emulate_permute(int layout, uint64_t n, uint64_t b, uint64_t *A, uint64_t *violations) {
    std::vector<uint64_t> A4(A, A + n), Af(A, A + n);
    uint64_t v8 = 0, v4 = 0, vf = 0;
    int rc = emulate_permute_kb(layout, n, b, 8, A, &v8, ORDER_ALWAYS);
    if (!rc) rc = emulate_permute_kb(layout, n, b, 4, A4.data(), &v4, ORDER_ALWAYS);
    if (!rc) rc = emulate_permute_kb(layout, n, b, 8, Af.data(), &vf, ORDER_NEVER);
    if (rc) return rc;
    uint64_t diff = 0;
    for (uint64_t x = 0; x < n; ++x) diff += (A[x] != A4[x]) + (A[x] != Af[x]);
    if (violations) *violations = v8 + v4 + vf + diff;
    return TL_SUCCESS;
}

}  // namespace tl
