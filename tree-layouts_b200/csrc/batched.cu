// Batched mode (no counterpart in the reference): many independent sorted
// arrays of uneven sizes, concatenated and described by an int64 offset table,
// are each permuted into a B-tree layout by ONE persistent kernel launch, and
// queried by one batch of (key, instance) pairs.
//
// Plan (built once per offset table): a setup kernel computes every instance's
// geometry and schedule (the same host/device helpers as the single-array
// path), its tile count, scratch size and copy-chunk count, and exclusive
// prefix sums of them; the host puts the instances of 64 tiles or more on the
// single-array path's ordered-tile schedule and interleaves the instances'
// tiles; a second kernel writes the owner instance of every copy chunk.
// Execute: a memset of the control words and one persistent kernel; tickets
// 0..T-1 are stream tiles (each instance's in its own schedule's order, the
// instances interleaved), tickets T.. are copy chunks (scratch -> final
// positions).  A chunk of instance j starts once all of j's tiles have stored
// (a per-instance counter, bounded wait); stream tiles never wait on chunks, so
// every wait ends.  Per size class (floor(log2 n_j)) the tile size comes from a
// tuning table that tl_batch_autotune fills by measurement.
#include <algorithm>
#include <atomic>
#include <cstring>
#include <string>
#include <thread>
#include <vector>

#include "batched.h"
#include "btree_order.h"
#include "btree_plan.cuh"
#include "bulk.cuh"
#include "internal.h"

namespace tl {

constexpr int kBatchThreads = 256;     // query kernel
// Permute kernel: blocks of three 32 KB stages, two an SM, with 8 store warps
// (plan threads 256) or 4 (512): a tuned choice.  1024 arrays of 2^10..2^22
// keys, b = 8 on B200: 8 store warps 1.65 ms, 6 1.63, 4 1.63; arrays of
// 2^8..2^14: 73, 80 and 88 us; at 10 and more the registers spill (1.9 ms).
constexpr int kBatchStages = 3, kBatchBlocksPerSM = 2;
constexpr int kBatchStoreWarps256 = 8, kBatchStoreWarps512 = 4;
constexpr size_t kBatchBlockSmem = 100 * 1024;  // dynamic shared memory of a block, beside the stages' plans
constexpr int kMaxClass = 48;

struct alignas(16) BatchInst {
    BtreeStream S;
    uint64_t off;          // first key of the instance
    uint64_t tile_base;    // first of the instance's tile flags
    uint64_t scr_base;     // first scratch slot (same 16-byte offset as the instance's keys)
    uint64_t chunk_base;   // first global copy chunk
    uint64_t nchunks;
    uint64_t item_base;    // ordered schedule: the instance's copy items in the plan's item list
    uint64_t nitems;
};

// Ordered-schedule instances (from kBatchOrderMinTiles tiles, as the single-array
// permutation): their scratch keys go back as copy items, a warp each (whole-tile
// runs in pieces of kRangePiece keys, and the fix pass's segments), grouped into
// copy chunks of at most kCopyChunk keys and kChunkItemsMax items.
constexpr uint64_t kBatchOrderMinTiles = 64;
constexpr uint64_t kChunkItemsMax = 64;
constexpr uint64_t kRangePiece = 2048;
// An instance takes the ordered schedule if that moves at most kOrderGain of the
// scratch keys of its fixed-direction schedule, and, above kOrderGainSpace, only
// in no more scratch space (the ordered schedule gives each tile that receives
// scratch keys a tile of scratch: without this, 300 arrays of 2^18..2^20 keys at
// b = 16 need 277 MB instead of 191).  Measured on B200, 1024 arrays of
// 2^10..2^22 keys, 0.3 everywhere against this: b = 8 1.75 -> 1.64 ms, b = 1 2.35
// -> 2.12, b = 4 2.03 -> 1.96 (1.88 whatever the space), b = 16 1.59 -> 1.57.
// Their tables and item lists are 1 to 2 ms of a plan of 9, which a plan that only
// answers queries pays too.
constexpr double kOrderGain = 0.9, kOrderGainSpace = 0.3;
constexpr uint64_t kInterleaveRun = 1;  // stream tiles an instance takes in a row
static_assert(sizeof(BatchInst) % 16 == 0, "BatchInst is copied to shared memory in 16-byte words");

struct BatchTotals {
    uint64_t tiles, chunks, scratch, max_tile;
};

// What a query needs of its instance, in one 32-byte load: its first key, its
// keys, and the last node index (plus one) that can have children.
struct alignas(32) BatchGeo {
    uint64_t off, n, cmax, pad;
};

struct tl_batch_plan_impl {
    uint32_t num = 0, key_bytes = 8;
    uint64_t b = 8;
    BatchInst *inst = nullptr;   // device
    BatchGeo *geo = nullptr;     // device, behind inst: per instance, for the queries
    BatchTotals tot{};
    uint32_t tile_keys[kMaxClass];
    uint32_t pin_levels[kMaxClass];  // kept for tl_batch_get_tuning; the queries do not use it
    uint32_t query_chunk = 2048;     // likewise
    uint32_t threads = 256;          // permute kernel block size
    uint32_t *owner = nullptr;   // device: owner instance of every tile ticket, then of every copy chunk
    uint32_t *tile = nullptr;    // device: the tile of its owner every tile ticket processes
    char *otab = nullptr;        // device: the ordered instances' tile tables (uint2 tab, then uint32 order)
    FixSeg *items = nullptr;     // device, behind otab: the ordered instances' copy items
    uint64_t *citem = nullptr;   // device, behind items: first copy item of every copy chunk of an ordered instance
    uint64_t ordered = 0;        // instances on the ordered schedule
    uint64_t ordered_keys = 0;   // their keys
    uint64_t off_flags = 0, off_done = 0, off_ctrl = 0, ws_bytes = 0;
    uint64_t total_keys = 0;
    uint64_t max_n = 0;          // keys of the largest instance
};

// ---------------------------------------------------------------- setup
__global__ void __launch_bounds__(256) batch_setup_kernel(const int64_t *__restrict__ offsets, uint32_t num, uint64_t b,
                                                          uint32_t key_bytes, FastDiv64 fd, FastDiv32 fd32,
                                                          FastDiv32 fd32b, const __grid_constant__ PowDivs pdivs,
                                                          const uint32_t *__restrict__ tile_keys,
                                                          BatchInst *__restrict__ inst, BatchGeo *__restrict__ geo,
                                                          BatchTotals *__restrict__ tot) {
    // one block: per-instance plans, then exclusive scans in instance order
    __shared__ unsigned long long s_part[3][1024];
    const uint32_t T = blockDim.x;
    const uint32_t per = (num + T - 1) / T;
    const uint32_t j0 = threadIdx.x * per, j1 = min(num, j0 + per);
    const uint64_t vec = 16 / key_bytes;
    unsigned long long st = 0, ss = 0, sc = 0;
    for (uint32_t j = j0; j < j1; ++j) {
        BatchInst I;
        memset(&I, 0, sizeof I);
        const uint64_t n = (uint64_t)(offsets[j + 1] - offsets[j]);
        I.off = (uint64_t)offsets[j];
        I.S.g = make_btree_geom(n, b);
        I.S.fd = fd;
        I.S.fd32 = fd32;
        I.S.fd32b = fd32b;
        btree_set_pow_divs(I.S, pdivs);
        const uint32_t cls = n ? bit_length(n) - 1 : 0;
        I.S.tile_keys = tile_keys[cls < kMaxClass ? cls : kMaxClass - 1];  // a power of two
        I.S.tile_shift = (uint32_t)__ffsll((long long)I.S.tile_keys) - 1;
        I.S.ntiles = (n + I.S.tile_keys - 1) / I.S.tile_keys;
        btree_choose_plan(I.S, key_bytes);
        if (n <= 1) {
            I.S.ntiles = 0;
            I.S.nscratch = 0;
        }
        uint64_t ncopy = 0;
        for (int k = 0; k < btree_copy_range_count(I.S); ++k) {
            CopyRange r;
            if (btree_copy_range(I.S, k, r)) ncopy += r.len;
        }
        I.nchunks = I.S.nscratch ? (ncopy + kCopyChunk - 1) / kCopyChunk : 0;
        st += I.S.ntiles;
        ss += I.S.nscratch ? I.S.nscratch + vec - 1 : 0;  // room to align the base
        sc += I.nchunks;
        inst[j] = I;
        geo[j] = BatchGeo{I.off, n, (n + 1) / (b + 1), 0};
    }
    s_part[0][threadIdx.x] = st;
    s_part[1][threadIdx.x] = ss;
    s_part[2][threadIdx.x] = sc;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long a = 0, c = 0, d = 0;
        for (uint32_t t = 0; t < T; ++t) {
            const unsigned long long x = s_part[0][t], y = s_part[1][t], z = s_part[2][t];
            s_part[0][t] = a;
            s_part[1][t] = c;
            s_part[2][t] = d;
            a += x;
            c += y;
            d += z;
        }
        tot->tiles = a;
        tot->scratch = c;
        tot->chunks = d;
        uint64_t mt = 0;
        for (int k = 0; k < kMaxClass; ++k) mt = max(mt, (uint64_t)tile_keys[k]);
        tot->max_tile = mt;
    }
    __syncthreads();
    unsigned long long bt = s_part[0][threadIdx.x], bs = s_part[1][threadIdx.x], bc = s_part[2][threadIdx.x];
    for (uint32_t j = j0; j < j1; ++j) {
        const uint64_t ns = inst[j].S.nscratch;
        inst[j].tile_base = bt;
        inst[j].scr_base = bs + ((inst[j].off % vec) + vec - (bs % vec)) % vec;
        inst[j].chunk_base = bc;
        bt += inst[j].S.ntiles;
        bs += ns ? ns + vec - 1 : 0;
        bc += inst[j].nchunks;
    }
}

// owner[tiles + c] = instance of copy chunk c; tile[t], for a tile ticket t, from
// the owner's own ticket (as the host interleaved them) to the tile it names
// under the owner's schedule.  (The owners of tile tickets come from the host.)
__global__ void batch_owner_kernel(const BatchInst *__restrict__ inst, uint32_t num, uint64_t tiles,
                                   uint32_t *__restrict__ owner, uint32_t *__restrict__ tile) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t i0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, ni = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t t = i0; t < tiles; t += ni) tile[t] = (uint32_t)btree_tile_of_ticket(inst[owner[t]].S, tile[t]);
    for (uint64_t j = i0 >> 5; j < num; j += ni >> 5) {
        const BatchInst &I = inst[j];
        for (uint64_t c = lane; c < I.nchunks; c += 32) owner[tiles + I.chunk_base + c] = (uint32_t)j;
    }
}

// ---------------------------------------------------------------- permute
// Ordered schedule: copy chunk c of instance I is a run of its copy items, a warp each.
template <typename K>
static __device__ __forceinline__ void batch_copy_items(K *__restrict__ keys, K *__restrict__ scr, const BatchInst &I,
                                                     const FixSeg *__restrict__ items,
                                                     const uint64_t *__restrict__ citem, uint64_t c, uint32_t tid,
                                                     uint32_t nt) {
    const uint64_t i0 = citem[I.chunk_base + c];
    const uint64_t i1 = c + 1 < I.nchunks ? citem[I.chunk_base + c + 1] : I.item_base + I.nitems;
    K *const dst = keys + I.off;
    const K *const src = scr + I.scr_base;
    for (uint64_t i = i0 + (tid >> 5); i < i1; i += nt >> 5) {
        const uint64_t dl = __ldg(reinterpret_cast<const unsigned long long *>(&items[i].dst_len));
        const uint64_t so = __ldg(reinterpret_cast<const unsigned long long *>(&items[i].src));
        warp_copy_keys(dst + (dl & kSegDstMask), src + so, 0, (uint32_t)(dl >> 48));
    }
}

// Fixed directions: copy chunk c of instance I is kCopyChunk keys of its copy
// ranges, taken as one concatenated range.
template <typename K>
static __device__ __forceinline__ void batch_copy_ranges(K *__restrict__ keys, K *__restrict__ scr, const BatchInst &I,
                                                      uint64_t c, uint32_t tid, uint32_t nt) {
    const uint64_t lo = c * kCopyChunk, hi = lo + kCopyChunk;
    uint64_t acc = 0;
    const int nr = btree_copy_range_count(I.S);
    for (int q = 0; q < nr && acc < hi; ++q) {
        CopyRange r;
        if (!btree_copy_range(I.S, q, r)) continue;
        const uint64_t a = lo > acc ? lo - acc : 0;
        const uint64_t e = min(hi - acc, r.len);
        if (a < e) copy_keys(keys + I.off + r.dst + a, scr + I.scr_base + r.src + a, e - a, tid, nt);
        acc += r.len;
    }
}

constexpr uint32_t kNoInst = 0xFFFFFFFFu;
constexpr uint32_t kPlanWords = sizeof(BatchInst) / 16;

// Work items in ticket order through a ring of stages.  Each stage has two warps
// of its own: the first claims an item, fetches its instance's plan, loads the
// tile, publishes it and waits for the tiles under its bulk keys (a copy chunk:
// for its instance's tiles); the second works out the tile's runs of top keys
// and waits for the tiles under them.  The store warps take the stages in turn
// and meet at no barrier.  A stage claims its next item, and fetches its plan,
// while its present one is stored; stages claim in turn, so a block stores its
// items in ticket order.  The smallest item not yet stored is its block's next,
// its stage is empty, and it waits only for smaller ones: it always progresses.
// What bounds it is traffic (2 n w plus 2 w a scratch key) once loads, waits and
// stores overlap: with a block holding one item at a time, load, publish, wait
// and store in turn, 1024 arrays of 2^10..2^22 keys took 1885 us at b = 8 and
// 1808 at b = 16; in the ring 1752 and 1589, and with the ordered schedule, whose
// instructions now hide, in more instances (kOrderGain) 1637 and 1572.  Claiming
// ahead is 2 % of it; two stages in three blocks took as long.
struct BatchStage {
    BatchInst I;
    TileShared ts;
    uint64_t t, next, p0, p1, base;
    int kind;  // kItemTile, kItemChunk, kItemNone
};
constexpr int kItemTile = 0, kItemChunk = 1, kItemNone = 2;

template <typename K, int kStoreWarps>
__global__ void __launch_bounds__(32 * (2 * kBatchStages + kStoreWarps), kBatchBlocksPerSM)
batch_permute_kernel(K *__restrict__ keys, K *__restrict__ scr, const BatchInst *__restrict__ inst,
                     const uint32_t *__restrict__ owner, const uint32_t *__restrict__ tile,
                     const FixSeg *__restrict__ items, const uint64_t *__restrict__ citem, BatchTotals tot,
                     Ctrl *ctrl, WaitCfg wc, unsigned int *flags, unsigned int *done, uint32_t ring,
                     uint32_t stage_bytes, bool ahead) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ __align__(16) unsigned char s_raw[kBatchStages * sizeof(BatchStage)];
    BatchStage *s_st = reinterpret_cast<BatchStage *>(s_raw);
    // per stage: claimed (its first warp has its ticket), plan (the item is known), ready, empty
    __shared__ uint64_t s_claimed[kBatchStages], s_plan[kBatchStages], s_ready[kBatchStages], s_empty[kBatchStages];
    const uint64_t total = tot.tiles + tot.chunks;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < ring; ++s) {
            mbar_init(&s_claimed[s], 1);
            mbar_init(&s_plan[s], 1);
            mbar_init(&s_ready[s], 2);
            mbar_init(&s_empty[s], kStoreWarps);
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
    if (warp < kBatchStages) {  // a stage's first warp
        const uint32_t s = warp;
        if (s >= ring) return;
        BatchStage &T = s_st[s];
        K *sm = tile_smem<K>(smem_raw) + (size_t)s * (stage_bytes / sizeof(K));
        uint32_t held = kNoInst, stored = kNoInst;  // the instance whose plan is at hand; of the tile being stored
        while (true) {
            // the next item's ticket and plan, while this stage's item is being stored
            if (!ahead && !wait_bar(&s_empty[s], phase ^ 1)) return;
            if (!wait_bar(&s_claimed[s ? s - 1 : ring - 1], s ? phase : phase ^ 1)) return;
            unsigned long long t = 0;
            if (lane == 0) {
                t = atomicAdd(&ctrl->ticket, 1ull);
                T.next = t;  // and so has its value before the next stage claims
                mbar_arrive(&s_claimed[s]);
            }
            t = __shfl_sync(0xFFFFFFFFu, t, 0);
            const bool is_tile = t < tot.tiles;
            const uint32_t j = t < total ? owner[t] : kNoInst;
            const uint64_t k = is_tile ? tile[t] : 0;
            const bool other = t < total && j != held;
            uint4 plan[(kPlanWords + 31) / 32];  // in registers until the stage's own copy is free
            if (other) {
                const uint4 *src = reinterpret_cast<const uint4 *>(inst + j);
#pragma unroll
                for (uint32_t i = 0; i < (kPlanWords + 31) / 32; ++i)
                    if (lane + 32 * i < kPlanWords) plan[i] = src[lane + 32 * i];
                held = j;
            }
            if (!wait_bar(&s_empty[s], phase ^ 1)) return;
            if (other) {
                uint4 *dst = reinterpret_cast<uint4 *>(&T.I);
#pragma unroll
                for (uint32_t i = 0; i < (kPlanWords + 31) / 32; ++i)
                    if (lane + 32 * i < kPlanWords) dst[lane + 32 * i] = plan[i];
                __syncwarp();
            }
            const BatchInst &I = T.I;
            const BtreeStream &S = I.S;
            K *A = keys + I.off;
            unsigned int *fl = flags + I.tile_base;
            uint64_t p0 = 0, p1 = 0, w_lo = 1, w_hi = 0;
            if (lane == 0) {
                T.t = t;
                T.kind = is_tile ? kItemTile : t < total ? kItemChunk : kItemNone;
            }
            if (is_tile) {
                btree_tile(S, k, p0, p1);
                const uint64_t base = tile_base(A, p0);
                if (lane == 0) {
                    T.p0 = p0, T.p1 = p1, T.base = base;
                    T.ts.ok0 = T.ts.ok1 = 1;
                    mbar_arrive(&s_plan[s]);
                }
                load_tile_issue(A, p0, p1, sm, lane, 32);
            }
            if (stored != kNoInst && lane == 0) {  // the last tile's stores, every warp's, before its count
                __threadfence();
                atomicAdd(&done[stored], 1u);
            }
            stored = kNoInst;
            if (is_tile) {
                if (lane == 0) T.ts.reg = btree_stream_regime(S, p0, p1);
                // a look at the flags while the copies are in flight mostly finds them set
                bool pending = false;
                if (btree_tile_wait(S, p0, p1, w_lo, w_hi))
                    for (uint64_t f = w_lo + lane; f <= w_hi; f += 32)
                        if (f != k && !(S.plan == PLAN_O && !btree_o_direct(S, k, f)))  // else its keys go to scratch
                            pending |= ld_acquire(&fl[f]) != wc.wait_value;
                load_tile_wait();
                __syncwarp();
                if (lane == 0) st_relaxed(&fl[k], wc.flag_value);  // published: every copy has landed
                if (pending)
                    for (uint64_t f = w_lo + lane; f <= w_hi; f += 32)
                        if (f != k && !(S.plan == PLAN_O && !btree_o_direct(S, k, f)))
                            if (!wait_flag(&fl[f], wc.wait_value, ctrl, wc)) T.ts.ok1 = 0;
                stored = j;
            } else if (lane == 0) {
                mbar_arrive(&s_plan[s]);
                if (t < total) T.ts.ok1 = wait_flag(&done[j], (unsigned int)S.ntiles, ctrl, wc) ? 1 : 0;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&s_ready[s]);
            if (t >= total) return;
            phase ^= 1;
        }
    } else if (warp < 2 * kBatchStages) {  // a stage's second warp
        const uint32_t s = warp - kBatchStages;
        if (s >= ring) return;
        BatchStage &T = s_st[s];
        while (wait_bar(&s_plan[s], phase)) {
            const int kind = T.kind;
            const BatchInst &I = T.I;
            if (kind == kItemTile)
                btree_tile_runs_warp(I.S, T.p0, T.p1, reinterpret_cast<uintptr_t>(keys + I.off),
                                     reinterpret_cast<uintptr_t>(scr + I.scr_base), (uint32_t)sizeof(K),
                                     flags + I.tile_base, ctrl, wc, T.ts);
            __syncwarp();
            if (lane == 0) mbar_arrive(&s_ready[s]);
            if (kind == kItemNone) break;
            phase ^= 1;
        }
    } else {  // store warps
        const uint32_t tb = threadIdx.x - 64 * kBatchStages, nb = 32 * kStoreWarps;
        uint32_t s = 0;
        while (wait_bar(&s_ready[s], phase)) {
            const BatchStage &T = s_st[s];
            if (T.kind == kItemNone) break;
            const BatchInst &I = T.I;
            if (T.kind == kItemTile) {
                if (T.ts.ok0 && T.ts.ok1) {
                    const K *tl = tile_smem<K>(smem_raw) + (size_t)s * (stage_bytes / sizeof(K)) + (T.p0 - T.base);
                    btree_store_bulk(I.S, keys + I.off, scr + I.scr_base, ctrl, T.p0, T.p1, tl, T.ts, tb, nb);
                    btree_store_top<K, true>(I.S, tl, T.ts, tb, nb);
                }
            } else if (T.ts.ok1) {
                const uint64_t c = T.t - tot.tiles - I.chunk_base;
                if (I.S.plan == PLAN_O)
                    batch_copy_items(keys, scr, I, items, citem, c, tb, nb);
                else
                    batch_copy_ranges(keys, scr, I, c, tb, nb);
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

// ---------------------------------------------------------------- queries
// A query descends its own instance; nothing but the answer is written.  G
// lanes read a node together: the aligned 32-byte sectors that hold it
// (instances start anywhere, so a node of B * w bytes spans up to
// B * w / 32 + 1 of them), lane g the sectors g, g + G, ...  Nodes start at
// multiples of B keys, so which keys of a lane's sectors belong to the node is
// the same mask at every level.  As in the single-array query the warp's
// control flow is uniform, the count is a shuffle sum and an equal key is found
// by ballot.
//
// What bounds it is where the descents go, not how many bytes they read: the
// instances' upper levels lie all over the key array, so a batch as given
// touches every 2 MB page of it at every level (measured on B200, 2^24 queries
// over 1024 arrays of 5.2e8 u64 keys, b = 8: 2.36 ms at a quarter of the DRAM
// and of the L1 bandwidth; over 32 arrays in 126 MB, 0.9 ms).  So a block
// takes a chunk of the batch, orders it by instance in shared memory (a
// counting sort of 16-bit offsets into kBatchBins bins of consecutive
// instances) and walks the chunk in that order, all blocks through the same
// instances at about the same time; the answers go to the chunk's own stretch.
// Same measurement: chunks of 4096 / 8192 / 16384 / 32768 queries 1.77 / 1.16 /
// 1.14 / 1.25 ms; the previous form (a global counting sort by two atomics a
// query, then a thread a query over the sorted copy) 4.50 ms.  In this order a
// thread a query (G = 1) beats groups of lanes (1.14 against 1.54 ms with G =
// 2, 2.28 with G = 4; b = 16 1.46 against 1.57): more descents in flight, and
// L1 serves the shared upper nodes.  One block of 1024 threads an SM: 512 x 2
// 1.24, 256 x 4 1.41 ms (each block has its own window of instances).
constexpr uint32_t kBatchBins = 1024;
constexpr int kBatchSortThreads = 1024;
constexpr uint32_t kBatchSortChunk = 16384;

// NB = node bytes (a multiple of 32), or 0 for any b: then the sectors are
// taken G at a time, their masks computed on the way.  I: an index type that
// holds every child index of a batch's instances.
template <typename K, int NB, int G, typename I>
__device__ __forceinline__ void batch_descend(const K *__restrict__ keys, uint64_t total,
                                              const BatchGeo *__restrict__ geo, uint32_t num, uint32_t b_rt,
                                              const K *__restrict__ Q, const uint32_t *__restrict__ qinst,
                                              uint64_t qi, bool have, uint64_t *__restrict__ ans) {
    constexpr int KPL = 32 / sizeof(K);                     // keys per sector
    constexpr int NI = NB ? (NB / 32 + 1 + G - 1) / G : 1;  // sectors per lane
    const int B = NB ? NB / (int)sizeof(K) : (int)b_rt;
    const uint32_t lane = threadIdx.x & 31, g = lane % G, gshift = lane - g;
    const uint32_t j = have ? __ldg(qinst + qi) : num;
    const K q = have ? __ldg(Q + qi) : K(0);
    uint64_t rec[4] = {0, 0, 0, 0};  // BatchGeo; an instance id out of range answers 0
    if (j < num) ldg32(reinterpret_cast<const uint64_t *>(geo + j), rec);
    const K *A = keys + rec[0];
    const I n = (I)rec[1], cmax = (I)rec[2];
    const uint32_t off = (uint32_t)(reinterpret_cast<uintptr_t>(A) & 31) / sizeof(K);
    const K *A32 = A - off;  // the sector of the instance's first key
    // an instance whose first or last sector reaches outside the key array is read key by key
    const bool edge = A32 < keys || A32 + ((uint64_t)n + off + KPL - 1) / KPL * KPL > keys + total;
    // slots rel .. rel + KPL - 1 against [0, valid)
    auto mask = [](int rel, int valid) -> uint32_t {
        return rel >= valid ? 0u : ((1u << KPL) - 1) & (rel < 0 ? ~0u << -rel : ~0u) &
                                       (valid - rel < KPL ? (1u << (valid - rel)) - 1 : ~0u);
    };
    uint32_t vm[NI];
    if constexpr (NB != 0) {
#pragma unroll
        for (int t = 0; t < NI; ++t) vm[t] = mask((int)(g + t * G) * KPL - (int)off, B);
    }
    I i = 0, res = n;
    bool live = n > 0;
    while (__any_sync(0xFFFFFFFFu, live)) {
        uint32_t lt = 0, eqm = 0;
        if (live) {
            const bool part = n - i < (I)B;  // slots at or past n do not count
            const int valid = part ? (int)(n - i) : B;
            uint32_t first = off;  // a node of an odd size starts anywhere in its sector
            const K *p = A32 + i;
            if constexpr (NB == 0) {
                first = (uint32_t)((off + i) % KPL);
                p = A + i - first;
            }
            for (int s0 = (int)g; NB ? s0 == (int)g : s0 * KPL - (int)first < valid; s0 += G) {
                K v[NI][KPL];
                uint32_t m[NI];
#pragma unroll
                for (int t = 0; t < NI; ++t) {
                    const int s = s0 + t * G;
                    if constexpr (NB == 0)
                        m[t] = mask(s * KPL - (int)first, valid);
                    else
                        m[t] = part ? vm[t] & mask(s * KPL - (int)first, valid) : vm[t];
                    if (m[t]) {
                        if (!edge) {
                            ldg32(p + s * KPL, v[t]);
                        } else {
#pragma unroll
                            for (int e = 0; e < KPL; ++e)
                                v[t][e] = (m[t] >> e) & 1u ? __ldg(p + s * KPL + e) : K(0);
                        }
                    }
                }
#pragma unroll
                for (int t = 0; t < NI; ++t) {
                    uint32_t l = 0, x = 0;
#pragma unroll
                    for (int e = 0; e < KPL; ++e) {
                        l |= (v[t][e] < q ? 1u : 0u) << e;
                        x |= (v[t][e] == q ? 1u : 0u) << e;
                    }
                    lt += __popc(l & m[t]);
                    eqm |= x & m[t];
                }
            }
        }
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) lt += __shfl_xor_sync(0xFFFFFFFFu, lt, o);
        bool hit = eqm != 0;
        if constexpr (G > 1) hit = ((__ballot_sync(0xFFFFFFFFu, hit) >> gshift) & ((1u << G) - 1)) != 0;
        if (live) {
            if (hit) {  // keys are unique: the equal key sits at slot lt
                res = i + lt;
                live = false;
            } else if (i + 1 > cmax) {  // every child starts past n
                live = false;
            } else {
                i = (i + 1) * (I)(B + 1) + (I)lt * (I)B - 1;
                live = i < n;
            }
        }
    }
    if (g == 0 && have) ans[qi] = (uint64_t)res;
}

// The batch as given, a grid stride (small batches: one launch, no sort).
template <typename K, int NB, int G, typename I>
__global__ void __launch_bounds__(kBatchThreads)
batch_query_kernel(const K *__restrict__ keys, uint64_t total, const BatchGeo *__restrict__ geo, uint32_t num,
                   uint32_t b, const K *__restrict__ Q, const uint32_t *__restrict__ qinst, uint64_t nq,
                   uint64_t *__restrict__ ans) {
    const uint64_t step = (uint64_t)gridDim.x * (blockDim.x / G);
    const uint64_t first = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) / 32 * (32 / G);  // the warp's
    for (uint64_t base = first; base < nq; base += step) {
        const uint64_t qi = base + (threadIdx.x & 31) / G;
        batch_descend<K, NB, G, I>(keys, total, geo, num, b, Q, qinst, qi, qi < nq, ans);
    }
}

// Chunk by chunk, each in the order of its queries' instances.
template <typename K, int NB, int G, typename I>
__global__ void __launch_bounds__(kBatchSortThreads, 1)
batch_query_sorted_kernel(const K *__restrict__ keys, uint64_t total, const BatchGeo *__restrict__ geo, uint32_t num,
                          uint32_t b, uint32_t bin_shift, uint32_t chunk, const K *__restrict__ Q,
                          const uint32_t *__restrict__ qinst, uint64_t nq, uint64_t *__restrict__ ans) {
    static_assert(kBatchBins == kBatchSortThreads, "one bin a thread in the scan");
    static_assert(kBatchSortChunk <= 65536, "16-bit offsets into the chunk");
    extern __shared__ uint16_t order[];  // [chunk]
    __shared__ uint32_t cnt[kBatchBins], wsum[32];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (uint64_t c0 = (uint64_t)blockIdx.x * chunk; c0 < nq; c0 += (uint64_t)gridDim.x * chunk) {
        const uint32_t len = (uint32_t)min((uint64_t)chunk, nq - c0);
        __syncthreads();
        cnt[threadIdx.x] = 0;
        __syncthreads();
#pragma unroll 4
        for (uint32_t x = threadIdx.x; x < len; x += kBatchSortThreads)
            atomicAdd(&cnt[min(__ldg(qinst + c0 + x) >> bin_shift, kBatchBins - 1)], 1u);
        __syncthreads();
        const uint32_t c = cnt[threadIdx.x];
        uint32_t inc = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, inc, o);
            if (lane >= (uint32_t)o) inc += y;
        }
        if (lane == 31) wsum[warp] = inc;
        __syncthreads();
        const uint32_t before = __reduce_add_sync(0xFFFFFFFFu, lane < warp ? wsum[lane] : 0u);
        cnt[threadIdx.x] = before + inc - c;
        __syncthreads();
#pragma unroll 4
        for (uint32_t x = threadIdx.x; x < len; x += kBatchSortThreads)
            order[atomicAdd(&cnt[min(__ldg(qinst + c0 + x) >> bin_shift, kBatchBins - 1)], 1u)] = (uint16_t)x;
        __syncthreads();
        for (uint32_t base = warp * (32 / G); base < len; base += kBatchSortThreads / G) {
            const uint32_t at = base + lane / G;
            const bool have = at < len;
            batch_descend<K, NB, G, I>(keys, total, geo, num, b, Q, qinst, c0 + (have ? order[at] : 0u), have, ans);
        }
    }
}

// ---------------------------------------------------------------- host
static int batch_sms() {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

static void default_tuning(tl_batch_plan_impl &P) {
    for (int c = 0; c < kMaxClass; ++c) {
        P.tile_keys[c] = (uint32_t)(32768 / P.key_bytes);
        P.pin_levels[c] = 3;
    }
    P.query_chunk = 2048;
}

static void free_order_buffers(tl_batch_plan_impl &P) {
    if (P.otab) cudaFree(P.otab);
    P.otab = nullptr;
    P.items = nullptr;
    P.citem = nullptr;
    P.ordered = P.ordered_keys = 0;
}

// Device memory of a plan: one cudaMalloc (0.1 to 0.2 ms) for what was built
// together.  Not from the pool: the cudaFree of such memory waits for the kernels
// that may still read the plan, that of pool memory does not.
static int plan_memory(void **p, size_t bytes) {
    if (cudaMalloc(p, bytes) == cudaSuccess) return TL_SUCCESS;
    cudaGetLastError();
    *p = nullptr;
    return TL_ERROR_OUT_OF_MEMORY;
}

// Keys through scratch under an instance's fixed-direction schedule and under
// the ordered one.
static uint64_t fixed_scratch_keys(const BtreeStream &S) {
    uint64_t c = 0;
    CopyRange r;
    for (int k = 0; k < btree_copy_range_count(S); ++k)
        if (btree_copy_range(S, k, r)) c += r.len;
    return c;
}

static uint64_t order_scratch_keys(const BtreeStream &S, const OrderVectors &v) {
    uint64_t c = 0;
    for (const uint4 &r : v.ranges)
        c += std::min<uint64_t>((uint64_t)r.y * S.tile_keys, S.g.n) - (uint64_t)r.x * S.tile_keys;
    for (const FixSeg &f : v.segs) c += f.dst_len >> 48;
    return c;
}

// Puts every instance of kBatchOrderMinTiles tiles or more (with a top tree) on
// the ordered schedule of the single-array permutation: its tile order and
// scratch tables are computed on the host (instances shared among a few host
// threads), its scratch keys listed as copy items and grouped into chunks; then
// every instance's scratch and chunk bases are recomputed in instance order
// (the same rules as batch_setup_kernel) and the plan is written back.
static int order_instances(tl_batch_plan_impl &P, const std::vector<int64_t> &off, cudaStream_t st) {
    free_order_buffers(P);
    if (fixed_schedule_only()) return TL_SUCCESS;
    std::vector<uint32_t> cand;
    for (uint32_t j = 0; j < P.num; ++j) {
        const uint64_t n = (uint64_t)(off[j + 1] - off[j]);
        const uint32_t cls = n ? bit_length(n) - 1 : 0;
        const uint64_t tk = P.tile_keys[cls < kMaxClass ? cls : kMaxClass - 1];
        if ((n + tk - 1) / tk >= kBatchOrderMinTiles) cand.push_back(j);
    }
    if (cand.empty()) return TL_SUCCESS;
    std::vector<BatchInst> h(P.num);
    TL_CUDA_TRY(cudaMemcpyAsync(h.data(), P.inst, h.size() * sizeof(BatchInst), cudaMemcpyDeviceToHost, st));
    TL_CUDA_TRY(cudaStreamSynchronize(st));
    if (P.b >= 2)  // the host's inverse map (sorted rank of a position) divides by b
        for (uint32_t j : cand) h[j].S.fdb = FastDiv64(P.b);
    std::vector<OrderVectors> ov(cand.size());
    std::vector<int32_t> ord_of(P.num, -1);
    {
        std::atomic<size_t> next{0};
        auto work = [&] {
            for (size_t i; (i = next.fetch_add(1)) < cand.size();) {
                const BtreeStream &S = h[cand[i]].S;
                if (S.g.h < 1 || S.ntiles < kBatchOrderMinTiles || S.ntiles >= (1ull << 32)) continue;
                btree_compute_order(S, ov[i]);
                const double moved = (double)order_scratch_keys(S, ov[i]), fixed = (double)fixed_scratch_keys(S);
                const bool wider = ov[i].scratch_tiles * S.tile_keys > S.nscratch;
                if (!ordered_schedule_forced() && moved > (wider ? kOrderGainSpace : kOrderGain) * fixed)
                    ov[i] = OrderVectors();
            }
        };
        const unsigned hw = std::max(1u, std::thread::hardware_concurrency());
        const size_t nth = std::min<size_t>({(size_t)hw, (size_t)16, cand.size()});
        std::vector<std::thread> pool;
        for (size_t k = 1; k < nth; ++k) pool.emplace_back(work);
        work();
        for (auto &t : pool) t.join();
    }
    // the tables of the ordered instances, each its tab then its order (8-byte aligned)
    std::vector<size_t> toff(cand.size(), 0);
    size_t tbytes = 0;
    for (size_t i = 0; i < cand.size(); ++i) {
        if (ov[i].order.empty()) continue;
        ord_of[cand[i]] = (int32_t)i;
        toff[i] = tbytes;
        const size_t N = ov[i].order.size();
        tbytes += N * sizeof(uint2) + (N * sizeof(uint32_t) + 7) / 8 * 8;
    }
    if (!tbytes) return TL_SUCCESS;
    std::vector<char> tb(tbytes, 0);
    for (size_t i = 0; i < cand.size(); ++i) {
        if (ord_of[cand[i]] < 0) continue;
        const size_t N = ov[i].order.size();
        memcpy(tb.data() + toff[i], ov[i].tab.data(), N * sizeof(uint2));
        memcpy(tb.data() + toff[i] + N * sizeof(uint2), ov[i].order.data(), N * sizeof(uint32_t));
    }
    std::vector<FixSeg> items;
    std::vector<uint64_t> citem;
    const uint64_t vec = 16 / P.key_bytes;
    uint64_t bs = 0;
    for (uint32_t j = 0; j < P.num; ++j) {
        BatchInst &I = h[j];
        I.chunk_base = citem.size();
        if (ord_of[j] >= 0) {
            const OrderVectors &v = ov[ord_of[j]];
            btree_set_ordered(I.S, nullptr, nullptr, v.scratch_tiles);  // its tables below
            const uint64_t T = I.S.tile_keys, n = I.S.g.n;
            I.item_base = items.size();
            for (const uint4 &r : v.ranges)  // whole-tile runs, in pieces
                for (uint64_t d = (uint64_t)r.x * T, s = (uint64_t)r.z * T, e = std::min<uint64_t>((uint64_t)r.y * T, n);
                     d < e;) {
                    const uint64_t len = std::min<uint64_t>(kRangePiece, e - d);
                    items.push_back(FixSeg{d | (len << 48), s});
                    d += len;
                    s += len;
                }
            items.insert(items.end(), v.segs.begin(), v.segs.end());
            I.nitems = items.size() - I.item_base;
            I.nchunks = 0;
            uint64_t keys = kCopyChunk, cnt = 0;
            for (uint64_t k = I.item_base; k < items.size(); ++k) {
                const uint64_t len = items[k].dst_len >> 48;
                if (keys + len > kCopyChunk || cnt == kChunkItemsMax) {
                    citem.push_back(k);
                    ++I.nchunks;
                    keys = cnt = 0;
                }
                keys += len;
                ++cnt;
            }
            ++P.ordered;
            P.ordered_keys += n;
        } else {
            citem.resize(citem.size() + I.nchunks, 0);  // plan R / L chunks: not read
        }
        const uint64_t ns = I.S.nscratch;
        I.scr_base = bs + ((I.off % vec) + vec - (bs % vec)) % vec;
        bs += ns ? ns + vec - 1 : 0;
    }
    P.tot.scratch = bs;
    P.tot.chunks = citem.size();
    const size_t items_at = (tbytes + 15) / 16 * 16, citem_at = items_at + items.size() * sizeof(FixSeg);
    const int rc = plan_memory(reinterpret_cast<void **>(&P.otab), citem_at + citem.size() * sizeof(uint64_t));
    if (rc) {
        free_order_buffers(P);
        return rc;
    }
    P.items = reinterpret_cast<FixSeg *>(P.otab + items_at);
    P.citem = reinterpret_cast<uint64_t *>(P.otab + citem_at);
    for (size_t i = 0; i < cand.size(); ++i) {
        if (ord_of[cand[i]] < 0) continue;
        BtreeStream &S = h[cand[i]].S;
        S.tab = reinterpret_cast<const uint2 *>(P.otab + toff[i]);
        S.order = reinterpret_cast<const uint32_t *>(P.otab + toff[i] + ov[i].order.size() * sizeof(uint2));
    }
    // copied on st, then waited for: a plain cudaMemcpy from pageable memory may return before its DMA lands
    TL_CUDA_TRY(cudaMemcpyAsync(P.otab, tb.data(), tbytes, cudaMemcpyHostToDevice, st));
    if (!items.empty())
        TL_CUDA_TRY(cudaMemcpyAsync(P.items, items.data(), items.size() * sizeof(FixSeg), cudaMemcpyHostToDevice, st));
    if (!citem.empty())
        TL_CUDA_TRY(cudaMemcpyAsync(P.citem, citem.data(), citem.size() * sizeof(uint64_t), cudaMemcpyHostToDevice, st));
    TL_CUDA_TRY(cudaMemcpyAsync(P.inst, h.data(), h.size() * sizeof(BatchInst), cudaMemcpyHostToDevice, st));
    TL_CUDA_TRY(cudaStreamSynchronize(st));
    return TL_SUCCESS;
}

// The order in which the persistent kernel takes the stream tiles: each
// instance's tiles in its own ticket order, the instances interleaved in
// proportion to their tile counts, kInterleaveRun tiles at a time.  A tile only
// waits for tiles of its own instance with smaller tickets; interleaved, those
// were claimed some thousands of tickets earlier and have long been read,
// where instance after instance they would be the tiles just claimed, often
// still loading (measured on B200, 4096 arrays of 2^10..2^22 keys, b = 8: the
// waits that found their flag unset fall from 4.2e5 to 1e4 and the launch from
// 11.1 to 9.6 ms).  Longer runs, which reload the owner's plan into shared
// memory less often, measured slower (runs of 4: 9.7 ms).
static int interleave_tiles(const tl_batch_plan_impl &P, const std::vector<int64_t> &off,
                            std::vector<uint32_t> &own, std::vector<uint32_t> &loc) {
    struct Run {
        double key;  // the instance's progress at the run's middle
        uint32_t j, r;
    };
    const uint64_t G = kInterleaveRun;
    std::vector<Run> runs;
    std::vector<uint64_t> nt(P.num);
    uint64_t sum = 0;
    for (uint32_t j = 0; j < P.num; ++j) {
        const uint64_t n = (uint64_t)(off[j + 1] - off[j]);
        const uint32_t cls = n ? bit_length(n) - 1 : 0;
        const uint64_t tk = P.tile_keys[cls < kMaxClass ? cls : kMaxClass - 1];
        nt[j] = n <= 1 ? 0 : (n + tk - 1) / tk;  // as batch_setup_kernel
        sum += nt[j];
        const uint64_t R = (nt[j] + G - 1) / G;
        for (uint64_t r = 0; r < R; ++r) runs.push_back(Run{((double)r + 0.5) / (double)R, j, (uint32_t)r});
    }
    // tile indices and the kernel's tickets are 32-bit
    if (sum != P.tot.tiles || sum + P.tot.chunks >= (1ull << 31)) return TL_ERROR_UNSUPPORTED;
    // by progress, ties in instance order: into as many buckets of equal width as there are runs, then each bucket
    // (sorted whole, 1.3e5 runs took 4.7 ms of a plan of 11)
    {
        const size_t M = runs.size();
        auto bucket = [&](const Run &q) { return std::min(M - 1, (size_t)(q.key * (double)M)); };
        std::vector<uint32_t> at(M + 1, 0);
        for (const Run &q : runs) ++at[bucket(q) + 1];
        for (size_t k = 0; k < M; ++k) at[k + 1] += at[k];
        std::vector<Run> in(std::move(runs));
        runs.resize(M);
        for (const Run &q : in) runs[at[bucket(q)]++] = q;  // at[k] is now the end of bucket k
        for (size_t k = 0, lo = 0; k < M; lo = at[k++])
            if (at[k] - lo > 1)
                std::stable_sort(runs.begin() + lo, runs.begin() + at[k],
                                 [](const Run &a, const Run &b) { return a.key < b.key; });
    }
    own.clear();
    loc.clear();
    own.reserve(sum);
    loc.reserve(sum);
    for (const Run &q : runs)
        for (uint64_t i = (uint64_t)q.r * G, e = std::min<uint64_t>(i + G, nt[q.j]); i < e; ++i) {
            own.push_back(q.j);
            loc.push_back((uint32_t)i);
        }
    return TL_SUCCESS;
}

// Frees a stream-ordered temporary on every exit path.
struct AsyncBuffer {
    void *p = nullptr;
    cudaStream_t st;
    explicit AsyncBuffer(cudaStream_t s) : st(s) {}
    ~AsyncBuffer() {
        if (p) cudaFreeAsync(p, st);
    }
};

static int build_plan(tl_batch_plan_impl &P, const int64_t *dev_offsets, cudaStream_t st) {
    AsyncBuffer tk_buf(st), tot_buf(st);
    keep_pool_memory();
    TL_CUDA_TRY(cudaMallocAsync(&tk_buf.p, sizeof(P.tile_keys), st));
    TL_CUDA_TRY(cudaMallocAsync(&tot_buf.p, sizeof(BatchTotals), st));
    uint32_t *d_tk = static_cast<uint32_t *>(tk_buf.p);
    BatchTotals *d_tot = static_cast<BatchTotals *>(tot_buf.p);
    TL_CUDA_TRY(cudaMemcpyAsync(d_tk, P.tile_keys, sizeof(P.tile_keys), cudaMemcpyHostToDevice, st));
    batch_setup_kernel<<<1, 256, 0, st>>>(dev_offsets, P.num, P.b, P.key_bytes, FastDiv64(P.b + 1),
                                           FastDiv32((uint32_t)(P.b + 1)),
                                           P.b >= 2 ? FastDiv32((uint32_t)P.b) : FastDiv32(), make_pow_divs(P.b), d_tk,
                                           P.inst, P.geo, d_tot);
    TL_CUDA_TRY(cudaGetLastError());
    int64_t last = 0;
    TL_CUDA_TRY(cudaMemcpyAsync(&P.tot, d_tot, sizeof(BatchTotals), cudaMemcpyDeviceToHost, st));
    TL_CUDA_TRY(cudaMemcpyAsync(&last, dev_offsets + P.num, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
    TL_CUDA_TRY(cudaStreamSynchronize(st));
    P.total_keys = (uint64_t)last;
    std::vector<int64_t> off(P.num + 1);
    TL_CUDA_TRY(cudaMemcpyAsync(off.data(), dev_offsets, off.size() * sizeof(int64_t), cudaMemcpyDeviceToHost, st));
    TL_CUDA_TRY(cudaStreamSynchronize(st));
    P.max_n = 0;
    for (uint32_t j = 0; j < P.num; ++j) P.max_n = std::max(P.max_n, (uint64_t)(off[j + 1] - off[j]));
    int rc = order_instances(P, off, st);
    if (rc) return rc;
    std::vector<uint32_t> own, loc;
    rc = interleave_tiles(P, off, own, loc);
    if (rc) return rc;
    if (P.owner) cudaFreeAsync(P.owner, st);
    if (P.tile) cudaFreeAsync(P.tile, st);
    P.owner = P.tile = nullptr;
    const uint64_t nowner = P.tot.tiles + P.tot.chunks;
    if (nowner) {
        keep_pool_memory();
        TL_CUDA_TRY(cudaMallocAsync(reinterpret_cast<void **>(&P.owner), nowner * sizeof(uint32_t), st));
        TL_CUDA_TRY(cudaMallocAsync(reinterpret_cast<void **>(&P.tile),
                                    std::max<uint64_t>(P.tot.tiles, 1) * sizeof(uint32_t), st));
        if (P.tot.tiles) {
            TL_CUDA_TRY(cudaMemcpyAsync(P.owner, own.data(), own.size() * sizeof(uint32_t), cudaMemcpyHostToDevice, st));
            TL_CUDA_TRY(cudaMemcpyAsync(P.tile, loc.data(), loc.size() * sizeof(uint32_t), cudaMemcpyHostToDevice, st));
        }
        const uint64_t work = std::max<uint64_t>((uint64_t)P.num * 32, P.tot.tiles);
        const unsigned g = (unsigned)std::min<uint64_t>((work + 255) / 256, (uint64_t)batch_sms() * 8);
        batch_owner_kernel<<<g, 256, 0, st>>>(P.inst, P.num, P.tot.tiles, P.owner, P.tile);
        TL_CUDA_TRY(cudaGetLastError());
        TL_CUDA_TRY(cudaStreamSynchronize(st));  // the plan is complete when this returns, for any stream
    }
    auto al = [](uint64_t x) { return (x + 255) / 256 * 256; };
    // + 16 bytes: the scratch starts at the keys' own offset within 16 bytes
    P.off_flags = al(P.tot.scratch * P.key_bytes + 16);
    P.off_done = P.off_flags + al(P.tot.tiles * sizeof(unsigned int));
    P.off_ctrl = P.off_done + al((uint64_t)P.num * sizeof(unsigned int));
    P.ws_bytes = P.off_ctrl + al(sizeof(Ctrl));
    return TL_SUCCESS;
}

int batch_plan_create(const int64_t *dev_offsets, uint32_t num, uint64_t b, uint32_t key_bytes, cudaStream_t st,
                      tl_batch_plan **out) {
    if (!dev_offsets || !out || num == 0 || num > (1u << 24) || b == 0 || b >= (1u << 20) ||
        (key_bytes != 4 && key_bytes != 8))
        return TL_ERROR_INVALID_VALUE;
    auto *P = new tl_batch_plan_impl;
    P->num = num;
    P->b = b;
    P->key_bytes = key_bytes;
    default_tuning(*P);
    const size_t geo_at = ((size_t)num * sizeof(BatchInst) + 31) / 32 * 32;
    int rc = plan_memory(reinterpret_cast<void **>(&P->inst), geo_at + (size_t)num * sizeof(BatchGeo));
    if (rc) {
        delete P;
        return rc;
    }
    P->geo = reinterpret_cast<BatchGeo *>(reinterpret_cast<char *>(P->inst) + geo_at);
    rc = build_plan(*P, dev_offsets, st);
    if (rc) {
        cudaFree(P->inst);
        if (P->owner) cudaFree(P->owner);
        if (P->tile) cudaFree(P->tile);
        free_order_buffers(*P);
        delete P;
        return rc;
    }
    *out = reinterpret_cast<tl_batch_plan *>(P);
    return TL_SUCCESS;
}

int batch_plan_destroy(tl_batch_plan *plan) {
    if (!plan) return TL_ERROR_INVALID_VALUE;
    auto *P = reinterpret_cast<tl_batch_plan_impl *>(plan);
    cudaFree(P->inst);  // first: it waits for work in flight, the frees of pool memory do not
    if (P->owner) cudaFree(P->owner);
    if (P->tile) cudaFree(P->tile);
    free_order_buffers(*P);
    delete P;
    return TL_SUCCESS;
}

int batch_ordered(const tl_batch_plan *plan, uint64_t *instances, uint64_t *keys) {
    if (!plan) return TL_ERROR_INVALID_VALUE;
    const auto &P = *reinterpret_cast<const tl_batch_plan_impl *>(plan);
    if (instances) *instances = P.ordered;
    if (keys) *keys = P.ordered_keys;
    return TL_SUCCESS;
}

int batch_workspace_bytes(const tl_batch_plan *plan, uint64_t *bytes) {
    if (!plan || !bytes) return TL_ERROR_INVALID_VALUE;
    *bytes = reinterpret_cast<const tl_batch_plan_impl *>(plan)->ws_bytes;
    return TL_SUCCESS;
}

template <typename K>
static int launch_batch_permute(const tl_batch_plan_impl &P, K *keys, char *ws, cudaStream_t st, int threads) {
    // every instance's scratch base shares its keys' offset within 16 bytes
    K *scr = reinterpret_cast<K *>(ws + (reinterpret_cast<uintptr_t>(keys) & 15));
    unsigned int *flags = reinterpret_cast<unsigned int *>(ws + P.off_flags);
    unsigned int *done = reinterpret_cast<unsigned int *>(ws + P.off_done);
    Ctrl *ctrl = reinterpret_cast<Ctrl *>(ws + P.off_ctrl);
    // flags, done counters and the control block are contiguous: one memset, no
    // host-to-device copy, so the launch can be captured in a CUDA graph
    TL_CUDA_TRY(cudaMemsetAsync(flags, 0, P.ws_bytes - P.off_flags, st));
    WaitCfg wc;
    wc.flag_value = 1;
    wc.wait_value = debug_force_timeout() ? 0xFFFFFFFFu : 1u;
    wc.spin_limit = debug_spin_limit();
    // as many stages as let kBatchBlocksPerSM blocks share an SM, each for the largest tile
    const size_t stage = ((size_t)P.tot.max_tile * sizeof(K) + 128 + 127) / 128 * 128;
    uint32_t ring = (uint32_t)std::max<size_t>(1, std::min<size_t>(kBatchStages, (kBatchBlockSmem - 128) / stage));
    const size_t smem = ring * stage + 128;
    auto kern = threads == 512 ? batch_permute_kernel<K, kBatchStoreWarps512> : batch_permute_kernel<K, kBatchStoreWarps256>;
    const int nthreads = 32 * (2 * kBatchStages + (threads == 512 ? kBatchStoreWarps512 : kBatchStoreWarps256));
    // the same limit whatever the plan's tiles: another thread's smaller plan must not lower it under this launch
    if (smem > kBatchBlockSmem) return TL_ERROR_UNSUPPORTED;  // (tiles are at most 64 KB: never)
    TL_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBatchBlockSmem));
    int per_sm = 0;
    TL_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, nthreads, smem));
    const uint64_t work = P.tot.tiles + P.tot.chunks;
    if (work == 0) return TL_SUCCESS;
    const uint64_t grid = std::min<uint64_t>((uint64_t)std::max(per_sm, 1) * batch_sms(), work);
    ring = (uint32_t)std::min<uint64_t>(ring, (work + grid - 1) / grid);
    kern<<<(unsigned)grid, nthreads, smem, st>>>(keys, scr, P.inst, P.owner, P.tile, P.items, P.citem, P.tot, ctrl, wc,
                                                 flags, done, ring, (uint32_t)stage, work >= kClaimAheadItems * grid * ring);
    TL_CUDA_TRY(cudaGetLastError());
    return TL_SUCCESS;
}

int batch_permute(const tl_batch_plan *plan, void *dev_keys, void *dev_ws, uint64_t ws_bytes, cudaStream_t st) {
    if (!plan || !dev_keys || !dev_ws) return TL_ERROR_INVALID_VALUE;
    const auto &P = *reinterpret_cast<const tl_batch_plan_impl *>(plan);
    if (ws_bytes < P.ws_bytes) return TL_ERROR_WORKSPACE_TOO_SMALL;
    if (reinterpret_cast<uintptr_t>(dev_ws) % 256 || reinterpret_cast<uintptr_t>(dev_keys) % P.key_bytes)
        return TL_ERROR_INVALID_VALUE;
    char *ws = static_cast<char *>(dev_ws);
    return P.key_bytes == 8 ? launch_batch_permute<uint64_t>(P, static_cast<uint64_t *>(dev_keys), ws, st, P.threads)
                            : launch_batch_permute<uint32_t>(P, static_cast<uint32_t *>(dev_keys), ws, st, P.threads);
}

int batch_status(const tl_batch_plan *plan, const void *dev_ws, cudaStream_t st) {
    if (!plan || !dev_ws) return TL_ERROR_INVALID_VALUE;
    const auto &P = *reinterpret_cast<const tl_batch_plan_impl *>(plan);
    const Ctrl *ctrl = reinterpret_cast<const Ctrl *>(static_cast<const char *>(dev_ws) + P.off_ctrl);
    unsigned int err = 0;
    int rc = read_error_word(&ctrl->error, &err, st);
    if (rc) return rc;
    // a bounded wait expired, or (never expected) the ordered schedule found a
    // scratch store without scratch and skipped it
    if (!err) return TL_SUCCESS;
    return (err & (1u << TL_ERROR_TIMEOUT)) ? TL_ERROR_TIMEOUT : TL_ERROR_UNSUPPORTED;
}

// The queries need no memory of their own; callers still pass a workspace.
int batch_query_workspace_bytes(const tl_batch_plan *plan, uint64_t q, uint64_t *bytes) {
    (void)q;
    if (!plan || !bytes) return TL_ERROR_INVALID_VALUE;
    *bytes = 256;
    return TL_SUCCESS;
}

// Batches of kBatchSortMin queries or more go through the sorted form: a block
// an SM needs some thousands of queries a chunk to pay for its sort.  Measured
// on B200, 1024 arrays of 5.2e8 u64 keys, as given against sorted: b = 8 2^17
// queries 30 / 40 us, 2^18 49 / 57, 2^19 85 / 74, 2^20 158 / 83; b = 16 2^18 55 /
// 74, 2^19 100 / 95.
constexpr uint64_t kBatchSortMin = 1ull << 19;

template <typename K, int NB, int G1, int GS, typename I>
static int launch_batch_query_as(const tl_batch_plan_impl &P, const K *keys, const K *Q, const uint32_t *qinst,
                                 uint64_t q, uint64_t *ans, cudaStream_t st) {
    const uint64_t sms = (uint64_t)batch_sms();
    // measurement hooks: variant 30 always sorts, 31 never
    if (query_variant() == 31 || (query_variant() != 30 && q < kBatchSortMin)) {
        auto kern = batch_query_kernel<K, NB, G1, I>;
        int per_sm = 0;
        TL_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kBatchThreads, 0));
        const uint64_t grid = std::min<uint64_t>((q * G1 + kBatchThreads - 1) / kBatchThreads,
                                                 (uint64_t)std::max(per_sm, 1) * sms);
        kern<<<(unsigned)grid, kBatchThreads, 0, st>>>(keys, P.total_keys, P.geo, P.num, (uint32_t)P.b, Q, qinst, q,
                                                       ans);
    } else {
        // equal chunks, one block an SM: the fewest rounds of at most kBatchSortChunk queries
        const uint64_t rounds = (q + sms * kBatchSortChunk - 1) / (sms * kBatchSortChunk);
        const uint64_t chunk = (q + sms * rounds - 1) / (sms * rounds);
        uint32_t shift = 0;  // bins of 2^shift consecutive instances
        while (((P.num - 1) >> shift) >= kBatchBins) ++shift;
        const size_t smem = chunk * sizeof(uint16_t);
        auto kern = batch_query_sorted_kernel<K, NB, GS, I>;
        kern<<<(unsigned)std::min<uint64_t>((q + chunk - 1) / chunk, sms), kBatchSortThreads, smem, st>>>(
            keys, P.total_keys, P.geo, P.num, (uint32_t)P.b, shift, (uint32_t)chunk, Q, qinst, q, ans);
    }
    TL_CUDA_TRY(cudaGetLastError());
    return TL_SUCCESS;
}

template <typename K>
static int launch_batch_query(const tl_batch_plan_impl &P, const K *keys, const K *Q, const uint32_t *qinst,
                              uint64_t q, uint64_t *ans, cudaStream_t st) {
    // 32-bit node indices: a child index is below n + 2 + b * b
    if (P.max_n < (1ull << 31) && P.b <= 1024) {
        switch (P.b * sizeof(K)) {
            case 32: return launch_batch_query_as<K, 32, 2, 1, uint32_t>(P, keys, Q, qinst, q, ans, st);
            case 64: return launch_batch_query_as<K, 64, 4, 1, uint32_t>(P, keys, Q, qinst, q, ans, st);
            case 128: return launch_batch_query_as<K, 128, 4, 1, uint32_t>(P, keys, Q, qinst, q, ans, st);
            case 256: return launch_batch_query_as<K, 256, 4, 4, uint32_t>(P, keys, Q, qinst, q, ans, st);
            default: return launch_batch_query_as<K, 0, 4, 1, uint32_t>(P, keys, Q, qinst, q, ans, st);
        }
    }
    return launch_batch_query_as<K, 0, 4, 4, uint64_t>(P, keys, Q, qinst, q, ans, st);
}

int batch_query(const tl_batch_plan *plan, const void *dev_keys, const void *dev_queries, const uint32_t *dev_inst,
                uint64_t q, uint64_t *dev_answers, void *dev_ws, uint64_t ws_bytes, cudaStream_t st, float *ms) {
    if (!plan || (q && (!dev_keys || !dev_queries || !dev_inst || !dev_answers || !dev_ws)))
        return TL_ERROR_INVALID_VALUE;
    const auto &P = *reinterpret_cast<const tl_batch_plan_impl *>(plan);
    uint64_t need = 0;
    batch_query_workspace_bytes(plan, q, &need);
    if (ws_bytes < need) return TL_ERROR_WORKSPACE_TOO_SMALL;
    if (q == 0) return TL_SUCCESS;
    EventTimer timer(ms != nullptr, st);
    timer.start();
    int rc = P.key_bytes == 8
                 ? launch_batch_query<uint64_t>(P, static_cast<const uint64_t *>(dev_keys),
                                                static_cast<const uint64_t *>(dev_queries), dev_inst, q, dev_answers, st)
                 : launch_batch_query<uint32_t>(P, static_cast<const uint32_t *>(dev_keys),
                                                static_cast<const uint32_t *>(dev_queries), dev_inst, q, dev_answers, st);
    timer.stop();
    if (rc) return rc;
    if (ms) {
        rc = sync_and_check(st);
        if (rc) return rc;
        *ms = timer.elapsed();
    }
    return TL_SUCCESS;
}

int batch_set_tuning(tl_batch_plan *plan, const uint32_t *tile_keys, const uint32_t *pin_levels, uint32_t query_chunk,
                     uint32_t threads, const int64_t *dev_offsets, cudaStream_t st) {
    if (!plan) return TL_ERROR_INVALID_VALUE;
    auto &P = *reinterpret_cast<tl_batch_plan_impl *>(plan);
    if (tile_keys) {
        for (int c = 0; c < kMaxClass; ++c) {
            const uint32_t t = tile_keys[c];
            if (t < 256 || t * P.key_bytes > 96 * 1024 || (t & (t - 1))) return TL_ERROR_INVALID_VALUE;
        }
        memcpy(P.tile_keys, tile_keys, sizeof(P.tile_keys));
        if (!dev_offsets) return TL_ERROR_INVALID_VALUE;
        int rc = build_plan(P, dev_offsets, st);
        if (rc) return rc;
    }
    if (pin_levels) memcpy(P.pin_levels, pin_levels, sizeof(P.pin_levels));
    if (query_chunk) P.query_chunk = query_chunk;
    if (threads) {
        if (threads != 256 && threads != 512) return TL_ERROR_INVALID_VALUE;
        P.threads = threads;
    }
    return TL_SUCCESS;
}

int batch_get_tuning(const tl_batch_plan *plan, uint32_t *tile_keys, uint32_t *pin_levels, uint32_t *query_chunk,
                     uint32_t *threads) {
    if (!plan) return TL_ERROR_INVALID_VALUE;
    const auto &P = *reinterpret_cast<const tl_batch_plan_impl *>(plan);
    if (tile_keys) memcpy(tile_keys, P.tile_keys, sizeof(P.tile_keys));
    if (pin_levels) memcpy(pin_levels, P.pin_levels, sizeof(P.pin_levels));
    if (query_chunk) *query_chunk = P.query_chunk;
    if (threads) *threads = P.threads;
    return TL_SUCCESS;
}

// Size classes present in the batch (floor(log2 n_j)) and the keys in each,
// read back from the plan (host).
static int batch_class_keys(const tl_batch_plan_impl &P, std::vector<uint64_t> &keys_per_class) {
    std::vector<BatchInst> h(P.num);
    TL_CUDA_TRY(cudaMemcpy(h.data(), P.inst, (size_t)P.num * sizeof(BatchInst), cudaMemcpyDeviceToHost));
    keys_per_class.assign(kMaxClass, 0);
    for (const auto &I : h) {
        const uint64_t n = I.S.g.n;
        const uint32_t c = n ? bit_length(n) - 1 : 0;
        keys_per_class[c < kMaxClass ? c : kMaxClass - 1] += n;
    }
    return TL_SUCCESS;
}

// Coordinate-descent autotuner of the permutation: the block size, then per size
// class (largest classes first) the tile size, each candidate timed on the whole
// batch (the sorted input restored from a copy before every trial).  The queries
// have nothing to tune; a batch of them is timed for the report.  The plan keeps
// the best values; the keys are left sorted.
int batch_autotune(tl_batch_plan *plan, const int64_t *dev_offsets, void *dev_keys, const void *dev_queries,
                   const uint32_t *dev_inst, uint64_t q, cudaStream_t st, char *report, size_t report_len) {
    if (!plan || !dev_offsets || !dev_keys) return TL_ERROR_INVALID_VALUE;
    auto &P = *reinterpret_cast<tl_batch_plan_impl *>(plan);
    const size_t kbytes = (size_t)P.total_keys * P.key_bytes;
    char *pristine = nullptr, *ws = nullptr;
    int rc = TL_SUCCESS;
    std::vector<uint64_t> cls_keys;
    rc = batch_class_keys(P, cls_keys);
    if (rc) return rc;
    if (cudaMalloc(reinterpret_cast<void **>(&pristine), kbytes) != cudaSuccess) return TL_ERROR_OUT_OF_MEMORY;
    TL_CUDA_TRY(cudaMemcpyAsync(pristine, dev_keys, kbytes, cudaMemcpyDeviceToDevice, st));
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    uint64_t ws_cap = 0;
    auto ensure_ws = [&](uint64_t need) -> int {
        if (need <= ws_cap) return TL_SUCCESS;
        if (ws) cudaFree(ws);
        ws = nullptr;
        ws_cap = 0;
        if (cudaMalloc(reinterpret_cast<void **>(&ws), need) != cudaSuccess) return TL_ERROR_OUT_OF_MEMORY;
        ws_cap = need;
        return TL_SUCCESS;
    };
    auto time_permute = [&](float &best) -> int {
        float total = 0.f;
        for (int rep = 0; rep < 3; ++rep) {
            TL_CUDA_TRY(cudaMemcpyAsync(dev_keys, pristine, kbytes, cudaMemcpyDeviceToDevice, st));
            int r = ensure_ws(P.ws_bytes);
            if (r) return r;
            cudaEventRecord(e0, st);
            r = batch_permute(plan, dev_keys, ws, ws_cap, st);
            if (r) return r;
            cudaEventRecord(e1, st);
            TL_CUDA_TRY(cudaEventSynchronize(e1));
            float ms = 0.f;
            cudaEventElapsedTime(&ms, e0, e1);
            if (rep) total += ms;  // first repetition warms up
        }
        best = total / 2;
        return TL_SUCCESS;
    };
    const uint32_t tiles[3] = {(uint32_t)(16384 / P.key_bytes), (uint32_t)(32768 / P.key_bytes),
                               (uint32_t)(65536 / P.key_bytes)};
    float cur = 0.f;
    rc = time_permute(cur);
    // block size
    for (uint32_t th : {512u, 256u}) {
        if (rc) break;
        const uint32_t keep = P.threads;
        P.threads = th;
        float ms = 0.f;
        rc = time_permute(ms);
        if (!rc && ms < cur) cur = ms; else P.threads = keep;
    }
    // tile size per class, largest classes first
    std::vector<int> order;
    for (int c = 0; c < kMaxClass; ++c)
        if (cls_keys[c]) order.push_back(c);
    std::sort(order.begin(), order.end(), [&](int a, int b2) { return cls_keys[a] > cls_keys[b2]; });
    for (int c : order) {
        if (rc) break;
        const uint32_t keep = P.tile_keys[c];
        uint32_t best_t = keep;
        for (uint32_t t : tiles) {
            if (t == keep) continue;
            P.tile_keys[c] = t;
            rc = build_plan(P, dev_offsets, st);
            if (rc) break;
            float ms = 0.f;
            rc = time_permute(ms);
            if (rc) break;
            if (ms < cur) {
                cur = ms;
                best_t = t;
            }
        }
        P.tile_keys[c] = best_t;
        if (!rc) rc = build_plan(P, dev_offsets, st);
    }
    float qcur = -1.f;
    if (!rc && q && dev_queries && dev_inst) {
        // a permuted copy for the query trials
        TL_CUDA_TRY(cudaMemcpyAsync(dev_keys, pristine, kbytes, cudaMemcpyDeviceToDevice, st));
        rc = ensure_ws(P.ws_bytes);
        if (!rc) rc = batch_permute(plan, dev_keys, ws, ws_cap, st);
        uint64_t qneed = 0;
        batch_query_workspace_bytes(plan, q, &qneed);
        char *qws = nullptr;
        uint64_t *ans = nullptr;
        if (!rc && (cudaMalloc(reinterpret_cast<void **>(&qws), qneed) != cudaSuccess ||
                    cudaMalloc(reinterpret_cast<void **>(&ans), q * 8) != cudaSuccess))
            rc = TL_ERROR_OUT_OF_MEMORY;
        auto time_query = [&](float &out) -> int {
            float total = 0.f;
            for (int rep = 0; rep < 3; ++rep) {
                float ms = 0.f;
                int r = batch_query(plan, dev_keys, dev_queries, dev_inst, q, ans, qws, qneed, st, &ms);
                if (r) return r;
                if (rep) total += ms;
            }
            out = total / 2;
            return TL_SUCCESS;
        };
        if (!rc) rc = time_query(qcur);
        if (qws) cudaFree(qws);
        if (ans) cudaFree(ans);
    }
    cudaMemcpyAsync(dev_keys, pristine, kbytes, cudaMemcpyDeviceToDevice, st);
    cudaStreamSynchronize(st);
    cudaFree(pristine);
    if (ws) cudaFree(ws);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (report && report_len) {
        std::string r = "{\"threads\":" + std::to_string(P.threads) + ",\"query_chunk\":" +
                        std::to_string(P.query_chunk) + ",\"permute_ms\":" + std::to_string(cur) +
                        ",\"query_ms\":" + std::to_string(qcur) + ",\"classes\":{";
        bool first = true;
        for (int c : order) {
            r += (first ? "" : ",") + std::string("\"") + std::to_string(c) + "\":{\"keys\":" +
                 std::to_string(cls_keys[c]) + ",\"tile_keys\":" + std::to_string(P.tile_keys[c]) +
                 ",\"pin_levels\":" + std::to_string(P.pin_levels[c]) + "}";
            first = false;
        }
        r += "}}";
        snprintf(report, report_len, "%s", r.c_str());
    }
    return rc;
}

}  // namespace tl
