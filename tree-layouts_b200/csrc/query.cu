// Batched exact point queries over the three layouts (sm_100a).
//
// Each kernel is persistent (grid = SMs x resident CTAs) and copies the top
// levels, the layout's first positions, once per CTA into shared memory, so the
// first levels of every descent cost a shared-memory load instead of an L2/HBM
// round trip.  The B-tree kernels walk the query array with a grid stride; the
// BST, vEB and sorted-array kernels take it in chunks that a block orders by
// value in shared memory first, so that neighbours share their lower nodes.
//
// Answers are the layout position of the key or n (gpu/src/query-bst.cuh:41,
// gpu/src/query-btree.cuh:59, gpu/src/query-mveb.cuh:65); of equal keys it is the
// one that the reference's search from the root meets first.
#include <algorithm>
#include <vector>

#include "internal.h"
#include "tl_common.cuh"

namespace tl {

constexpr int kQueryThreads = 256;
constexpr uint32_t kPinBytes = 48 * 1024;
// The search of a grouped batch over a large BST pins 16 KB of top levels,
// leaving room for 8 blocks an SM: measured on B200, 2^27 grouped queries, 2^30 -
// 1 u64 keys 13.25 -> 12.14 ms against 32 KB, 2^27 - 1 u32 10.23 -> 9.79 ms (8
// KB: the same)
constexpr uint32_t kBstGroupPinBytes = 16 * 1024;

template <typename K>
__device__ __forceinline__ void pin_prefix(const K *__restrict__ A, uint64_t P, K *sm) {
    for (uint64_t x = threadIdx.x; x < P; x += blockDim.x) sm[x] = __ldg(A + x);
    __syncthreads();
}

template <typename K>
__device__ __forceinline__ K key_at(const K *__restrict__ A, const K *sm, uint64_t P, uint64_t i) {
    return i < P ? sm[i] : __ldg(A + i);
}

// ---------------------------------------------------------------- BST
// searchBST (gpu/src/query-bst.cuh:31-42): i = 2i + 1 + (q > A[i]).  The batch
// grouped by value (partition_queries), answers through the carried index.
template <typename K>
__global__ void __launch_bounds__(kQueryThreads)
bst_query_kernel(const K *__restrict__ A, uint64_t n, uint64_t P, const K *__restrict__ Q, uint64_t nq,
                 const uint32_t *__restrict__ perm, uint64_t *__restrict__ ans) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    K *sm = reinterpret_cast<K *>(smem_raw);
    pin_prefix(A, P, sm);
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t qi = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; qi < nq; qi += stride) {
        const K q = __ldcs(Q + qi);
        uint64_t i = 0, res = n;
        while (i < n) {
            const K cur = key_at(A, sm, P, i);
            if (q == cur) {
                res = i;
                break;
            }
            i = 2 * i + 1 + (q > cur);
        }
        const uint64_t out = __ldg(perm + qi);
        if (out < nq) __stcs(ans + out, res);
    }
}

// ---------------------------------------------------------------- sorted array
// The binary-search comparator (gpu/src/binary-search.cuh:27-57 searches the
// sorted array before any permutation).  Branch-free lower bound: with
// len_0 = n and base_0 = 0, step d probes base_d + half_d (half_d = len_d / 2),
// base_{d+1} = base_d + half_d when that key is below the query, len_{d+1} =
// len_d - half_d; then the answer is the lower bound if it holds the query,
// else n.  The lengths do not depend on the query, so the keys probed in the
// first L steps form a complete binary tree of 2^L - 1 positions; they are
// pinned in shared memory in breadth-first order (node i has children 2i and
// 2i + 1, path bit = "went right"), which turns those steps into
// shared-memory loads.
template <typename K>
__global__ void __launch_bounds__(kQueryThreads)
sorted_query_kernel(const K *__restrict__ A, uint64_t n, uint32_t L, const K *__restrict__ Q, uint64_t nq,
                    uint64_t *__restrict__ ans) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    K *tree = reinterpret_cast<K *>(smem_raw);  // tree[1 .. 2^L - 1]
    const uint32_t nodes = (1u << L) - 1;
    for (uint32_t node = threadIdx.x + 1; node <= nodes; node += blockDim.x) {
        // replay the path of `node`: its bits below the leading one, high to low
        const uint32_t depth = 31 - __clz(node);
        uint64_t base = 0, len = n;
        for (uint32_t d = 0; d < depth; ++d) {
            const uint64_t half = len >> 1;
            if ((node >> (depth - 1 - d)) & 1u) base += half;
            len -= half;
        }
        tree[node] = __ldg(A + base + (len >> 1));
    }
    __syncthreads();
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t qi = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; qi < nq; qi += stride) {
        const K q = __ldcs(Q + qi);
        uint64_t base = 0, len = n;
        uint32_t node = 1;
        for (uint32_t d = 0; d < L; ++d) {  // len > 1 throughout: L < log2(n)
            const uint64_t half = len >> 1;
            const bool right = tree[node] < q;
            base += right ? half : 0;
            len -= half;
            node = 2 * node + right;
        }
        while (len > 1) {
            const uint64_t half = len >> 1;
            base += __ldg(A + base + half) < q ? half : 0;
            len -= half;
        }
        const K at = __ldg(A + base);
        const uint64_t lb = base + (at < q);
        __stcs(ans + qi, (lb < n && (lb == base ? at : __ldg(A + lb)) == q) ? lb : n);
    }
}

// ---------------------------------------------------------------- B-tree
// searchBtree (cpu/src/query-btree.h:33-54): the child followed is the number of
// node keys smaller than the query; an equal key ends the search.  A group of G
// lanes reads one node cooperatively: lane j of the group owns node slots
// j, j+G, ...; slots at or past n (the partial last leaf) count as +infinity.
template <typename K, int G>
__global__ void __launch_bounds__(kQueryThreads)
btree_query_kernel(const K *__restrict__ A, uint64_t n, uint64_t b, uint64_t P, const K *__restrict__ Q,
                   uint64_t nq, uint64_t *__restrict__ ans) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    K *sm = reinterpret_cast<K *>(smem_raw);
    pin_prefix(A, P, sm);
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t gl = lane % G;                      // lane within the group
    const uint32_t gbase = lane - gl;                  // first lane of the group
    const unsigned gmask = (G == 32 ? 0xFFFFFFFFu : ((1u << G) - 1)) << gbase;
    const uint64_t groups = (uint64_t)gridDim.x * blockDim.x / G;
    const uint64_t gid = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) / G;
    const uint64_t rounds = (nq + groups - 1) / groups;  // uniform trip count keeps warps converged
    for (uint64_t rd = 0; rd < rounds; ++rd) {
        const uint64_t qi = rd * groups + gid;
        const bool active = qi < nq;
        const K q = active ? Q[qi] : K(0);
        uint64_t i = 0, res = n;
        bool done = !active;
        while (__any_sync(0xFFFFFFFFu, !done)) {
            if (!done && i >= n) done = true;
            uint32_t lt = 0;
            int eq_slot = -1;
            if (!done) {
                for (uint64_t s = gl; s < b; s += G) {
                    const uint64_t p = i + s;
                    if (p < n) {
                        const K cur = key_at(A, sm, P, p);
                        lt += cur < q;
                        if (cur == q && eq_slot < 0) eq_slot = (int)s;
                    }
                }
            }
            // group reductions (all 32 lanes take part; inactive lanes add zero)
            for (int off = G / 2; off > 0; off >>= 1) {
                lt += __shfl_xor_sync(0xFFFFFFFFu, lt, off);
                const int o = __shfl_xor_sync(0xFFFFFFFFu, eq_slot, off);
                if (o >= 0 && (eq_slot < 0 || o < eq_slot)) eq_slot = o;
            }
            (void)gmask;
            if (!done) {
                // The reference returns the first equal key of the node whose
                // preceding keys are all smaller; with sorted nodes that is the
                // equal key at slot lt.
                if (eq_slot >= 0 && (uint64_t)eq_slot == lt) {
                    res = i + (uint64_t)eq_slot;
                    done = true;
                } else if (i + 1 > (n + 1) / (b + 1)) {
                    done = true;  // every child starts past n; also keeps (i+1)(b+1) from overflowing
                } else {
                    i = (i + 1) * (b + 1) + lt * b - 1;
                }
            }
        }
        if (active && gl == 0) ans[qi] = res;
    }
}

// One thread per query, for nodes of b*w = 16*NV bytes (node starts are then
// 16-byte aligned): the node is fetched with NV independent 16-byte loads.
template <typename K, int NV>
__global__ void __launch_bounds__(kQueryThreads)
btree_query_vec_kernel(const K *__restrict__ A, uint64_t n, uint64_t b, const K *__restrict__ Q, uint64_t nq,
                       uint64_t *__restrict__ ans) {
    constexpr int KPV = 16 / sizeof(K);  // keys per 16-byte vector
    constexpr int B = NV * KPV;          // == b
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t cmax = (n + 1) / (B + 1);
    for (uint64_t qi = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; qi < nq; qi += stride) {
        const K q = __ldcs(Q + qi);
        uint64_t i = 0, res = n;
        while (i < n) {
            uint32_t lt = 0;
            bool eq = false;
            if (i + B <= n) {
                const uint4 *node = reinterpret_cast<const uint4 *>(A + i);
                uint4 v[NV];
#pragma unroll
                for (int j = 0; j < NV; ++j) v[j] = __ldg(node + j);
#pragma unroll
                for (int j = 0; j < NV; ++j) {
                    const K *kk = reinterpret_cast<const K *>(&v[j]);
#pragma unroll
                    for (int e = 0; e < KPV; ++e) lt += kk[e] < q;
                }
                if (lt < (uint32_t)B) {
                    const K *all = reinterpret_cast<const K *>(v);
                    K at = all[0];
#pragma unroll
                    for (int j = 1; j < B; ++j)
                        if ((uint32_t)j == lt) at = all[j];
                    eq = at == q;
                }
            } else {
                const uint64_t valid = n - i;
                for (uint64_t j = 0; j < valid; ++j) lt += __ldg(A + i + j) < q;
                if (lt < valid) eq = __ldg(A + i + lt) == q;
            }
            if (eq) {
                res = i + lt;
                break;
            }
            if (i + 1 > cmax) break;
            i = (i + 1) * (B + 1) + (uint64_t)lt * B - 1;
        }
        __stcs(ans + qi, res);
    }
}

// One thread per query for nodes of NB = b * w bytes, NB a multiple of 32 on a
// 32-byte aligned layout: a node is NB / 32 independent 32-byte loads (one L1
// wavefront each when the warp's nodes are distinct lines, half the 16-byte
// loads' count).  The first P keys (whole top levels) may be pinned in shared
// memory.  The partial last leaf is read with guarded scalar loads.
template <typename K, int NB, bool kPin>
__global__ void __launch_bounds__(kQueryThreads)
btree_query_v32_kernel(const K *__restrict__ A, uint64_t n, uint64_t P, const K *__restrict__ Q, uint64_t nq,
                       uint64_t *__restrict__ ans) {
    constexpr int KPL = 32 / sizeof(K);  // keys per 32-byte load
    constexpr int NL = NB / 32;          // loads per node
    constexpr int B = NB / sizeof(K);    // == b
    extern __shared__ __align__(16) unsigned char smem_raw[];
    K *sm = reinterpret_cast<K *>(smem_raw);
    if constexpr (kPin) pin_prefix(A, P, sm);
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t cmax = (n + 1) / (B + 1);
    for (uint64_t qi = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; qi < nq; qi += stride) {
        const K q = __ldcs(Q + qi);
        uint64_t i = 0, res = n;
        while (i < n) {
            uint32_t lt = 0;
            bool eq = false;
            if (i + B <= n) {
                K v[NL][KPL];
                if (kPin && i < P) {
#pragma unroll
                    for (int j = 0; j < NL; ++j) {
                        const uint4 *s4 = reinterpret_cast<const uint4 *>(sm + i + j * KPL);
                        const uint4 a = s4[0], c = s4[1];
                        const K *ka = reinterpret_cast<const K *>(&a);
                        const K *kc = reinterpret_cast<const K *>(&c);
#pragma unroll
                        for (int e = 0; e < KPL / 2; ++e) {
                            v[j][e] = ka[e];
                            v[j][KPL / 2 + e] = kc[e];
                        }
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < NL; ++j) ldg32(A + i + j * KPL, v[j]);
                }
#pragma unroll
                for (int j = 0; j < NL; ++j)
#pragma unroll
                    for (int e = 0; e < KPL; ++e) lt += v[j][e] < q;
#pragma unroll
                for (int j = 0; j < NL; ++j)
#pragma unroll
                    for (int e = 0; e < KPL; ++e) eq |= v[j][e] == q;
            } else {
                const uint64_t valid = n - i;
                for (uint64_t j = 0; j < valid; ++j) {
                    const K cur = __ldg(A + i + j);
                    lt += cur < q;
                    eq |= cur == q;
                }
            }
            if (eq) {
                res = i + lt;
                break;
            }
            if (i + 1 > cmax) break;
            i = (i + 1) * (B + 1) + (uint64_t)lt * B - 1;
        }
        __stcs(ans + qi, res);
    }
}

// G lanes per query read a node together with NL = NB / (32 G) 32-byte loads
// each (lane g holds slots g * KPL + j * G * KPL + [0, KPL) for load j).  Each
// load instruction of a warp then touches 32 / G node lines with G sectors of
// a line in one L1 wavefront, where a thread per query spends a wavefront per
// sector; fewer lanes per node keep more descents in flight.  Control flow is
// warp-uniform (a warp takes 32 / G queries per round and descends while any of
// them is live), so the group's count is a full-warp shuffle sum and an equal
// key in any of its lanes, found by ballot, ends its descent.  (Descending to
// the last level on counts alone and checking q's successor with one load at
// the end measured 9 % slower on B200: that load adds a dependent step to every
// warp's round.)
template <typename K, int NB, int G>
__global__ void __launch_bounds__(kQueryThreads)
btree_query_group32_kernel(const K *__restrict__ A, uint64_t n, const K *__restrict__ Q, uint64_t nq,
                           uint64_t *__restrict__ ans) {
    constexpr int KPL = 32 / sizeof(K);  // keys per 32-byte load
    constexpr int NL = NB / 32 / G;      // 32-byte loads per lane and node
    constexpr int B = NB / sizeof(K);    // == b
    constexpr int QPW = 32 / G;          // queries per warp and round
    static_assert(G >= 2 && G <= 8 && (G & (G - 1)) == 0 && NL >= 1 && NL * G * 32 == NB,
                  "group of 2, 4 or 8 lanes");
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t g = lane % G;
    const uint32_t gshift = lane - g;
    const uint64_t warps = (uint64_t)gridDim.x * (blockDim.x / 32);
    const uint64_t wid = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) / 32;
    const uint64_t cmax = (n + 1) / (B + 1);
    for (uint64_t base = wid * QPW; base < nq; base += warps * QPW) {
        const uint64_t qi = base + lane / G;
        bool live = qi < nq && n > 0;
        const K q = qi < nq ? __ldcs(Q + qi) : K(0);
        uint64_t i = 0, res = n;
        while (__any_sync(0xFFFFFFFFu, live)) {
            uint32_t lt = 0;
            bool eq = false;
            if (live) {
                const uint64_t s0 = i + (uint64_t)g * KPL;  // lane g: slots s0 + j * G * KPL + e
                if (i + B <= n) {
                    K v[NL][KPL];
#pragma unroll
                    for (int j = 0; j < NL; ++j) ldg32(A + s0 + (uint64_t)j * G * KPL, v[j]);
#pragma unroll
                    for (int j = 0; j < NL; ++j)
#pragma unroll
                        for (int e = 0; e < KPL; ++e) {
                            lt += v[j][e] < q;
                            eq |= v[j][e] == q;
                        }
                } else {  // the partial last leaf: slots at or past n do not count
#pragma unroll
                    for (int j = 0; j < NL; ++j)
#pragma unroll
                        for (int e = 0; e < KPL; ++e) {
                            const uint64_t p = s0 + (uint64_t)j * G * KPL + e;
                            if (p < n) {
                                const K cur = __ldg(A + p);
                                lt += cur < q;
                                eq |= cur == q;
                            }
                        }
                }
            }
#pragma unroll
            for (int off = G / 2; off > 0; off >>= 1) lt += __shfl_xor_sync(0xFFFFFFFFu, lt, off);
            const bool hit = ((__ballot_sync(0xFFFFFFFFu, eq) >> gshift) & ((1u << G) - 1)) != 0;
            if (live) {
                if (hit) {
                    res = i + lt;
                    live = false;
                } else if (i + 1 > cmax) {
                    live = false;
                } else {
                    i = (i + 1) * (B + 1) + (uint64_t)lt * B - 1;
                    live = i < n;
                }
            }
        }
        if (g == 0 && qi < nq) __stcs(ans + qi, res);
    }
}

// The same read of a node by G lanes, below a top of T whole levels searched in
// shared memory: their m = (b + 1)^T - 1 keys in sorted order, and kTopBins bins
// of equal width over their value range holding the first rank of each, so a
// query finds its rank among them with a bin and a binary search inside it (one
// or two probes where keys are spread evenly, log2(m) at worst) and starts at
// the node of level T with that number.
// What bounds it: each level read from global memory costs a query NL L1
// wavefronts (two for 128-byte nodes; ncu, 2^24 queries over 1e8 u64 keys, b =
// 16: L1 data pipe 92 % before and after), a probe of shared memory about a
// fifth of one, and three of the seven levels there fit 40 KB.  Measured on
// B200, without and with the top: b = 16 u64, 2^24 queries over 1e8 keys 1068 ->
// 704 us, over 2^20 keys 751 -> 408, 2^27 over 5e8 9.43 -> 7.5 to 8.4 ms (there
// the three levels in DRAM, 400 bytes a query, are 8.2 ms of the copy
// bandwidth); b = 32 u64 over 2^28 keys 1866 -> 1262; b = 8 u64 1024 -> 921; b =
// 16 u32 over 5e8 keys 899 -> 740.  Ordering the batch by value in chunks first
// gains nothing here (a level's wavefronts stay, 704 -> 820 us), nor does a
// thread a query whose nodes four lanes read together (half the wavefronts, 48
// warps' registers: 1028).  Two blocks of 1024 threads an SM at 32 registers;
// the wide form of I would not fit, so layouts of 2^31 keys or more keep the
// kernel above.
constexpr uint32_t kTopBins = 4096;
constexpr int kTopThreads = 1024;
constexpr uint64_t kTopBytes = 40 * 1024;
// 128-byte nodes keep the kernel above over larger layouts, whose deep levels are
// no longer bound by wavefronts (the cause beyond that was not isolated): b = 16
// u64, kernel above against this, 2^27 queries over 2^29 keys 9.48 / 8.51 ms, over
// 8e8 9.68 / 9.83, over 2^30 9.92 / 10.62; 2^26 over 6.4e8 4.78 / 4.53.  Other
// nodes gain at every size (64-byte over 7.6 GB 4.26 / 3.94, 256-byte over 7.2 GB
// 7.39 / 5.57).  Skewed batches would gain there too (2^28 Zipf queries over 2^30
// keys 20.0 / 14.8 ms), but a batch's skew is not known at the launch.
constexpr uint64_t kTopMaxBytes128 = 5ull << 30;

// Keys of the whole levels that kTopBytes hold (0: not one).
template <typename K>
constexpr uint64_t btree_top_keys(uint64_t n, uint64_t b) {
    uint64_t m = 0;
    for (uint64_t t = b; t <= n && t <= kTopBytes / sizeof(K); t = t * (b + 1) + b) m = t;
    return m;
}

// The top's index arithmetic, shared with its host replay (emulate_btree_top).
// Keys that are not in layout order give no meaningful answer, but every index
// stays in range for them too: bin numbers are clamped and no bin is left unset.

// Sorted rank of the top's position p: the x-th multiple of mult (x not a
// multiple of B + 1) on its level.
template <uint32_t B>
TL_HD uint32_t top_rank_of(uint32_t p, uint32_t m) {
    uint32_t end = B + 1, mult = (m + 1) / (B + 1);  // the level's end + 1, its keys' spacing
    while (p + 1 >= end) {
        end *= B + 1;
        mult /= B + 1;
    }
    const uint32_t t = p + 1 - end / (B + 1);
    return (t + 1 + t / B) * mult - 1;
}

// The position of sorted rank r.
template <uint32_t B>
TL_HD uint32_t top_position(uint32_t r, uint32_t m) {
    uint32_t x = r + 1, end = m + 1;
    while (x % (B + 1) == 0) {
        x /= B + 1;
        end /= B + 1;
    }
    return end / (B + 1) - 1 + (x - x / (B + 1) - 1);
}

// Equal keys: of those at sorted rank r and after, the one that the search from
// the root meets first.  Its path holds, a level up, the next multiple of that
// level's spacing, and its keys do not fall on the way up.
template <uint32_t B, typename Top>
TL_HD uint32_t top_first_on_path(Top top, uint32_t m, uint32_t r) {
    const auto q = top[r];
    uint32_t x = r + 1;
    for (uint32_t s = B + 1; s <= m; s *= B + 1) {
        const uint32_t up = (x + s - 1) / s * s;
        if (up > m || top[up - 1] != q) break;
        x = up;
    }
    return x - 1;
}

template <typename K>
TL_HD uint32_t top_shift(K first, K last) {
    const uint32_t span = bit_length((uint64_t)(K)(last - first)), bits = bit_length(kTopBins - 1);
    return span > bits ? span - bits : 0;
}

// The bin of a key, kTopBins for all past the last.
template <typename K>
TL_HD uint32_t top_bin(K key, K first, uint32_t shift) {
    const K k = (K)(key - first) >> shift;
    return k < (K)kTopBins ? (uint32_t)k : kTopBins;
}

// Rank r in the bins it is the first rank of: those past the bin of rank r - 1, up to its own.
template <typename Top, typename K, typename Bin>
TL_HD void top_fill(Top top, uint32_t m, K first, uint32_t shift, uint32_t r, Bin bin) {
    const uint32_t hi = r < m ? top_bin((K)top[r], first, shift) : kTopBins;
    for (uint32_t k = r ? top_bin((K)top[r - 1], first, shift) + 1 : 0; k <= hi; ++k) bin[k] = (uint16_t)r;
}

// The number of top keys below q.
template <typename Top, typename K, typename Bin>
TL_HD uint32_t top_rank(Top top, Bin bin, uint32_t m, K first, uint32_t shift, K q) {
    if (q < first) return 0;
    const uint32_t k = top_bin(q, first, shift);
    if (k == kTopBins) return m;
    uint32_t r = bin[k], r1 = bin[k + 1];
    while (r < r1) {
        const uint32_t mid = (r + r1) >> 1;
        if ((K)top[mid] < q)
            r = mid + 1;
        else
            r1 = mid;
    }
    return r;
}

template <typename K, int NB, int G>
__global__ void __launch_bounds__(kTopThreads, 2)
btree_query_top_kernel(const K *__restrict__ A, uint32_t n, uint32_t m, const K *__restrict__ Q, uint64_t nq,
                       uint64_t *__restrict__ ans) {
    constexpr uint32_t KPL = 32 / sizeof(K);  // keys per 32-byte load
    constexpr int NL = NB / 32 / G;           // 32-byte loads per lane and node
    constexpr uint32_t B = NB / sizeof(K);    // == b
    extern __shared__ __align__(16) unsigned char smem_raw[];
    K *top = reinterpret_cast<K *>(smem_raw);               // [m]
    uint16_t *bin = reinterpret_cast<uint16_t *>(top + m);  // [kTopBins + 1]
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t g = lane % G;
    const uint32_t gshift = lane - g;
    const uint32_t cmax = (uint32_t)(((uint64_t)n + 1) / (B + 1));
    for (uint32_t p = threadIdx.x; p < m; p += kTopThreads) top[top_rank_of<B>(p, m)] = __ldg(A + p);
    for (uint32_t k = threadIdx.x; k <= kTopBins; k += kTopThreads) bin[k] = 0;
    __syncthreads();
    const K first = top[0];
    const uint32_t shift = top_shift(first, top[m - 1]);
    for (uint32_t r = threadIdx.x; r <= m; r += kTopThreads) top_fill(top, m, first, shift, r, bin);
    __syncthreads();
    const uint64_t warps = (uint64_t)gridDim.x * (kTopThreads / 32);
    const uint64_t wid = ((uint64_t)blockIdx.x * kTopThreads + threadIdx.x) / 32;
    for (uint64_t base = wid * (32 / G); base < nq; base += warps * (32 / G)) {
        const uint64_t qi = base + lane / G;
        const bool have = qi < nq;
        const K q = have ? __ldcs(Q + qi) : K(0);
        const uint32_t r = top_rank(top, bin, m, first, shift, q);  // top keys below q
        uint32_t i = m + r * B, res = n;
        bool live = have && i < n;
        if (r < m && top[r] == q) {  // a key of the top: its position there
            res = top_position<B>(top_first_on_path<B>(top, m, r), m);
            live = false;
        }
        while (__any_sync(0xFFFFFFFFu, live)) {
            uint32_t lt = 0;
            bool eq = false;
            if (live) {
                const uint32_t s0 = i + g * KPL;  // lane g: slots s0 + j * G * KPL + e
                if (n - i >= B) {
                    K v[NL][KPL];
#pragma unroll
                    for (int j = 0; j < NL; ++j) ldg32(A + s0 + j * G * KPL, v[j]);
#pragma unroll
                    for (int j = 0; j < NL; ++j)
#pragma unroll
                        for (uint32_t e = 0; e < KPL; ++e) {
                            lt += v[j][e] < q;
                            eq |= v[j][e] == q;
                        }
                } else {  // the partial last leaf: slots at or past n do not count
#pragma unroll
                    for (int j = 0; j < NL; ++j)
#pragma unroll
                        for (uint32_t e = 0; e < KPL; ++e) {
                            const uint32_t p = s0 + j * G * KPL + e;
                            if (p < n) {
                                const K cur = __ldg(A + p);
                                lt += cur < q;
                                eq |= cur == q;
                            }
                        }
                }
            }
#pragma unroll
            for (int off = G / 2; off > 0; off >>= 1) lt += __shfl_xor_sync(0xFFFFFFFFu, lt, off);
            const bool hit = ((__ballot_sync(0xFFFFFFFFu, eq) >> gshift) & ((1u << G) - 1)) != 0;
            if (live) {
                if (hit) {
                    res = i + lt;
                    live = false;
                } else if (i + 1 > cmax) {
                    live = false;
                } else {
                    i = (i + 1) * (B + 1) + lt * B - 1;
                    live = i < n;
                }
            }
        }
        if (g == 0 && have) __stcs(ans + qi, (uint64_t)res);
    }
}

static int g_query_variant = 0;
void set_query_variant(int v) { g_query_variant = v; }
int query_variant() { return g_query_variant; }

// ---------------------------------------------------------------- chunk order
// A block takes a chunk of the batch at a time and searches it in value order:
// a counting sort of 16-bit offsets in shared memory, into kSortBins bins of
// equal width over the chunk's value range (the order inside a bin does not
// matter, and a skewed batch only loses locality).  All blocks then sweep the
// layout from low to high values at about the same time, so a page, a line of an
// upper subtree and a DRAM row serve many descents while they are hot, and the
// answers go to the chunk's own stretch of the output.
constexpr int kSortThreads = 1024;  // one block an SM
constexpr uint32_t kSortBins = 1024;
constexpr uint32_t kSortChunk = 16384;
static_assert(kSortBins == kSortThreads, "one bin a thread in the scan");
static_assert(kSortChunk <= 65536, "16-bit offsets into the chunk");

struct ChunkSort {
    unsigned long long lo, hi;
    uint32_t cnt[kSortBins], wsum[32];
};

// order[0, len): the chunk's offsets by value.  With kPer > 0 the chunk is read
// once, kPer keys a thread (kPer * kSortThreads >= len), and stays in registers;
// with 0 it is read at each of the three steps (16 keys a thread would spill:
// the vEB search over 3e8 u64 keys 7.1 -> 7.6 ms).
template <int kPer, typename K>
__device__ __forceinline__ void chunk_order(const K *__restrict__ Q, uint32_t len, uint16_t *order, ChunkSort &cs) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    K v[kPer ? kPer : 1];
    K lo = ~K(0), hi = 0;
    // f(x, key) for this thread's entries of the chunk
    auto each = [&](auto f) {
        if constexpr (kPer > 0) {
#pragma unroll
            for (int i = 0; i < kPer; ++i) {
                const uint32_t x = threadIdx.x + i * kSortThreads;
                if (x < len) f(x, v[i]);
            }
        } else {
#pragma unroll 4
            for (uint32_t x = threadIdx.x; x < len; x += kSortThreads) f(x, __ldg(Q + x));
        }
    };
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
        const uint32_t x = threadIdx.x + i * kSortThreads;
        if (x < len) v[i] = __ldg(Q + x);
    }
    __syncthreads();  // the previous chunk is done with its order
    if (threadIdx.x == 0) {
        cs.lo = ~0ull;
        cs.hi = 0;
    }
    cs.cnt[threadIdx.x] = 0;
    __syncthreads();
    each([&](uint32_t, K k) {
        lo = min(lo, k);
        hi = max(hi, k);
    });
    for (int o = 16; o > 0; o >>= 1) {
        lo = min(lo, __shfl_xor_sync(0xFFFFFFFFu, lo, o));
        hi = max(hi, __shfl_xor_sync(0xFFFFFFFFu, hi, o));
    }
    if (lane == 0 && warp * 32 < len) {
        atomicMin(&cs.lo, (unsigned long long)lo);
        atomicMax(&cs.hi, (unsigned long long)hi);
    }
    __syncthreads();
    const K base = (K)cs.lo;
    const uint32_t span = bit_length(cs.hi - cs.lo), bits = bit_length(kSortBins - 1);
    const uint32_t shift = span > bits ? span - bits : 0;
    each([&](uint32_t, K k) { atomicAdd(&cs.cnt[(uint32_t)((K)(k - base) >> shift)], 1u); });
    __syncthreads();
    const uint32_t c = cs.cnt[threadIdx.x];
    uint32_t inc = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, inc, o);
        if (lane >= (uint32_t)o) inc += y;
    }
    if (lane == 31) cs.wsum[warp] = inc;
    __syncthreads();
    const uint32_t before = __reduce_add_sync(0xFFFFFFFFu, lane < warp ? cs.wsum[lane] : 0u);
    cs.cnt[threadIdx.x] = before + inc - c;
    __syncthreads();
    each([&](uint32_t x, K k) { order[atomicAdd(&cs.cnt[(uint32_t)((K)(k - base) >> shift)], 1u)] = (uint16_t)x; });
    __syncthreads();
}

// ---------------------------------------------------------------- BST, ordered chunks
// Chunks of the batch in value order, the top P = 2^T - 1 keys (as they lie) in
// shared memory.  With 1-based nodes x the children are 2x and 2x + 1; the top is
// walked without tests for equality, and an equal key there is where the path
// last went left (of several, the first such turn).  Neighbours in the order
// share their nodes far down (a level of 2^k nodes is 2^k consecutive keys), so a
// level's loads fall into a few lines.
// Measured on B200, before (as given below 2^21 queries or 64 MB, else grouped in
// device memory) -> now: 2^24 queries over 2^27 - 1 u32 keys 1118 -> 1054 us, over
// 2^26 - 1 1181 -> 844, over 2^24 - 1 1574 -> 660; 2^20 over 2^27 - 1 keys 265 -> 87, over
// 2^20 - 1 62 -> 31.  Chunks of 8192 or 16384, or 64 KB of top levels, take L1 from
// the descents (1205, 1193, 1471 us); one block an SM 1.5 times the time.
// Trees of up to 1 MB, and arrays of up to 8 MB in the search below, are searched in
// the batch's order: L1 and L2 serve them in any, and the ordering only costs (2^24
// queries, as given / in ordered chunks, us: BST over 255 u64 keys 95 / 187, over
// 65535 250 / 278, over 4e5 395 / 361, u32 over 1.5e5 222 / 248, over 4e5 304 / 291;
// sorted u64 over 255 115 / 191, over 4e5 552 / 579, over 1e6 622 / 657).
constexpr uint64_t kBstOrderBytes = 1ull << 20, kSortedOrderBytes = 8ull << 20;
constexpr uint32_t kBstChunk = 4096;
constexpr int kBstBlocksPerSM = 2;

template <typename K, typename I>
__global__ void __launch_bounds__(kSortThreads, kBstBlocksPerSM)
bst_query_sorted_kernel(const K *__restrict__ A, uint64_t n64, uint32_t P, uint32_t chunk, bool sorted,
                        const K *__restrict__ Q, uint64_t nq, uint64_t *__restrict__ ans) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    K *sm = reinterpret_cast<K *>(smem_raw);                     // [P + 1], from 1
    uint16_t *order = reinterpret_cast<uint16_t *>(sm + P + 1);  // [chunk]
    __shared__ ChunkSort cs;
    const I n = (I)n64;
    for (uint32_t x = threadIdx.x; x < P; x += kSortThreads) sm[x + 1] = __ldg(A + x);
    __syncthreads();
    const uint32_t levels = bit_length((uint64_t)P);
    for (uint64_t c0 = (uint64_t)blockIdx.x * chunk; c0 < nq; c0 += (uint64_t)gridDim.x * chunk) {
        const uint32_t len = (uint32_t)min((uint64_t)chunk, nq - c0);
        if (sorted) chunk_order<kBstChunk / kSortThreads>(Q + c0, len, order, cs);
        for (uint32_t slot = threadIdx.x; slot < len; slot += kSortThreads) {
            const uint64_t qi = c0 + (sorted ? order[slot] : slot);
            const K q = __ldg(Q + qi);
            uint32_t y = 1;
            for (uint32_t c = 0; c < levels; ++c) y = 2 * y + (sm[y] < q);
            uint32_t at = y >> __ffs(~y);
            I x = y, res = n;
            if (at && sm[at] == q) {
                // of equal keys the highest: the path's left turns above it, while they are equal too
                for (uint32_t up = at >> __ffs(~at); up && sm[up] == q; up = at >> __ffs(~at)) at = up;
                res = at - 1;
                x = n + 1;
            }
            while (x <= n) {
                const K cur = __ldg(A + (x - 1));
                if (cur == q) {
                    res = x - 1;
                    break;
                }
                x = 2 * x + (cur < q);
            }
            ans[qi] = (uint64_t)res;
        }
    }
}

// ---------------------------------------------------------------- sorted array, ordered chunks
// The same search over chunks of the batch in value order: neighbours probe the
// same keys until their intervals part, where a batch as given has every probe
// below the pinned ones in a line of its own.  Measured on B200, as given -> in
// ordered chunks: 2^24 queries over 5e8 u32 keys 7.93 -> 2.67 ms, over 9.2e7 4.12 ->
// 1.19, over 2^20 0.64 -> 0.58; 2^20 over 5e8 545 -> 189 us, 2^17 80 -> 58; 2^24 over 3e8
// u64 keys 8.22 -> 2.86 ms.  Below kSortedChunkMin the sort costs more (2^14 over 5e8
// keys 25 -> 29 us, 2^10 18 -> 23).
constexpr uint64_t kSortedChunkMin = 1ull << 16;

template <typename K, typename I>
__global__ void __launch_bounds__(kSortThreads, kBstBlocksPerSM)
sorted_query_chunk_kernel(const K *__restrict__ A, uint64_t n64, uint32_t L, uint32_t chunk, bool sorted,
                          const K *__restrict__ Q, uint64_t nq, uint64_t *__restrict__ ans) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    K *tree = reinterpret_cast<K *>(smem_raw);                              // tree[1 .. 2^L - 1]
    uint16_t *order = reinterpret_cast<uint16_t *>(tree + ((size_t)1 << L));  // [chunk]
    __shared__ ChunkSort cs;
    const I n = (I)n64;
    for (uint32_t node = threadIdx.x + 1; node < (1u << L); node += kSortThreads) {
        // replay the path of `node`: its bits below the leading one, high to low
        const uint32_t depth = 31 - __clz(node);
        I base = 0, len = n;
        for (uint32_t d = 0; d < depth; ++d) {
            const I half = len >> 1;
            if ((node >> (depth - 1 - d)) & 1u) base += half;
            len -= half;
        }
        tree[node] = __ldg(A + base + (len >> 1));
    }
    __syncthreads();
    for (uint64_t c0 = (uint64_t)blockIdx.x * chunk; c0 < nq; c0 += (uint64_t)gridDim.x * chunk) {
        const uint32_t cl = (uint32_t)min((uint64_t)chunk, nq - c0);
        if (sorted) chunk_order<kBstChunk / kSortThreads>(Q + c0, cl, order, cs);
        for (uint32_t slot = threadIdx.x; slot < cl; slot += kSortThreads) {
            const uint64_t qi = c0 + (sorted ? order[slot] : slot);
            const K q = __ldg(Q + qi);
            I base = 0, len = n;
            uint32_t node = 1;
            for (uint32_t d = 0; d < L; ++d) {  // len > 1 throughout: L < log2(n)
                const I half = len >> 1;
                const bool right = tree[node] < q;
                base += right ? half : 0;
                len -= half;
                node = 2 * node + right;
            }
            while (len > 1) {
                const I half = len >> 1;
                base += __ldg(A + base + half) < q ? half : 0;
                len -= half;
            }
            const K at = __ldg(A + base);
            const I lb = base + (at < q);
            ans[qi] = (lb < n && (lb == base ? at : __ldg(A + lb)) == q) ? (uint64_t)lb : n64;
        }
    }
}

// ---------------------------------------------------------------- mvEB
// searchvEB (gpu/src/query-mveb.cuh:43-66) finds the node at depth c of a path
// with BFS index i at pos[c] = pos[D_c] + R_c + (i & R_c) * L_c, one dependent
// key load a level.  A vEB layout stores every subtree of its recursion in one
// stretch, so here a descent goes down a piece of up to kVebPieceLevels levels
// at a time: a thread reads the piece's 2^h - 1 keys together (aligned 32-byte
// sectors), and the number of them below q is q's path through all h levels.
// With keys equal to q among them, the number of those tells which node of the
// path the highest of them is.  The order inside a piece is looked at only for
// that node's place (VebSchedule::slot): each block works out from the tables as
// given what is contiguous (veb_piece_levels), so tables of any split rule do,
// and a depth where nothing longer is contiguous is a piece of one level.  pos[]
// needs an entry per piece (8 for the 29 levels of a 3e8-key mvEB), one column per
// thread in shared memory.  The levels above the first pieces (division 0 only, as
// many as the budget holds) are gathered into shared memory in BFS order, where a
// level costs one bank access.
//
// What bounds it: a load of a thread's own line is an L1 wavefront, so a level
// at a time costs 29 a query; a 15-key piece costs at most 3 for 4 levels and a
// pinned level about a tenth.  ncu, 2^24 queries over 3e8 u32 keys: L1 data pipe
// 78 %, DRAM 48 %, issue 41 %.  Measured on B200, 2^26 queries over 3e8 u32 mvEB
// keys: a level at a time over a batch grouped by value in device memory 7.10
// ms (18.7 as given); pieces over the same grouped batch 6.2, with pinned
// levels 5.2, over chunks ordered in shared memory 4.24 (over the batch as
// given 17.1: the descents then share no pages).  Two or four lanes a piece
// 6.0 and 9.7 ms, four lanes reading each other's pieces 5.5 (half the
// wavefronts, twice the instructions); 512-thread blocks 5.8; chunks of 4096 /
// 8192 / 32768 queries 4.76 / 4.46 / 4.62; 64 KB of pinned levels 4.6 (L1 is
// smaller).  It holds for every batch: 2^10 queries 27 -> 14 us, 2^20 369 -> 95.
// From 2^22 keys equal keys are met in the pieces on the way (kPieceEq): a compare
// more a key, and no load at the end.  Below, where L1 and L2 serve the layout and
// instructions bound it, they are looked for at the path's left turns, a load for a
// miss and two for a hit.  2^24 queries, pieces / left turns (us): u32 mvEB 2e4 keys
// 502 / 430, 4e5 707 / 669, 3e6 741 / 795, 3e8 1012 / 1144; u32 standard vEB 1e6 796 /
// 707, 1e7 797 / 783, 3e7 819 / 885; u64 mvEB 1.6e4 532 / 507, 1e6 1040 / 1088, 1e7
// 1202 / 1263.
//
// A layout whose first division fits 64 KB (16 KB below 2^22 queries, where the
// blocks' gathering counts) is held whole, its batch searched as given if it has no
// other division: 2^24 queries over 255 u64 keys 391 -> 221 us, 4095 437 -> 258, 4101
// 559 -> 485, 8191 486 -> 270 (with the layout's first keys pinned and a level at a
// time 292, 481, 830 and 702).
//
// Tables whose pieces do not chain (not built by buildTable), a piece that
// reaches past its division, and divisions beyond the first kVebSchedTables
// take the descent level by level (veb_descend_levels); a descent past the
// deepest level ends as "absent" (the reference reads past its table there; it
// only ever issues hits).
constexpr uint32_t kVebPieceLevels = 4;
constexpr uint32_t kVebMaxSteps = 16;
constexpr uint64_t kVebPieceEqMin = 1ull << 22;  // keys
constexpr uint32_t kVebSchedTables = 4;  // divisions with a piece schedule (the rest hold a few keys)

struct VebStep {
    uint64_t L, R;
    uint32_t D, h;  // the earlier step the position is relative to; the piece's levels
    uint32_t c;     // the depth of the piece's root
};
struct VebSchedule {
    VebStep step[kVebMaxSteps];
    unsigned char slot[kVebMaxSteps][1u << kVebPieceLevels];  // the place in its piece of a node, in BFS order from 1
    unsigned char at[64];  // the step whose piece holds a depth
    uint32_t steps;  // 0: level by level
    uint32_t top, ktop;  // levels held in shared memory, and the step that starts below them
};

// 1-based position of the node at depth c with BFS index i.
__device__ __forceinline__ uint64_t veb_node_pos(const tl_veb_table *tab, uint32_t c, uint64_t i) {
    uint64_t p = 1;
    while (c) {
        p += tab[c].R + (i & tab[c].R) * tab[c].L;
        i >>= c - tab[c].D;
        c = tab[c].D;
    }
    return p;
}

// Whether the table stores the subtree of h levels rooted at depth c in one
// stretch of 2^h - 1 positions from its root's on: the recursion splits it at
// some depth e into a top tree and bottoms that are contiguous themselves, the
// bottoms one after the other behind the top tree.  tab has d entries.
__device__ __forceinline__ bool veb_splits(const tl_veb_table *tab, uint32_t c, uint32_t e, uint32_t h) {
    return tab[e].D == c && tab[e].R == low_mask(e - c) && tab[e].L == low_mask(c + h - e);
}
__device__ __forceinline__ bool veb_contiguous2(const tl_veb_table *tab, uint32_t d, uint32_t c) {
    return c + 2 <= d && veb_splits(tab, c, c + 1, 2);
}
__device__ __forceinline__ bool veb_contiguous3(const tl_veb_table *tab, uint32_t d, uint32_t c) {
    return c + 3 <= d && ((veb_splits(tab, c, c + 1, 3) && veb_contiguous2(tab, d, c + 1)) ||
                          (veb_splits(tab, c, c + 2, 3) && veb_contiguous2(tab, d, c)));
}
__device__ __forceinline__ uint32_t veb_piece_levels(const tl_veb_table *tab, uint32_t d, uint32_t c) {
    const bool c2 = veb_contiguous2(tab, d, c), c3 = veb_contiguous3(tab, d, c);
    if (c + 4 <= d && ((veb_splits(tab, c, c + 1, 4) && veb_contiguous3(tab, d, c + 1)) ||
                       (veb_splits(tab, c, c + 2, 4) && c2 && veb_contiguous2(tab, d, c + 2)) ||
                       (veb_splits(tab, c, c + 3, 4) && c3)))
        return 4;
    return c3 ? 3 : c2 ? 2 : 1;
}

// The piece schedule of a table of d levels, by one warp: tab gets the table,
// piece is 64 bytes of scratch.  The levels [0, out.top) go to shared memory:
// down to the start of a piece, at most max_top, all of their keys below
// position `limit` (the rightmost node of a depth has the largest position); or
// all d of them where max_top allows it.
__device__ void veb_schedule(const tl_veb_table *__restrict__ gtab, uint32_t d, uint32_t max_steps, uint32_t max_top,
                             uint64_t limit, VebSchedule &out, tl_veb_table *tab, unsigned char *piece) {
    const uint32_t lane = threadIdx.x & 31;
    for (uint32_t e = lane; e < d; e += 32) tab[e] = gtab[e];
    __syncwarp();
    bool bad = false;  // this lane's depth has a key past the limit (max_top <= 32)
    for (uint32_t c = lane; c < d; c += 32) piece[c] = (unsigned char)veb_piece_levels(tab, d, c);
    __syncwarp();
    uint32_t k = 0;
    if (lane == 0) {
        unsigned char at[64];  // the step that starts at a depth, or 255
        for (uint32_t e = 0; e < d; ++e) at[e] = 255;
        bool ok = true;
        for (uint32_t c = 0; c < d; ++k) {
            const uint32_t D = c ? tab[c].D : 0;
            ok = k < max_steps && (c == 0 || (D < c && at[D] != 255));
            if (!ok) break;
            at[c] = (unsigned char)k;
            VebStep &st = out.step[k];
            st.L = c ? tab[c].L : 0;
            st.R = c ? tab[c].R : 0;
            st.D = at[D];
            st.h = piece[c];
            st.c = c;
            c += piece[c];
        }
        k = ok ? k : 0;
        out.steps = k;
    }
    k = __shfl_sync(0xFFFFFFFFu, k, 0);
    if (k && lane < max_top) bad = veb_node_pos(tab, lane, (2ull << lane) - 1) > limit;
    const uint32_t b = __ballot_sync(0xFFFFFFFFu, bad), full = b ? __ffs(b) - 1 : 32;
    if (lane == 0) {
        uint32_t kt = 0;
        while (kt + 1 < k && out.step[kt + 1].c <= min(max_top, full)) ++kt;
        out.ktop = kt;
        out.top = k ? (max_top >= d ? d : out.step[kt].c) : 0;
    }
}

// VebSchedule::slot and ::at of one piece's node (0: none).  The recurrence of its
// position goes through nodes of the piece, up to the piece's root.
__device__ __forceinline__ void veb_slot(const tl_veb_table *tab, VebSchedule &sch, uint32_t k, uint32_t node) {
    if (k >= sch.steps || !node || node >= 1u << sch.step[k].h) return;
    const uint32_t c = sch.step[k].c, e = 31 - __clz(node);
    uint32_t p = 0, i = node;
    for (uint32_t d = c + e; d != c;) {
        const uint32_t R = (uint32_t)tab[d].R, D = tab[d].D;
        p += R + (i & R) * (uint32_t)tab[d].L;
        i >>= d - D;
        d = D;
    }
    sch.slot[k][node] = (unsigned char)p;
    if (node == 1u << e) sch.at[c + e] = (unsigned char)k;
}

// One descent level by level.  Returns 1 found (res), 2 absent, 0 left the
// division [offset, limit) (the caller tries the next one).
template <typename K>
__device__ __noinline__ int veb_descend_levels(const K *__restrict__ A, const tl_veb_table *__restrict__ tab, uint32_t d,
                                               K q, uint64_t offset, uint64_t limit, uint64_t &res) {
    uint64_t pos[64];
    uint64_t i = 1, index = 0;
    pos[0] = 1;
    for (uint32_t c = 0;;) {
        if (index + offset >= limit) return 0;
        const K cur = __ldg(A + offset + index);
        if (q == cur) {
            res = offset + index;
            return 1;
        }
        if (++c >= d) return 2;
        const uint64_t L = __ldg(&tab[c].L), R = __ldg(&tab[c].R);
        const uint32_t D = __ldg(&tab[c].D);
        if (D >= c) return 2;  // not a table built by buildTable: stop instead of reading outside pos[]
        i = 2 * i + (q > cur);
        pos[c] = pos[D] + R + (i & R) * L;
        index = pos[c] - 1;
    }
}

// idx == nullptr: perfect layout, one table (timeQueryvEB); otherwise the
// non-perfect table set (timeQueryvEB_nonperfect): the divisions in order, each
// query until it is resolved.  I: index type (32 bits when n < 2^31).  kPieceEq:
// equal keys are met in the pieces on the way; else the path is followed to its
// end on counts, and they are where it last went left (of several, the first such
// turn while the one below is equal too).
template <typename K, typename I, bool kPieceEq>
__global__ void __launch_bounds__(kSortThreads, 1)
veb_query_kernel(const K *__restrict__ A, uint64_t n64, uint32_t cols, uint32_t max_top, uint32_t chunk, bool sorted,
                 const tl_veb_table *__restrict__ tables, const uint64_t *__restrict__ idx,
                 const uint32_t *__restrict__ table_idx, uint32_t num_tables, const K *__restrict__ Q, uint64_t nq,
                 uint64_t *__restrict__ ans) {
    constexpr uint32_t KPL = 32 / sizeof(K);             // keys per sector
    constexpr uint32_t M = (1u << kVebPieceLevels) - 1;  // keys of the longest piece
    constexpr int NS = (M + KPL - 1 + KPL - 1) / KPL;    // sectors it may span
    constexpr K kAbsent = ~K(0);  // in the tree: no key there (a parent's position is below its children's)
    extern __shared__ __align__(16) unsigned char smem_raw[];
    I *pos = reinterpret_cast<I *>(smem_raw) + threadIdx.x;  // [cols][kSortThreads], this thread's column
    K *tree = reinterpret_cast<K *>(smem_raw + (size_t)cols * kSortThreads * sizeof(I));  // [2^max_top], from 1
    uint16_t *order = reinterpret_cast<uint16_t *>(tree + (1ull << max_top));             // [chunk]
    __shared__ ChunkSort cs;
    __shared__ VebSchedule sched[kVebSchedTables];
    __shared__ tl_veb_table s_tabs[kVebSchedTables][64];
    __shared__ unsigned char s_piece[kVebSchedTables][64];
    const tl_veb_table *s_tab = s_tabs[0];
    const I n = (I)n64;
    static_assert(kSortThreads / 32 >= kVebSchedTables, "a warp a division");
    if (const uint32_t j = threadIdx.x / 32; j < min(num_tables, kVebSchedTables)) {
        const uint64_t first = idx && j ? __ldg(idx + j - 1) : 0;
        veb_schedule(idx ? tables + __ldg(table_idx + j) : tables, bit_length(n64 - first), cols, j == 0 ? max_top : 0,
                     idx ? __ldg(idx + j) : n64, sched[j], s_tabs[j], s_piece[j]);
    }
    __syncthreads();
    constexpr uint32_t kSlots = kVebMaxSteps << kVebPieceLevels;  // a schedule's
    static_assert(kVebSchedTables * kSlots <= kSortThreads, "a slot a thread");
    if (const uint32_t j = threadIdx.x / kSlots; j < min(num_tables, kVebSchedTables))
        veb_slot(s_tabs[j], sched[j], (threadIdx.x % kSlots) >> kVebPieceLevels, threadIdx.x & ((1u << kVebPieceLevels) - 1));
    const uint32_t top = sched[0].top;
    const uint64_t end0 = min(n64, idx ? __ldg(idx) : n64);  // of division 0
    const bool whole = top >= bit_length(n64);               // it is all in shared memory
    for (uint32_t x = threadIdx.x + 1; x < (1u << top); x += kSortThreads) {
        const uint64_t p = veb_node_pos(s_tab, 31 - __clz(x), x) - 1;
        tree[x] = p < end0 ? __ldg(A + p) : kAbsent;
    }
    __syncthreads();
    const uint32_t a_off = (uint32_t)(reinterpret_cast<uintptr_t>(A) & 31) / sizeof(K);
    const I low = a_off ? KPL : 0;  // a piece from here on can be read in whole sectors
    for (uint64_t c0 = (uint64_t)blockIdx.x * chunk; c0 < nq; c0 += (uint64_t)gridDim.x * chunk) {
        const uint32_t len = (uint32_t)min((uint64_t)chunk, nq - c0);
        if (sorted) chunk_order<0>(Q + c0, len, order, cs);
        for (uint32_t slot = threadIdx.x; slot < len; slot += kSortThreads) {
            const uint64_t qi = c0 + (sorted ? order[slot] : slot);
            const K q = __ldg(Q + qi);
            I res = n, offset = 0;
            for (uint32_t j = 0; j < num_tables; ++j) {
                const uint64_t lim64 = idx ? __ldg(idx + j) : n64;
                const I limit = (I)lim64;
                const uint32_t steps = j < kVebSchedTables ? sched[j].steps : 0;
                bool slow = steps == 0, left = false;
                I i = 1;
                uint32_t k = 0, c = 0;
                if (j == 0 && top) {
                    uint32_t x = 1;
                    for (; c < top; ++c) x = 2 * x + (tree[x] < q);
                    i = x;
                    // an equal key is where the path last went left, or above that at a left turn equal too
                    uint32_t at = x >> __ffs(~x), hit = 0;
                    if (whole && q != kAbsent)
                        while (at && tree[at] == kAbsent) at >>= __ffs(~at);
                    if (kPieceEq || whole)
                        for (; at && tree[at] == q; at >>= __ffs(~at)) hit = at;
                    if (hit) {
                        const I p = (I)(veb_node_pos(s_tab, 31 - __clz(hit), hit) - 1);
                        if (p < limit) {
                            res = p;
                            break;
                        }
                    }
                    if (whole) {  // absent, or past the division's end where the path's last node is
                        if (!idx || veb_node_pos(s_tab, top - 1, x >> 1) <= lim64) break;
                        offset = limit;
                        continue;
                    }
                    for (; k < sched[0].ktop; ++k) {
                        const VebStep &st = sched[0].step[k];
                        const I b = i >> (top - st.c);
                        pos[k * kSortThreads] =
                            k ? (I)(pos[st.D * kSortThreads] + (I)st.R + (b & (I)st.R) * (I)st.L) : (I)1;
                    }
                }
                for (; k < steps; ++k) {
                    const VebStep &st = sched[j].step[k];
                    const uint32_t h = st.h, m = (1u << h) - 1;
                    const I p = k ? (I)(pos[st.D * kSortThreads] + (I)st.R + (i & (I)st.R) * (I)st.L) : (I)1;
                    pos[k * kSortThreads] = p;
                    const I s = offset + p - 1;
                    if (s >= limit || limit - s < (I)m) {
                        slow = s < limit;  // a piece across the division's end; else left the division
                        left = true;
                        break;
                    }
                    const uint32_t o = (uint32_t)((s + a_off) % KPL);  // the piece's first slot in its sector
                    K v[NS][KPL];
                    if (s >= low && n - s >= (I)(M + KPL)) {
                        const K *at = A + s - o;
#pragma unroll
                        for (int t = 0; t < NS; ++t)
                            if (t * KPL < o + m) ldg32(at + t * KPL, v[t]);
                    } else {
#pragma unroll
                        for (int t = 0; t < NS; ++t)
#pragma unroll
                            for (uint32_t e = 0; e < KPL; ++e) {
                                const uint32_t sl = t * KPL + e;
                                v[t][e] = sl >= o && sl < o + m ? __ldg(A + s + (sl - o)) : K(0);
                            }
                    }
                    uint32_t l = 0;
                    bool some = false;  // a slot with q's low word, in the piece or next to it
#pragma unroll
                    for (int t = 0; t < NS; ++t)
#pragma unroll
                        for (uint32_t e = 0; e < KPL; ++e) {
                            l |= (v[t][e] < q ? 1u : 0u) << (t * KPL + e);
                            if constexpr (kPieceEq) some |= (uint32_t)v[t][e] == (uint32_t)q;
                        }
                    const uint32_t piece = ((1u << m) - 1) << o, lt = __popc(l & piece);
                    if (kPieceEq && some) {
                        uint32_t eq = 0;
#pragma unroll
                        for (int t = 0; t < NS; ++t)
#pragma unroll
                            for (uint32_t e = 0; e < KPL; ++e) eq |= (v[t][e] == q ? 1u : 0u) << (t * KPL + e);
                        eq = __popc(eq & piece);
                        if (eq) {  // of the piece's keys lt + 1 .. lt + eq in order, the highest in the tree
                            const uint32_t x = (lt + eq) & ~0u << (31 - __clz(lt ^ (lt + eq))), z = __ffs(x);
                            res = s + sched[j].slot[k][1u << (h - z) | x >> z];
                            break;
                        }
                    }
                    i = (i << h) + (I)lt;
                    c += h;
                }
                const tl_veb_table *tab = idx ? tables + __ldg(table_idx + j) : tables;
                if (slow) {
                    uint64_t r = 0;
                    const int rc = veb_descend_levels(A, tab, bit_length(n64 - (uint64_t)offset), q, (uint64_t)offset,
                                                      lim64, r);
                    if (rc == 1) res = (I)r;
                    if (rc) break;
                } else {
                    if constexpr (!kPieceEq)
                        while (true) {
                            const I right = ~i;
                            const uint32_t up = sizeof(I) == 8 ? __ffsll((long long)right) : __ffs((int)right);
                            i = (i >> (up - 1)) >> 1;
                            if (!i) break;
                            c -= up;
                            const uint32_t kk = sched[j].at[c], d = c - sched[j].step[kk].c;
                            const I at = offset + (I)(pos[kk * kSortThreads] - 1 +
                                                      sched[j].slot[kk][(1u << d) | ((uint32_t)i & ((1u << d) - 1))]);
                            if (__ldg(A + at) != q) break;
                            res = at;
                        }
                    if (res != n || !left) break;  // found, or past the deepest level: absent
                }
                offset = limit;
            }
            ans[qi] = (uint64_t)res;
        }
    }
}

// ---------------------------------------------------------------- partition
// Queries close in value walk close paths through a BST, whose
// lower levels hold each subtree's keys together.  Grouping a batch by value
// lets a node fetched once from HBM serve the rest of its group from L2 or L1.
// The batch is split into 2^bits buckets of its value range [min q, max q]
// (bucket = (q - min q) >> shift, shift fitting the range to `bits` bits) by
// bits / 4 passes over 4 bits each, most significant first; `bits` grows with
// the batch (part_bits) up to 20.  A pass gives every block
// tiles of kPartTile entries; within each segment of the previous pass that a
// tile touches it ranks the entries into 16 bins in shared memory, reserves
// one global range per (segment, bin) with a single atomic, and writes each
// bin's entries out as one contiguous run.  The same pass counts the entries
// of every (segment, bin) by the next digit, so only the first pass needs a
// counting sweep of its own.  Order within a bucket is not kept (the search
// does not need it).  The search kernels write each answer through the
// carried index, so the answers keep the batch's order.
constexpr uint32_t kPartMaxBits = 20, kPartBuckets = 1u << kPartMaxBits;
constexpr uint32_t kPartDigit = 4, kPartBins = 1u << kPartDigit;
// Entries a segment of the last pass holds on average, at least: a tile that
// meets many small segments takes one portion at a time (measured on B200,
// 2^20 queries into 2^20 buckets: the last pass 0.61 ms, the whole search
// 0.06 ms; 2048 measured as fast as 1024 or faster from 2^20 to 2^27 queries)
constexpr uint64_t kPartMinSegment = 2048;
constexpr int kPartThreads = 256;
constexpr uint32_t kPartScanChunk = 4096;  // counts scanned by one block of 1024 threads
static_assert(kPartBins * kPartBins == kPartThreads, "one next-digit counter per thread");
static_assert(kPartBuckets / kPartScanChunk <= 1024, "chunk totals fit one block");
// entries per tile: the staging area of values, indices and bins in under 48 KB
template <typename K>
constexpr uint32_t part_tile() {
    return sizeof(K) == 8 ? 3584 : 4096;
}

template <typename K>
__global__ void qpart_minmax_kernel(const K *__restrict__ Q, uint64_t q, unsigned long long *__restrict__ mm) {
    unsigned long long lo = ~0ull, hi = 0;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < q; i += (uint64_t)gridDim.x * blockDim.x) {
        const unsigned long long v = (unsigned long long)Q[i];
        lo = v < lo ? v : lo;
        hi = v > hi ? v : hi;
    }
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long a = __shfl_xor_sync(0xFFFFFFFFu, lo, o), b = __shfl_xor_sync(0xFFFFFFFFu, hi, o);
        lo = a < lo ? a : lo;
        hi = b > hi ? b : hi;
    }
    __shared__ unsigned long long s_lo[32], s_hi[32];  // one atomic pair per block, not per warp
    if ((threadIdx.x & 31) == 0) {
        s_lo[threadIdx.x >> 5] = lo;
        s_hi[threadIdx.x >> 5] = hi;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (uint32_t w = 1; w < blockDim.x / 32; ++w) {
            lo = s_lo[w] < lo ? s_lo[w] : lo;
            hi = s_hi[w] > hi ? s_hi[w] : hi;
        }
        atomicMin(&mm[0], lo);
        atomicMax(&mm[1], hi);
    }
}

// The bucket of value v is the `bits` bits of (v - min q) below the top of
// the range [min q, max q]: (v - min q) >> qpart_bucket_shift(mm, bits)
__device__ __forceinline__ uint32_t qpart_bucket_shift(const unsigned long long *mm, uint32_t bits) {
    const uint32_t span = bit_length((uint64_t)(mm[1] - mm[0]));
    return span > bits ? span - bits : 0;
}

// The first segment s in [lo, nseg) whose end seg_end[s] is above a, found by
// one warp: each round probes 32 ends spread over the open range.  Needs
// seg_end non-decreasing, seg_end[s] <= a for s < lo and seg_end[nseg - 1] > a.
// consecutive: probe lo .. lo + 31 first (a portion that ended at a segment's
// end is usually followed by the next segment).
__device__ __forceinline__ uint32_t qpart_find_segment(const uint32_t *__restrict__ seg_end, uint32_t lo,
                                                       uint32_t nseg, uint64_t a, bool consecutive) {
    const uint32_t lane = threadIdx.x & 31;
    uint32_t hi = nseg;
    uint32_t step = consecutive ? 1 : (hi - lo + 31) / 32;
    for (;;) {
        const uint32_t at = min(lo + (lane + 1) * step - 1, hi - 1);
        const uint32_t hit = __ballot_sync(0xFFFFFFFFu, seg_end[at] > a);
        if (hit == 0) {  // all 32 probes at or below a (only in a consecutive round below hi)
            lo += 32 * step;
            step = (hi - lo + 31) / 32;
            continue;
        }
        const uint32_t f = __ffs(hit) - 1;
        const uint32_t at_f = min(lo + (f + 1) * step - 1, hi - 1);
        if (step == 1) return at_f;
        lo += f * step;  // just past the probe before the first hit
        hi = at_f + 1;
        step = (hi - lo + 31) / 32;
    }
}

// One pass (pass p takes bucket bits [bits - 4(p+1), bits - 4p))
// over entries [0, q) of (vals, idx) (idx == nullptr: the entry's own index).
// seg_end[0 .. nseg) are the exclusive ends of the previous pass's segments
// (nseg = 16^p; pass 0: one segment).  mode 0 adds the tiles' bin counts to
// count[seg * 16 + bin]; mode 1 scatters through cursor[] (count[] scanned)
// into (ovals, oidx) and, with next != nullptr, adds the counts of the next
// digit to next[(seg * 16 + bin) * 16 + next digit].
template <typename K>
__global__ void __launch_bounds__(kPartThreads)
qpart_pass_kernel(int mode, uint32_t bits, uint32_t pass, const K *__restrict__ vals, const uint32_t *__restrict__ idx, uint64_t q,
                  const unsigned long long *__restrict__ mm, const uint32_t *__restrict__ seg_end, uint32_t nseg,
                  uint32_t *__restrict__ count, K *__restrict__ ovals, uint32_t *__restrict__ oidx,
                  uint32_t *__restrict__ next) {
    constexpr uint32_t kPartTile = part_tile<K>();
    constexpr int kItems = kPartTile / kPartThreads;
    __shared__ K sv[kPartTile];
    __shared__ uint32_t si[kPartTile];
    __shared__ uint8_t sb[kPartTile];  // the bin of each staged entry
    __shared__ uint32_t cnt[kPartBins], off[kPartBins], run[kPartBins], base[kPartBins];
    __shared__ uint32_t nxt[kPartBins * kPartBins];
    __shared__ uint32_t s_seg[2];
    const uint64_t qmin = mm[0];
    const uint32_t shift = qpart_bucket_shift(mm, bits) + bits - kPartDigit * (pass + 1);  // this digit
    const bool count_next = mode == 1 && next != nullptr && pass + 1 < bits / kPartDigit;
    for (uint64_t t0 = (uint64_t)blockIdx.x * kPartTile; t0 < q; t0 += (uint64_t)gridDim.x * kPartTile) {
        const uint64_t t1 = min(q, t0 + kPartTile);
        uint64_t a = t0;
        uint32_t seg = 0;
        while (a < t1) {  // one segment of the previous pass at a time
            __syncthreads();
            if (threadIdx.x < 32) {  // the segment holding entry a
                const uint32_t s =
                    nseg > 1 ? qpart_find_segment(seg_end, a == t0 ? 0 : seg + 1, nseg, a, a != t0) : 0;
                if (threadIdx.x == 0) {
                    s_seg[0] = s;
                    s_seg[1] = nseg > 1 ? seg_end[s] : (uint32_t)q;  // pass 0: one segment [0, q)
                }
            }
            if (threadIdx.x < kPartBins) {
                cnt[threadIdx.x] = 0;
                run[threadIdx.x] = 0;
            }
            nxt[threadIdx.x] = 0;
            __syncthreads();
            seg = s_seg[0];
            uint64_t b = min(t1, (uint64_t)s_seg[1]);
            if (b <= a) b = t1;  // cannot happen (the last end is q); both modes take the same steps
            const uint32_t len = (uint32_t)(b - a);
            // this thread's entries j = threadIdx.x + i * kPartThreads of the
            // portion, values and indices loaded together (their latencies
            // overlap) and kept in registers
            K v[kItems];
            uint32_t id[kItems];
#pragma unroll
            for (int i = 0; i < kItems; ++i) {
                const uint32_t j = threadIdx.x + i * kPartThreads;
                v[i] = j < len ? vals[a + j] : K(0);
                id[i] = mode == 1 && idx && j < len ? idx[a + j] : (uint32_t)(a + j);
            }
#pragma unroll
            for (int i = 0; i < kItems; ++i) {
                const uint32_t j = threadIdx.x + i * kPartThreads;
                if (j < len) atomicAdd(&cnt[(((uint64_t)v[i] - qmin) >> shift) & (kPartBins - 1)], 1u);
            }
            __syncthreads();
            if (mode == 0) {
                if (threadIdx.x < kPartBins && cnt[threadIdx.x])
                    atomicAdd(&count[seg * kPartBins + threadIdx.x], cnt[threadIdx.x]);
            } else {
                if (threadIdx.x == 0) {
                    uint32_t o = 0;
                    for (uint32_t k = 0; k < kPartBins; ++k) {
                        off[k] = o;
                        o += cnt[k];
                    }
                }
                if (threadIdx.x < kPartBins && cnt[threadIdx.x])
                    base[threadIdx.x] = atomicAdd(&count[seg * kPartBins + threadIdx.x], cnt[threadIdx.x]);
                __syncthreads();
#pragma unroll
                for (int i = 0; i < kItems; ++i) {  // rank into the staging area
                    const uint32_t j = threadIdx.x + i * kPartThreads;
                    if (j < len) {
                        const uint64_t rel = (uint64_t)v[i] - qmin;
                        const uint32_t bin = (uint32_t)(rel >> shift) & (kPartBins - 1);
                        const uint32_t r = off[bin] + atomicAdd(&run[bin], 1u);
                        sv[r] = v[i];
                        si[r] = id[i];
                        sb[r] = (uint8_t)bin;
                        if (count_next)
                            atomicAdd(&nxt[bin * kPartBins +
                                           ((uint32_t)(rel >> (shift - kPartDigit)) & (kPartBins - 1))],
                                      1u);
                    }
                }
                if (threadIdx.x < kPartBins) base[threadIdx.x] -= off[threadIdx.x];  // bin's entry j goes to base + j
                __syncthreads();
                for (uint32_t j = threadIdx.x; j < len; j += blockDim.x) {  // each bin as one run
                    const uint32_t p = base[sb[j]] + j;
                    ovals[p] = sv[j];
                    oidx[p] = si[j];
                }
                // (segment, bin) of this pass is segment seg * 16 + bin of the
                // next: its counters start at (seg * 16 + bin) * 16
                if (count_next && nxt[threadIdx.x])
                    atomicAdd(&next[(uint64_t)seg * kPartBins * kPartBins + threadIdx.x], nxt[threadIdx.x]);
            }
            a = b;
        }
    }
}

// Exclusive scan of count[0, m) in place, m a multiple of kPartScanChunk: block
// c scans chunk c; ends (when given) gets the inclusive sums and total[c] the
// chunk's sum.  With more than one chunk, qpart_scan_add_kernel then adds the
// sums of the chunks before each one.
__global__ void __launch_bounds__(1024) qpart_scan_kernel(uint32_t *__restrict__ count, uint32_t *__restrict__ ends,
                                                          uint32_t *__restrict__ total) {
    static_assert(kPartScanChunk == 4 * 1024, "four counts a thread");
    __shared__ uint32_t wsum[32];
    const uint64_t at = (uint64_t)blockIdx.x * kPartScanChunk + threadIdx.x * 4;
    const uint4 c = *reinterpret_cast<const uint4 *>(count + at);
    const uint32_t sum = c.x + c.y + c.z + c.w;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t inc = sum;  // inclusive scan within the warp
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, inc, o);
        if (lane >= (uint32_t)o) inc += t;
    }
    if (lane == 31) wsum[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = wsum[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, w, o);
            if (lane >= (uint32_t)o) w += t;
        }
        wsum[lane] = w;  // inclusive over warps
        if (lane == 31 && total) total[blockIdx.x] = w;
    }
    __syncthreads();
    const uint32_t r0 = (warp ? wsum[warp - 1] : 0) + inc - sum;
    const uint4 ex = make_uint4(r0, r0 + c.x, r0 + c.x + c.y, r0 + c.x + c.y + c.z);
    *reinterpret_cast<uint4 *>(count + at) = ex;
    if (ends) *reinterpret_cast<uint4 *>(ends + at) = make_uint4(ex.y, ex.z, ex.w, ex.w + c.w);
}

// Block c of the grid adds the sums of chunks [0, c + 1) to chunk c + 1.
__global__ void __launch_bounds__(1024) qpart_scan_add_kernel(uint32_t *__restrict__ count,
                                                              uint32_t *__restrict__ ends,
                                                              const uint32_t *__restrict__ total) {
    __shared__ uint32_t s_off;
    const uint32_t chunk = blockIdx.x + 1;
    if (threadIdx.x < 32) {
        uint32_t o = 0;
        for (uint32_t k = threadIdx.x; k < chunk; k += 32) o += total[k];
        o = __reduce_add_sync(0xFFFFFFFFu, o);
        if (threadIdx.x == 0) s_off = o;
    }
    __syncthreads();
    const uint32_t o = s_off;
    const uint64_t at = (uint64_t)chunk * kPartScanChunk + threadIdx.x * 4;
    uint4 c = *reinterpret_cast<const uint4 *>(count + at);
    *reinterpret_cast<uint4 *>(count + at) = make_uint4(c.x + o, c.y + o, c.z + o, c.w + o);
    if (ends) {
        c = *reinterpret_cast<const uint4 *>(ends + at);
        *reinterpret_cast<uint4 *>(ends + at) = make_uint4(c.x + o, c.y + o, c.z + o, c.w + o);
    }
}

static int query_sm_count();

// Device memory of one partitioned batch: stream-ordered, freed (on the same
// stream, after the search kernel) when the launch function returns.
struct QueryPartition {
    void *buf = nullptr;
    const void *qs = nullptr;
    const uint32_t *perm = nullptr;
    cudaStream_t st = nullptr;
    ~QueryPartition() {
        if (buf) cudaFreeAsync(buf, st);
    }
};

// Bucket bits for a batch of q queries: the most (a multiple of 4, at most
// kPartMaxBits) whose last pass still has kPartMinSegment entries a segment
// on average, and at least 4.
static uint32_t part_bits(uint64_t q) {
    uint32_t bits = kPartDigit;
    while (bits + kPartDigit <= kPartMaxBits && (q >> bits) >= kPartMinSegment) bits += kPartDigit;
    return bits;
}

template <typename K>
static int partition_queries(const K *Q, uint64_t q, cudaStream_t st, QueryPartition &out) {
    auto al = [](uint64_t x) { return (x + 255) / 256 * 256; };
    auto padded = [](uint32_t m) { return (m + kPartScanChunk - 1) / kPartScanChunk * kPartScanChunk; };
    const uint32_t bits = part_bits(q), passes = bits / kPartDigit;
    // mm and the scan's chunk totals | the counts of this pass and of the
    // next (up to 2^bits each) | segment ends of the previous pass and of
    // this one | two (vals, idx) buffers
    const uint64_t b_mm = 256 + 4096, b_c = al(padded(1u << bits) * 4ull), b_v = al(q * sizeof(K)),
                   b_i = al(q * 4);
    char *buf = nullptr;
    keep_pool_memory();
    if (cudaMallocAsync(reinterpret_cast<void **>(&buf), b_mm + 4 * b_c + 2 * (b_v + b_i), st) != cudaSuccess) {
        cudaGetLastError();
        return TL_ERROR_OUT_OF_MEMORY;
    }
    out.buf = buf;  // freed by out's destructor on every path from here
    out.st = st;
    char *p = buf;
    unsigned long long *mm = reinterpret_cast<unsigned long long *>(p);
    uint32_t *total = reinterpret_cast<uint32_t *>(p + 256);
    p += b_mm;
    uint32_t *cnt[2] = {reinterpret_cast<uint32_t *>(p), reinterpret_cast<uint32_t *>(p + b_c)};
    p += 2 * b_c;
    uint32_t *ends[2] = {reinterpret_cast<uint32_t *>(p), reinterpret_cast<uint32_t *>(p + b_c)};
    p += 2 * b_c;
    K *v[2] = {reinterpret_cast<K *>(p), reinterpret_cast<K *>(p + b_v + b_i)};
    uint32_t *ix[2] = {reinterpret_cast<uint32_t *>(p + b_v), reinterpret_cast<uint32_t *>(p + 2 * b_v + b_i)};
    TL_CUDA_TRY(cudaMemsetAsync(mm, 0xFF, 8, st));  // min: all ones
    TL_CUDA_TRY(cudaMemsetAsync(mm + 1, 0, 8, st));
    const unsigned g = (unsigned)std::min<uint64_t>((q + 255) / 256, (uint64_t)query_sm_count() * 8);
    qpart_minmax_kernel<K><<<g, 256, 0, st>>>(Q, q, mm);
    const unsigned gt =
        (unsigned)std::min<uint64_t>((q + part_tile<K>() - 1) / part_tile<K>(), (uint64_t)query_sm_count() * 8);
    const K *src_v = Q;
    const uint32_t *src_i = nullptr;
    uint32_t nseg = 1;
    TL_CUDA_TRY(cudaMemsetAsync(cnt[0], 0, (size_t)padded(kPartBins) * 4, st));
    qpart_pass_kernel<K><<<gt, kPartThreads, 0, st>>>(0, bits, 0, src_v, src_i, q, mm, ends[1], 1, cnt[0], nullptr,
                                                      nullptr, nullptr);
    for (uint32_t pass = 0; pass < passes; ++pass) {
        const uint32_t m = nseg * kPartBins;  // this pass's buckets
        const uint32_t *seg = ends[(pass + 1) & 1];
        uint32_t *next_ends = ends[pass & 1];
        uint32_t *count = cnt[pass & 1], *next = nullptr;
        const uint32_t chunks = padded(m) / kPartScanChunk;
        qpart_scan_kernel<<<chunks, 1024, 0, st>>>(count, next_ends, total);
        if (chunks > 1) qpart_scan_add_kernel<<<chunks - 1, 1024, 0, st>>>(count, next_ends, total);
        if (pass + 1 < passes) {
            next = cnt[(pass + 1) & 1];
            TL_CUDA_TRY(cudaMemsetAsync(next, 0, (size_t)padded(m * kPartBins) * 4, st));
        }
        K *dv = v[pass & 1];
        uint32_t *di = ix[pass & 1];
        qpart_pass_kernel<K><<<gt, kPartThreads, 0, st>>>(1, bits, pass, src_v, src_i, q, mm, seg, nseg, count, dv,
                                                          di, next);
        src_v = dv;
        src_i = di;
        nseg = m;
    }
    TL_CUDA_TRY(cudaGetLastError());
    out.qs = src_v;
    out.perm = src_i;
    return TL_SUCCESS;
}

// ---------------------------------------------------------------- host
static int g_qsm = 0;
static int query_sm_count() {
    if (!g_qsm) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&g_qsm, cudaDevAttrMultiProcessorCount, dev);
        if (g_qsm <= 0) g_qsm = 148;
    }
    return g_qsm;
}

// Dynamic shared memory a launch of each kernel may ask for at most.  A launch
// sets this as its kernel's limit, not its own need: the limit belongs to the
// kernel, and a smaller call on another host thread, between this one's limit and
// its launch, would have the launch refused (seen with 2^10 beside 2^22 vEB
// queries; below 48 KB too, once a limit has been set).
constexpr size_t kSmemLimit = 64 * 1024;                                                       // persistent_grid
constexpr size_t kChunkSmemMax = 32768 + kBstChunk * sizeof(uint16_t);                         // BST and sorted chunks
constexpr size_t kTopSmemMax = kTopBytes + (kTopBins + 1) * sizeof(uint16_t);                  // btree_query_top_kernel
constexpr size_t kVebTopMax = 32768;
constexpr size_t kVebWholeMax = 65536;
constexpr size_t veb_smem_max(size_t index_bytes) {  // (the wide index comes with layouts that are not held whole)
    return kVebMaxSteps * kSortThreads * index_bytes + (index_bytes == 4 ? kVebWholeMax : kVebTopMax) +
           kSortChunk * sizeof(uint16_t);
}

// Resident blocks per SM of a kernel, asked of the runtime once per thread, device
// and shape (the question and the attribute cost a small batch's call a
// microsecond of its four).
static int resident_blocks(const void *kern, size_t smem, int *per_sm) {
    struct Known {
        const void *kern;
        size_t smem;
        int dev, per_sm;
    };
    constexpr int kKnown = 32;
    static thread_local Known known[kKnown];
    static thread_local int count = 0;
    int dev = 0;
    TL_CUDA_TRY(cudaGetDevice(&dev));
    for (int i = 0; i < std::min(count, kKnown); ++i)
        if (known[i].kern == kern && known[i].smem == smem && known[i].dev == dev) {
            *per_sm = known[i].per_sm;
            return TL_SUCCESS;
        }
    // all ask for at most kPinBytes
    static_assert(kPinBytes <= kSmemLimit, "the pinned prefix fits the limit");
    if (smem > kSmemLimit) return TL_ERROR_UNSUPPORTED;
    TL_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemLimit));
    TL_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, kern, kQueryThreads, smem));
    known[count++ % kKnown] = Known{kern, smem, dev, *per_sm};  // the oldest goes first
    if (count == 2 * kKnown) count = kKnown;
    return TL_SUCCESS;
}

template <typename Kern>
static int persistent_grid(Kern kern, size_t smem, uint64_t work_threads, unsigned *grid) {
    int per_sm = 0;
    const int rc = resident_blocks(reinterpret_cast<const void *>(kern), smem, &per_sm);
    if (rc) return rc;
    uint64_t g = (uint64_t)std::max(per_sm, 1) * query_sm_count();
    uint64_t need = (work_threads + kQueryThreads - 1) / kQueryThreads;
    *grid = (unsigned)std::max<uint64_t>(1, std::min(g, need));
    return TL_SUCCESS;
}

template <typename K>
static int launch_query(const QueryArgs &a, cudaStream_t st) {
    const K *A = static_cast<const K *>(a.layout_keys);
    const K *Q = static_cast<const K *>(a.queries);
    uint64_t P = std::min<uint64_t>(a.n, kPinBytes / sizeof(K));
    unsigned grid = 1;
    // A large batch over a large BST is grouped by value in device memory: its
    // warps then share nodes much further down than a chunk's do, for two passes
    // over the batch per 4 bits and answers written to random places.  Measured on
    // B200, grouped / in ordered chunks (us): 2^27 - 1 u32 keys (512 MB) 2^24
    // queries 1129 / 1063, 2^27 9617 / 8487; 2^28 - 1 u32 (1 GB) 2^21 230 / 188, 2^22
    // 370 / 355, 2^23 650 / 702, 2^24 1196 / 1371; 2^30 - 1 u32 2^21 297 / 274, 2^22
    // 513 / 553, 2^24 1458 / 2455; u64 of 512 MB 2^24 1265 / 1136, of 2 GB 1442 / 2086.
    // From 4 GB smaller batches gain too: 2^21 / 3 * 2^20 / 2^22 queries over 2^30 - 1 u32
    // keys 280 / 386 / 481 grouped, 260 / 395 / 534 in chunks, over 2^30 - 1 u64 333 / 451 /
    // 577 and 321 / 495 / 676; over 2 GB 239 / 324 / 398 and 214 / 309 / 413.
    // Measurement hooks: variant 19 never groups, 20 always.
    QueryPartition part;
    const uint32_t *perm = nullptr;
    const uint64_t tree_bytes = a.n * sizeof(K);
    const bool large = tree_bytes >= (1ull << 30) - 1024;  // 2^28 - 1 u32 keys included
    const bool huge = tree_bytes >= (4ull << 30) - 1024;   // 2^30 - 1 u32 keys included
    if (a.layout == Q_BST && g_query_variant != 19 && a.q < (1ull << 32) &&
        (g_query_variant == 20 || (large && a.q > (1ull << 22)) || (huge && a.q >= (3ull << 20)))) {
        const int rc = partition_queries<K>(Q, a.q, st, part);
        if (rc == TL_SUCCESS) {
            Q = static_cast<const K *>(part.qs);
            perm = part.perm;
        } else if (rc != TL_ERROR_OUT_OF_MEMORY) {
            return rc;  // out of memory: the batch is searched as given
        }
    }
    if (a.layout == Q_SORTED) {
        // pinned probe tree: L levels with 2^L - 1 < n (so every pinned step has
        // len > 1) and at most 32 KB of keys
        uint32_t L = 0;
        while (L < 12 && ((2ull << L) - 1) * sizeof(K) <= 32768 && (2ull << L) <= a.n) ++L;
        if (a.q >= kSortedChunkMin) {
            const uint64_t slots = (uint64_t)query_sm_count() * kBstBlocksPerSM;
            const uint64_t rounds = (a.q + slots * kBstChunk - 1) / (slots * kBstChunk);
            const uint64_t chunk = (a.q + slots * rounds - 1) / (slots * rounds);  // equal chunks, the fewest rounds
            const size_t bytes = ((size_t)1 << L) * sizeof(K) + chunk * sizeof(uint16_t);
            auto launch = [&](auto kern) -> int {
                TL_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kChunkSmemMax));
                kern<<<(unsigned)std::min(slots, (a.q + chunk - 1) / chunk), kSortThreads, bytes, st>>>(
                    A, a.n, L, (uint32_t)chunk, tree_bytes > kSortedOrderBytes, Q, a.q, a.answers);
                TL_CUDA_TRY(cudaGetLastError());
                return TL_SUCCESS;
            };
            return a.n < (1ull << 31) ? launch(sorted_query_chunk_kernel<K, uint32_t>)
                                      : launch(sorted_query_chunk_kernel<K, uint64_t>);
        }
        const size_t smem = ((size_t)1 << L) * sizeof(K);
        auto kern = sorted_query_kernel<K>;
        int rc = persistent_grid(kern, smem, a.q, &grid);
        if (rc) return rc;
        kern<<<grid, kQueryThreads, smem, st>>>(A, a.n, L, Q, a.q, a.answers);
    } else if (a.layout == Q_BST && perm) {
        uint64_t top = 1;  // whole top levels: 2^T - 1 keys
        while ((top * 2 + 1) * sizeof(K) <= kBstGroupPinBytes) top = top * 2 + 1;
        P = std::min<uint64_t>(top, a.n);
        size_t smem = P * sizeof(K);
        auto kern = bst_query_kernel<K>;
        int rc = persistent_grid(kern, smem, a.q, &grid);
        if (rc) return rc;
        kern<<<grid, kQueryThreads, smem, st>>>(A, a.n, P, Q, a.q, perm, a.answers);
    } else if (a.layout == Q_BST) {
        uint64_t top = 1;  // whole top levels, at most 32 KB with the unused slot 0
        while (top * 2 + 1 <= a.n && (top * 2 + 2) * sizeof(K) <= 32768) top = top * 2 + 1;
        const uint64_t slots = (uint64_t)query_sm_count() * kBstBlocksPerSM;
        const uint64_t rounds = (a.q + slots * kBstChunk - 1) / (slots * kBstChunk);
        const uint64_t chunk = (a.q + slots * rounds - 1) / (slots * rounds);  // equal chunks, the fewest rounds
        const size_t smem = (top + 1) * sizeof(K) + chunk * sizeof(uint16_t);
        auto launch = [&](auto kern) -> int {
            TL_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kChunkSmemMax));
            kern<<<(unsigned)std::min(slots, (a.q + chunk - 1) / chunk), kSortThreads, smem, st>>>(
                A, a.n, (uint32_t)top, (uint32_t)chunk, tree_bytes > kBstOrderBytes, Q, a.q, a.answers);
            return TL_SUCCESS;
        };
        const int rc = a.n < (1ull << 31) ? launch(bst_query_sorted_kernel<K, uint32_t>)
                                          : launch(bst_query_sorted_kernel<K, uint64_t>);
        if (rc) return rc;
    } else if (a.layout == Q_BTREE) {
        uint64_t top = 0, lvl = a.b;
        while (top + lvl <= P) {  // whole top levels: (b+1)^L - 1 keys
            top += lvl;
            if (lvl > UINT64_MAX / (a.b + 1)) break;
            lvl *= a.b + 1;
        }
        P = std::min<uint64_t>(top, a.n);
        size_t smem = P * sizeof(K);
        // a group of max(2, b * w / 64) lanes per query with 32-byte loads (b * w
        // = 64, 128 or 256 on a 32-byte aligned layout), else a thread per query
        // with 32-byte node loads (b * w a multiple of 32), else 16-byte ones
        // (b * w a multiple of 16), else a group of lanes per query with one key
        // per lane
        const uint64_t node_bytes = a.b * sizeof(K);
        const uintptr_t base = reinterpret_cast<uintptr_t>(A);
        int rc = TL_SUCCESS;
        bool done = false;
        auto v32 = [&](auto kern, bool pin) -> int {
            rc = persistent_grid(kern, pin ? smem : 0, a.q, &grid);
            if (rc) return rc;
            kern<<<grid, kQueryThreads, pin ? smem : 0, st>>>(A, a.n, pin ? P : 0, Q, a.q, a.answers);
            done = true;
            return TL_SUCCESS;
        };
        auto v16 = [&](auto kern) -> int {
            rc = persistent_grid(kern, 0, a.q, &grid);
            if (rc) return rc;
            kern<<<grid, kQueryThreads, 0, st>>>(A, a.n, a.b, Q, a.q, a.answers);
            done = true;
            return TL_SUCCESS;
        };
        const bool pin = g_query_variant == 5;
        auto grp = [&](auto kern, uint64_t lanes_per_query) -> int {
            rc = persistent_grid(kern, 0, a.q * lanes_per_query, &grid);
            if (rc) return rc;
            kern<<<grid, kQueryThreads, 0, st>>>(A, a.n, Q, a.q, a.answers);
            done = true;
            return TL_SUCCESS;
        };
        // default: nodes of 64, 128 or 256 bytes on a 32-byte aligned layout are
        // read by a group of max(2, node_bytes / 64) lanes.  Measured on B200,
        // 2^27 queries, q/s with 2 / 4 / 8 lanes per node against a thread per
        // query with 32-byte loads: b = 16 u64 over 5e8 keys 14.2e9 / 9.53e9 /
        // - against 6.54e9; b = 32 u64 over 2^28 keys 8.33e9 / 9.08e9 / 6.06e9
        // against 4.28e9; b = 16 u32 over 2^30 keys 17.7e9 against 11.7e9;
        // b = 8 u64 over 2^30 keys 12.7e9 against 8.56e9
        // from 2^20 queries (a block gathers and indexes its top first: over 5e8
        // u64 keys 2^18 queries 32 / 32 us, 2^19 50 / 49, 2^20 88 / 83; over 2^20
        // keys 20 / 23, 32 / 31, 54 / 42) the whole top levels that 40 KB hold are
        // searched in shared memory (10 KB, two levels at b = 16: 838 against 702
        // us over 1e8 keys).  Variant 9 takes this form at any size.
        const uint64_t m = btree_top_keys<K>(a.n, a.b);
        auto topped = [&](auto kern, uint64_t lanes_per_query) -> int {
            const size_t bytes = m * sizeof(K) + (kTopBins + 1) * sizeof(uint16_t);
            TL_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTopSmemMax));
            const uint64_t need = (a.q * lanes_per_query + kTopThreads - 1) / kTopThreads;
            kern<<<(unsigned)std::min<uint64_t>(2 * (uint64_t)query_sm_count(), need), kTopThreads, bytes, st>>>(
                A, (uint32_t)a.n, (uint32_t)m, Q, a.q, a.answers);
            done = true;
            return TL_SUCCESS;
        };
        if ((base & 31) == 0 && m && a.n < (1ull << 31) &&
            (g_query_variant == 9 ||
             (g_query_variant == 0 && a.q >= (1ull << 20) && (node_bytes != 128 || a.n * sizeof(K) <= kTopMaxBytes128)))) {
            switch (node_bytes) {
                case 64: rc = topped(btree_query_top_kernel<K, 64, 2>, 2); break;
                case 128: rc = topped(btree_query_top_kernel<K, 128, 2>, 2); break;
                case 256: rc = topped(btree_query_top_kernel<K, 256, 4>, 4); break;
                default: break;
            }
        }
        if (!done && (base & 31) == 0 && g_query_variant != 2 && g_query_variant != 5 && g_query_variant != 6) {
            if (g_query_variant == 7) {  // one 32-byte load per lane
                switch (node_bytes) {
                    case 128: rc = grp(btree_query_group32_kernel<K, 128, 4>, 4); break;
                    case 256: rc = grp(btree_query_group32_kernel<K, 256, 8>, 8); break;
                    default: break;
                }
            }
            if (!done) {  // two 32-byte loads per lane (one for 64-byte nodes)
                switch (node_bytes) {
                    case 64: rc = grp(btree_query_group32_kernel<K, 64, 2>, 2); break;
                    case 128: rc = grp(btree_query_group32_kernel<K, 128, 2>, 2); break;
                    case 256: rc = grp(btree_query_group32_kernel<K, 256, 4>, 4); break;
                    default: break;
                }
            }
        }
        if (!done && (base & 31) == 0 && node_bytes % 32 == 0 && g_query_variant != 2) {
            switch (node_bytes) {
                case 32: rc = pin ? v32(btree_query_v32_kernel<K, 32, true>, true) : v32(btree_query_v32_kernel<K, 32, false>, false); break;
                case 64: rc = pin ? v32(btree_query_v32_kernel<K, 64, true>, true) : v32(btree_query_v32_kernel<K, 64, false>, false); break;
                case 128: rc = pin ? v32(btree_query_v32_kernel<K, 128, true>, true) : v32(btree_query_v32_kernel<K, 128, false>, false); break;
                case 256: rc = pin ? v32(btree_query_v32_kernel<K, 256, true>, true) : v32(btree_query_v32_kernel<K, 256, false>, false); break;
                default: break;
            }
        }
        if (!done && (base & 15) == 0 && node_bytes % 16 == 0) {
            switch (node_bytes / 16) {
                case 1: rc = v16(btree_query_vec_kernel<K, 1>); break;
                case 2: rc = v16(btree_query_vec_kernel<K, 2>); break;
                case 4: rc = v16(btree_query_vec_kernel<K, 4>); break;
                case 8: rc = v16(btree_query_vec_kernel<K, 8>); break;
                case 16: rc = v16(btree_query_vec_kernel<K, 16>); break;
                default: break;
            }
        }
        if (rc) return rc;
        if (done) {
            TL_CUDA_TRY(cudaGetLastError());
            return TL_SUCCESS;
        }
        int G = 1;
        while (G < 32 && (uint64_t)G < a.b) G <<= 1;
#define TL_BT(GG)                                                                          \
    case GG: {                                                                             \
        auto kern = btree_query_kernel<K, GG>;                                             \
        rc = persistent_grid(kern, smem, a.q * GG, &grid);                                 \
        if (rc) return rc;                                                                 \
        kern<<<grid, kQueryThreads, smem, st>>>(A, a.n, a.b, P, Q, a.q, a.answers);        \
        break;                                                                             \
    }
        switch (G) {
            TL_BT(1)
            TL_BT(2)
            TL_BT(4)
            TL_BT(8)
            TL_BT(16)
            TL_BT(32)
        }
#undef TL_BT
    } else {
        const uint32_t dmax = bit_length(a.n);
        if (dmax > 63) return TL_ERROR_UNSUPPORTED;
        const bool np = a.layout == Q_VEB_NP;
        const bool narrow = a.n < (1ull << 31);
        // pieces are 2.5 levels long on average at worst (heights 2, 3, 2, 3, ...)
        const uint32_t cols = std::min<uint32_t>(kVebMaxSteps, (2 * dmax + 4) / 5 + 1);
        // pinned levels: at most 32 KB from 2^20 queries, else 16 KB (a block
        // gathers them; 2^18 queries over 3e8 u32 keys 41 against 44 us, 2^20 97
        // against 94)
        const size_t top_bytes = a.q >= (1ull << 20) ? kVebTopMax : kVebTopMax / 2;
        // a small layout is held whole, and its batch searched as given
        const bool whole = (sizeof(K) << dmax) <= (a.q >= (1ull << 22) ? kVebWholeMax : kVebTopMax / 2);
        uint32_t max_top = whole ? dmax : 0;
        while (max_top + 1 < dmax && (sizeof(K) << (max_top + 1)) <= top_bytes) ++max_top;
        auto launch = [&](auto kern) -> int {
            const uint64_t slots = query_sm_count();
            const uint64_t rounds = (a.q + slots * kSortChunk - 1) / (slots * kSortChunk);
            const uint64_t chunk = (a.q + slots * rounds - 1) / (slots * rounds);  // equal chunks, the fewest rounds
            const size_t smem = (size_t)cols * kSortThreads * (narrow ? 4 : 8) + (sizeof(K) << max_top) +
                                chunk * sizeof(uint16_t);
            TL_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)veb_smem_max(narrow ? 4 : 8)));
            const uint64_t blocks = std::min(slots, (a.q + chunk - 1) / chunk);
            kern<<<(unsigned)blocks, kSortThreads, smem, st>>>(A, a.n, cols, max_top, (uint32_t)chunk, !whole || (np && a.num_tables > 1), a.tables,
                                                              np ? a.idx : nullptr, np ? a.table_idx : nullptr,
                                                              np ? a.num_tables : 1u, Q, a.q, a.answers);
            return TL_SUCCESS;
        };
        const int rc = a.n < kVebPieceEqMin ? launch(veb_query_kernel<K, uint32_t, false>)
                       : narrow             ? launch(veb_query_kernel<K, uint32_t, true>)
                                            : launch(veb_query_kernel<K, uint64_t, true>);
        if (rc) return rc;
    }
    TL_CUDA_TRY(cudaGetLastError());
    return TL_SUCCESS;
}

int query(const QueryArgs &a, cudaStream_t st, float *ms) {
    if (a.q == 0) {
        if (ms) *ms = 0.f;
        return TL_SUCCESS;
    }
    if (!a.queries || !a.answers) return TL_ERROR_INVALID_VALUE;
    if (a.n == 0) {
        TL_CUDA_TRY(cudaMemsetAsync(a.answers, 0, a.q * sizeof(uint64_t), st));
        if (ms) *ms = 0.f;
        return sync_and_check(st);
    }
    if (!a.layout_keys) return TL_ERROR_INVALID_VALUE;
    if (a.layout == Q_BTREE && a.b == 0) return TL_ERROR_INVALID_VALUE;
    if ((a.layout == Q_VEB || a.layout == Q_VEB_NP) && !a.tables) return TL_ERROR_INVALID_VALUE;
    if (a.layout == Q_VEB_NP && (!a.idx || !a.table_idx || a.num_tables == 0)) return TL_ERROR_INVALID_VALUE;
    EventTimer timer(ms != nullptr, st);
    timer.start();
    int rc = a.key_bytes == 8 ? launch_query<uint64_t>(a, st) : launch_query<uint32_t>(a, st);
    timer.stop();
    if (rc) return rc;
    if (ms) {
        rc = sync_and_check(st);
        if (rc) return rc;
        *ms = timer.elapsed();
    }
    return TL_SUCCESS;
}

// ---------------------------------------------------------------- replay
namespace {
// An array whose accesses are checked: one out of range counts and goes nowhere.
template <typename V>
struct Checked {
    V *v;
    uint32_t len;
    uint64_t *violations;
    mutable V nowhere{};
    TL_HD V &operator[](uint32_t i) const {
        if (i < len) return v[i];
        ++*violations;
        return nowhere;
    }
};

template <typename K, uint32_t B>
void replay_top(const K *A, uint32_t m, const K *Q, uint64_t q, uint64_t *ranks, uint64_t *violations) {
    std::vector<K> top_keys(m);
    std::vector<uint16_t> bins(kTopBins + 1, 0);
    const Checked<K> top{top_keys.data(), m, violations};
    const Checked<uint16_t> bin{bins.data(), kTopBins + 1, violations};
    for (uint32_t p = 0; p < m; ++p) {
        const uint32_t r = top_rank_of<B>(p, m);
        top[r] = A[p];
        if (top_position<B>(r, m) != p) ++*violations;
    }
    const K first = top_keys[0];
    const uint32_t shift = top_shift(first, top_keys[m - 1]);
    for (uint32_t r = 0; r <= m; ++r) top_fill(top, m, first, shift, r, bin);
    for (uint64_t i = 0; i < q; ++i) {
        ranks[i] = top_rank(top, bin, m, first, shift, Q[i]);
        if (ranks[i] > m) ++*violations;
    }
}

template <typename K>
int emulate_top(const K *A, uint64_t n, uint64_t b, const K *Q, uint64_t q, uint64_t *ranks, uint64_t *violations) {
    const uint64_t m = btree_top_keys<K>(n, b);
    if (!m) return TL_ERROR_UNSUPPORTED;
    switch (b * sizeof(K)) {
        case 64: replay_top<K, 64 / sizeof(K)>(A, (uint32_t)m, Q, q, ranks, violations); break;
        case 128: replay_top<K, 128 / sizeof(K)>(A, (uint32_t)m, Q, q, ranks, violations); break;
        case 256: replay_top<K, 256 / sizeof(K)>(A, (uint32_t)m, Q, q, ranks, violations); break;
        default: return TL_ERROR_UNSUPPORTED;
    }
    return TL_SUCCESS;
}
}  // namespace

// Host replay of btree_query_top_kernel's set-up and of its search of the top
// levels (test hook): the top keys below each query, and the accesses that left
// their array.  The words of A need not be in layout order.
int emulate_btree_top(const void *A, uint64_t n, uint64_t b, uint32_t key_bytes, const void *Q, uint64_t q,
                      uint64_t *ranks, uint64_t *violations) {
    if (!A || !Q || !ranks || !violations || b == 0) return TL_ERROR_INVALID_VALUE;
    *violations = 0;
    if (key_bytes == 8)
        return emulate_top(static_cast<const uint64_t *>(A), n, b, static_cast<const uint64_t *>(Q), q, ranks,
                           violations);
    if (key_bytes == 4)
        return emulate_top(static_cast<const uint32_t *>(A), n, b, static_cast<const uint32_t *>(Q), q, ranks,
                           violations);
    return TL_ERROR_INVALID_VALUE;
}

}  // namespace tl
