// Reverse permutations (layout -> sorted order) and the schedule they share
// with the forward permutation (permute.cu, unpermute.cu).
#pragma once

#include <algorithm>

#include "btree_order.h"
#include "btree_plan.cuh"
#include "bulk.cuh"
#include "mveb_plan.cuh"

namespace tl {

// A permutation's schedule: its tiles and their order, which keys go through
// scratch, and the workspace regions.  The reverse permutation runs the same
// schedule backwards.
struct PermutePlan {
    int layout = 0;
    uint32_t key_bytes = 8;
    uint64_t n = 0, b = 1;
    uint64_t tile_keys = 0, ntiles = 0, scratch_keys = 0;
    bool ordered = false;  // B-tree plan O, with these tables (host, then device pointers)
    OrderTables ot;
    BtreeStream bs;
    MvebParams mp;
    uint64_t off_flags = 0, off_ctrl = 0, bytes = 0;
};

// The plan a permutation takes by default: the ordered schedule where it
// applies and its tables reach the device (its pointers are then device
// pointers), else the fixed directions.
int permute_plan_device(int layout, uint64_t n, uint64_t b, uint32_t key_bytes, cudaStream_t st, PermutePlan &pl);
// The plan with the fixed directions, which needs no tables.
int permute_plan_fixed(int layout, uint64_t n, uint64_t b, uint32_t key_bytes, PermutePlan &pl);
// Whether the default plan is on the ordered schedule, its tables permitting.
bool permute_takes_order(int layout, uint64_t n, uint64_t b, uint32_t key_bytes);
// The plan for a host replay: the ordered schedule wherever there is one (its
// tables in ov), or the fixed directions.
int permute_plan_replay(int layout, uint64_t n, uint64_t b, uint32_t key_bytes, bool ordered, OrderVectors &ov,
                        PermutePlan &pl);

// Arrays of up to kKeysBytes in a B-tree or BST layout are moved key by key
// through a copy, either way: two launches, no tiles, no waits.  False (rc 0)
// when the layout or the size asks for a plan; the argument checks are make_plan's.
// Measured on B200, one call's wall time by tiles / key by key (us): 2^10 to 2^17
// keys 50 to 66 / 18 to 22, BST of 2^20 - 1 u64 61 / 26, b = 16 3 * 2^18 u64 68 / 29, b =
// 2 2^21 u32 76 / 37; back from the layout 23 to 40 / 18 to 37 (from a copy tile by
// tile).  At 16 MB both ways are even for narrow nodes.
constexpr uint64_t kKeysBytes = 12ull << 20;
struct KeysGeometry {
    BtreeGeom g;
    FastDiv64 fd;
};
bool permute_by_keys(int layout, uint64_t n, uint64_t b, uint32_t key_bytes, KeysGeometry &kg);

// One copy range for the bulk engine: its 16-byte-aligned interior in
// kBulkChunk pieces, its ragged keys apart.  The scratch shares A's offset
// within 16 bytes at both range bases, so the interiors line up.
template <typename K>
int add_bulk_range(const K *A, const K *scr, const CopyRange &r, BulkPlan &P) {
    if (P.nr == kMaxBulkRanges) return TL_ERROR_UNSUPPORTED;
    const uintptr_t da = reinterpret_cast<uintptr_t>(A + r.dst), sa = reinterpret_cast<uintptr_t>(scr + r.src);
    if ((da ^ sa) & 15) return TL_ERROR_INVALID_VALUE;
    BulkRange R{};
    R.key_dst = r.dst;
    R.key_src = r.src;
    R.len = r.len;
    const uint64_t head = std::min<uint64_t>(((16 - (da & 15)) & 15) / sizeof(K), r.len);
    const uint64_t body = ((r.len - head) * sizeof(K)) & ~15ull;
    R.head = (uint32_t)head;
    R.tail = (uint32_t)(r.len - head - body / sizeof(K));
    R.dst = (r.dst + head) * sizeof(K);
    R.src = (r.src + head) * sizeof(K);
    R.bytes = body;
    R.chunk0 = P.nchunks;
    P.nchunks += (body + kBulkChunk - 1) / kBulkChunk;
    P.r[P.nr++] = R;
    return TL_SUCCESS;
}

// The copy ranges of a plan: per level (plans R, L), or the runs of whole
// scratch tiles (plan O: tiles [x, y) from scratch slot z on).
template <typename K>
int make_bulk_plan(const BtreeStream &S, const OrderTables &ot, const K *A, const K *scr, BulkPlan &P) {
    P.nr = 0;
    P.nchunks = 0;
    if (S.plan == PLAN_O) {
        for (uint64_t i = 0; i < ot.nranges; ++i) {
            const uint64_t u0 = ot.ranges[i].x, u1 = ot.ranges[i].y;
            const uint64_t d0 = u0 << S.tile_shift, d1 = std::min<uint64_t>(u1 << S.tile_shift, S.g.n);
            const uint64_t s0 = (uint64_t)ot.ranges[i].z << S.tile_shift;  // host data: S.tab may be device memory
            const int rc = add_bulk_range(A, scr, CopyRange{d0, s0, d1 - d0}, P);
            if (rc) return rc;
        }
        return TL_SUCCESS;
    }
    for (int j = 0; j < btree_copy_range_count(S); ++j) {
        CopyRange r;
        if (!btree_copy_range(S, j, r)) continue;
        const int rc = add_bulk_range(A, scr, r, P);
        if (rc) return rc;
    }
    return TL_SUCCESS;
}

int unpermute(int layout, void *dev_A, uint64_t n, uint64_t b, uint32_t key_bytes, void *dev_ws, uint64_t ws_bytes,
              cudaStream_t st, float *ms);
int unpermute_workspace_bytes(int layout, uint64_t n, uint64_t b, uint32_t key_bytes, uint64_t *bytes);
int emulate_unpermute(int layout, uint64_t n, uint64_t b, uint64_t *A);

}  // namespace tl
