// st_treecheck.h — what a tree in the reference's node layout must hold before a walk may use it, node by
// node (the device's check of a newly built TLAS, tlas_check_kernel).  Plain code for the host too.
#pragma once
#include <cstdint>
#include "slimtracin_types.h"

#ifdef __CUDACC__
#define ST_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define ST_HOST_DEVICE inline
#endif

namespace st {

constexpr uint32_t kClaimsNone = 0xFFFFFFFFu;

// The pair of children (pair k: nodes 1 + 2k and 2 + 2k) that a node claims, below n.
ST_HOST_DEVICE uint32_t claimed_pair(const BVHNode &nd, uint32_t n) {
    const uint32_t f = nd.first_child_id;
    return !nd.child_count && f && (f - 1) / 2 < n ? (f - 1) / 2 : kClaimsNone;
}

// Node i of `count` (at most 2n - 1) over n items: its children pair lies inside the array and is its own,
// or its items do; and it reaches the root by at most `stack` - 2 parents.  parent_of_pair: for every pair
// that some node claims, one that does (n words; the others are not looked at for what they hold).
ST_HOST_DEVICE bool tree_node_ok(const BVHNode *nodes, uint32_t count, uint32_t n, const uint32_t *parent_of_pair, uint32_t stack,
                                 uint32_t i) {
    const uint32_t f = nodes[i].first_child_id, c = nodes[i].child_count;
    bool ok = c ? (uint64_t)f + c <= n : (f & 1u) && (uint64_t)f + 1 < count && parent_of_pair[(f - 1) / 2] == i;
    uint32_t steps = 0;
    for (uint32_t at = i; at && ok; steps++) {
        const uint32_t pair = (at - 1) / 2, p = parent_of_pair[pair];
        ok = steps + 2 < stack && p < count && !nodes[p].child_count && nodes[p].first_child_id == 1 + 2 * pair;
        at = p;
    }
    return ok;
}

}  // namespace st
