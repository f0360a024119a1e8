// tree_node_ok (csrc/st_treecheck.h) over arrays read from standard input, as tlas_finish_kernel and
// tlas_check_kernel go over them; one line each.  A case: n, the pairs the build reports, 2n nodes, and n
// words for what parent_of_pair held before.
#include <cstdio>
#include <vector>
#include "st_treecheck.h"

using namespace st;

int main() {
    uint32_t head[2];
    while (fread(head, 4, 2, stdin) == 2) {
        const uint32_t n = head[0], most = head[1] < n - 1 ? head[1] : n - 1, count = 1 + 2 * most;
        std::vector<BVHNode> all(2 * n);
        std::vector<uint32_t> before(n);
        if (fread(all.data(), sizeof(BVHNode), 2 * n, stdin) != 2 * n || fread(before.data(), 4, n, stdin) != n) return 1;
        const std::vector<BVHNode> nodes(all.begin(), all.begin() + count);     // (nothing beyond is to be read)
        bool ok[2];
        for (int order = 0; order < 2; order++) {      // of several nodes that claim a pair, any may win
            std::vector<uint32_t> parent(before);
            for (uint32_t k = 0; k < count; k++) {
                const uint32_t i = order ? count - 1 - k : k, pair = claimed_pair(nodes[i], n);
                if (pair != kClaimsNone) parent[pair] = i;
            }
            ok[order] = head[1] < n;
            for (uint32_t i = 0; i < count; i++) ok[order] = tree_node_ok(nodes.data(), count, n, parent.data(), 64, i) && ok[order];
        }
        printf("%d%d\n", ok[0], ok[1]);
    }
    return 0;
}
