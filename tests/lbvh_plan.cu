// Prints, for each triangle count given, the layout of a tree that steps and queries walk
// and of one that is only read out: bytes in all, buckets of the bucket sort, bytes of
// its slots and whether they overlap the nodes or leaves.
#include <cstdio>
#include <cstdlib>

#include "visg_internal.cuh"

int main(int argc, char** argv) {
    for (int k = 1; k < argc; ++k)
        for (int walked = 0; walked < 2; ++walked) {
            const int nt = std::atoi(argv[k]);
            visg::BvhBuffers b;
            visg::Arena a;
            b.plan(a, VISG_NOALLOC_MAX_VERTICES, nt, true, walked != 0);
            size_t at = 4096, slots = 0;  // as the arena lays the arrays out, from some address
            for (auto& w : a.plan) {
                *w.first = reinterpret_cast<void*>(at);
                if (w.first == (void**)&b.bslot) slots = w.second;
                at += w.second;
            }
            const size_t s0 = (size_t)b.bslot, s1 = s0 + slots, n0 = (size_t)b.nodes, l0 = (size_t)b.leaves;
            const size_t n1 = n0 + sizeof(visg::Node) * (size_t)(nt > 1 ? nt - 1 : 1), l1 = l0 + 32 * (size_t)nt;
            const int over = slots && ((s0 < n1 && n0 < s1) || (s0 < l1 && l0 < s1));
            std::printf("%d %d %zu %d %zu %d\n", nt, walked, at - 4096, b.buckets, slots, over);
        }
}
