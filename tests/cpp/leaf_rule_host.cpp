// leaf_pays and leaf_load for the launches on standard input, one a line:
// transcendental, root words, node words, nodes, levels, dims...
#include "leaf_rule.h"

#include <cstdio>

int main() {
    unsigned trans, levels;
    unsigned long long root, words, nodes;
    while (std::scanf("%u %llu %llu %llu %u", &trans, &root, &words, &nodes, &levels) == 5) {
        uint32_t dims[8] = {};
        for (unsigned l = 0; l < levels; l++)
            if (std::scanf("%u", &dims[l]) != 1) return 1;
        const uint32_t d = dims[levels - 1];
        std::printf("%d %.3f\n", frep::leaf_pays(d, trans != 0, root, words, nodes * d * d * d) ? 1 : 0,
                    frep::leaf_load(dims, levels));
    }
}
