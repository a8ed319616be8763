// Host check of the item walk (proto_b200/csrc/pb_walk.cuh): the reciprocal division against the division,
// and items against the cells they stand for, up to more than 2^32 of them.
#include <cstdio>
#include <random>
#include <vector>

#include "proto_b200/csrc/pb_walk.cuh"

namespace pb {
int cached_sm_count() { return 148; }
void set_cuda_error(cudaError_t) {}
}
using namespace pb;

static int failures = 0;
static void check(bool ok, const char* what, unsigned long long a, unsigned long long b)
{
    if (!ok && failures++ < 10) printf("%s: %llu %llu\n", what, a, b);
}

int main()
{
    std::mt19937_64 rng(1);
    std::vector<unsigned> ds = {1, 2, 3, 5, 6, 7, 9, 10, 31, 32, 33, 641, 65535, 65536, 65537, 0x7fffffffu};
    for (int k = 0; k < 300; k++) ds.push_back(1 + (unsigned)(rng() >> (33 + rng() % 30)));
    for (unsigned d : ds) {
        const FastDiv f = fast_div(d);
        std::vector<unsigned> ns = {0u, 1u, d - 1, d, d + 1, 0x7fffffffu, 0x80000000u, 0xfffffffeu, 0xffffffffu};
        for (int k = 0; k < 200; k++) {
            const unsigned q = (unsigned)(rng() % (0xffffffffull / d + 1));
            ns.push_back(q * d);
            ns.push_back(q * d - 1);
            ns.push_back((unsigned)rng());
        }
        for (unsigned n : ns) check(quotient(n, f) == n / d, "quotient", n, d);
    }
    // every cell once, items x fastest, whatever the shape and the planes of an item
    const int shapes[][3] = {{1, 1, 1}, {5, 1, 1}, {1, 7, 1}, {1, 1, 9}, {33, 2, 3}, {3, 33, 2}, {2, 3, 33}, {8, 8, 8}, {17, 5, 7}};
    for (auto& s : shapes)
        for (int planes : {1, 4, 8}) {
            const Walk w = walk_of(Region{{-3, 4, 9}, {s[0], s[1], s[2]}}, planes);
            std::vector<int> seen(s[0] * s[1] * s[2], 0);
            for (long long i = 0; i < w.items; i++) {
                int x, y, g;
                walk_item(w, i, x, y, g);
                check(x >= 0 && x < s[0] && y >= 0 && y < s[1] && g * planes < s[2], "item in range", i, planes);
                for (int z = g * planes; z < s[2] && z < (g + 1) * planes; z++) seen[x + s[0] * (y + s[1] * z)]++;
            }
            for (int c : seen) check(c == 1, "cell count", c, planes);
            check(walk_grid(w, 3).x == (w.items + kWalkThreads - 1) / kWalkThreads, "grid", w.items, 0);
        }
    // about and above 2^32 items
    const int big[][3] = {{65536, 65535, 4}, {65536, 65536, 4}, {65537, 65536, 9}, {2147483647, 3, 1}, {1, 1, 2147483647}};
    for (auto& s : big)
        for (int planes : {1, 4}) {
            const Walk w = walk_of(Region{{0, 0, 0}, {s[0], s[1], s[2]}}, planes);
            for (int k = 0; k < 1000; k++) {
                const long long i = k == 0 ? 0 : k == 1 ? w.items - 1 : (long long)(rng() % (unsigned long long)w.items);
                int x, y, g;
                walk_item(w, i, x, y, g);
                check(x + (long long)s[0] * (y + (long long)s[1] * g) == i && x < s[0] && y < s[1], "large item", i, planes);
            }
        }
    // an empty region has no item
    check(walk_of(Region{{0, 0, 0}, {0, 0, 0}}).items == 0, "empty", 0, 0);
    // thin boxes turn once; single cells up to two blocks per SM
    Region r{{0, 0, 0}, {9, 50, 1}};
    FieldView<int> v{nullptr, 9, 450};
    check(turn_thin(r, v) && r.n[1] == 1 && r.n[2] == 50 && v.sy == 450 && v.sz == 9, "turned", r.n[1], r.n[2]);
    check(!turn_thin(r, v) && walk_spread(r).planes == 1, "turned again", r.n[1], r.n[2]);
    check(walk_spread(Region{{0, 0, 0}, {64, 64, 64}}).planes == kWalkZ, "solid", 0, 0);
    printf("failures %d\n", failures);
    return failures != 0;
}
