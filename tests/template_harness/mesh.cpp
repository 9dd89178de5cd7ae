// Checks the mesh-ordered layer template and the ranges of teams on local
// tables: every node has one slot and every slot at most one node; each node's
// in-edge list holds the same template edges, in the same order and with the
// same sources, as in the template ordered by node ids; plan_even_cuts covers
// the slices in order and no range's work exceeds the best bound (an exact
// search over contiguous partitions).
// Usage: mesh EX.bin nVX conj prune nY
#include "graph_template.hpp"

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <vector>

namespace pgc {
void* host_buffer_alloc(size_t b) { return b ? std::malloc(b) : nullptr; }
void host_buffer_free(void* p) { std::free(p); }
}  // namespace pgc

using namespace pgc;

int main(int argc, char** argv) {
    if (argc != 6) return 2;
    std::vector<int> ex;
    FILE* f = std::fopen(argv[1], "rb");
    if (!f) return 2;
    int x;
    while (std::fread(&x, 4, 1, f) == 1) ex.push_back(x);
    std::fclose(f);
    const int nY = std::atoi(argv[5]);
    std::vector<int> ey;
    for (int i = 0; i < nY; ++i) ey.insert(ey.end(), {i, (i + 1) % nY});
    LayerTemplate A, B;
    const bool conj = std::atoi(argv[3]) != 0, prune = std::atoi(argv[4]) != 0;
    for (int m = 0; m < 2; ++m) {
        const std::string err = build_template(ex.data(), (int64_t)ex.size() / 2, ey.data(), nY, std::atoll(argv[2]),
                                               conj, prune, m ? B : A, m == 1);
        if (!err.empty()) {
            std::printf("error %s\n", err.c_str());
            return 1;
        }
    }
    long long bad = 0;
    auto fail = [&](const char* what, long long a, long long b) {
        if (++bad <= 10) std::printf("%s (%lld, %lld)\n", what, a, b);
    };
    if (A.n != B.n || A.eBlock != B.eBlock) fail("sizes", A.n, B.n);
    if ((long long)B.slotNode.size() != 32LL * B.nslices || (long long)B.nodeSlot.size() != B.n) fail("slots", 0, 0);
    long long held = 0;
    for (size_t s = 0; s < B.slotNode.size(); ++s)
        if (B.slotNode[s] >= 0) {
            ++held;
            if (B.nodeSlot[(size_t)B.slotNode[s]] != (int)s) fail("slot of node", B.slotNode[s], (long long)s);
        }
    if (held != B.n) fail("nodes with a slot", held, B.n);
    for (int p = 0; p < 2; ++p)
        for (int v = 0; v < A.n; ++v) {
            std::vector<int> la, lb;
            auto list = [&](const LayerTemplate& T, int slot, std::vector<int>& out) {
                for (int j = T.sp[p][(size_t)(slot >> 5)]; j < T.sp[p][(size_t)(slot >> 5) + 1]; ++j) {
                    const size_t at = (size_t)j * 32 + (size_t)(slot & 31);
                    if (T.tedge[p][at] < 0) {
                        if (T.src[p][at] != -1) fail("padding with a source", v, T.src[p][at]);
                        continue;
                    }
                    out.push_back(T.tedge[p][at]);
                    out.push_back(T.src[p][at]);
                }
            };
            list(A, v, la);
            list(B, B.nodeSlot[(size_t)v], lb);
            if (la != lb) fail("in-edges of node", p, v);
        }
    for (int K = 1; K <= 4; ++K)
        for (int blocks : {1, 2, 3, 5, 8}) {
            const std::vector<int> cut = plan_even_cuts(B, blocks, K);
            if ((int)cut.size() != blocks + 1 || cut.front() != 0 || cut.back() != B.nslices) fail("cut ends", K, blocks);
            // the plan's weights, restated
            const int reps = B.entries[INTRA] > 0 ? K - 1 : 0, nk = reps > 0 ? K : 1;
            std::vector<long long> w;
            for (int s = 0; s < B.nslices; ++s) {
                const int ri = B.sp[INTER][(size_t)s + 1] - B.sp[INTER][(size_t)s];
                const int ra = reps ? B.sp[INTRA][(size_t)s + 1] - B.sp[INTRA][(size_t)s] : 0;
                w.push_back((ri ? 30 + ri * (9LL + 6 * nk) : 0) + (ra ? reps * (30 + ra * 15LL) : 0) + 1);
            }
            long long worst = 0;
            for (int c = 0; c < blocks; ++c) {
                if (cut[(size_t)c + 1] < cut[(size_t)c]) fail("cut order", K, blocks);
                long long sum = 0;
                for (int s = cut[(size_t)c]; s < cut[(size_t)c + 1]; ++s) sum += w[(size_t)s];
                worst = std::max(worst, sum);
            }
            std::vector<long long> best((size_t)B.nslices + 1, 1LL << 60), next;
            best[0] = 0;
            for (int c = 0; c < blocks; ++c) {
                next.assign((size_t)B.nslices + 1, 1LL << 60);
                for (int e = 0; e <= B.nslices; ++e) {
                    long long sum = 0;
                    for (int b = e; b >= 0; --b) {
                        next[(size_t)e] = std::min(next[(size_t)e], std::max(best[(size_t)b], sum));
                        if (b > 0) sum += w[(size_t)b - 1];
                    }
                }
                best = next;
            }
            if (worst != best[(size_t)B.nslices]) fail("largest range", worst, best[(size_t)B.nslices]);
        }
    std::printf("bad %lld\n", bad);
    return bad ? 1 : 0;
}
