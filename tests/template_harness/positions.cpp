// Checks stream_positions between the template ordered by node ids and the
// mesh-ordered one, both ways: an entry with an edge finds the entry of the
// same template edge in the same part, an empty one finds none, and both
// templates' edges are all found.
// Usage: positions EX.bin nVX conj prune nY
#include "graph_template.hpp"

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
    std::vector<int> ex, ey;
    FILE* f = std::fopen(argv[1], "rb");
    if (!f) return 2;
    int x;
    while (std::fread(&x, 4, 1, f) == 1) ex.push_back(x);
    std::fclose(f);
    const int nY = std::atoi(argv[5]);
    for (int i = 0; i < nY; ++i) ey.insert(ey.end(), {i, (i + 1) % nY});
    LayerTemplate T[2];
    for (int m = 0; m < 2; ++m)
        if (!build_template(ex.data(), (int64_t)ex.size() / 2, ey.data(), nY, std::atoll(argv[2]), argv[3][0] == '1',
                            argv[4][0] == '1', T[m], m == 1).empty())
            return 2;
    // template edge of an entry of a layer's streams, -2 outside them
    auto edge = [](const LayerTemplate& t, int64_t i) {
        if (i < 0 || i >= t.layerStride()) return -2;
        return i < t.entries[INTER] ? t.tedge[INTER][(size_t)i] : t.tedge[INTRA][(size_t)(i - t.entries[INTER])];
    };
    long long bad = 0, held = 0;
    for (int m = 0; m < 2; ++m) {
        const LayerTemplate &from = T[m], &to = T[1 - m];
        const std::vector<int> at = stream_positions(from, to);
        bad += (int64_t)at.size() != to.layerStride();
        for (int64_t i = 0; i < to.layerStride() && i < (int64_t)at.size(); ++i) {
            const int t = edge(to, i);
            if (t < 0) {
                bad += at[(size_t)i] != -1;
                continue;
            }
            ++held;
            bad += edge(from, at[(size_t)i]) != t;
            bad += (i < to.entries[INTER]) != (at[(size_t)i] < from.entries[INTER]);
        }
    }
    bad += held != T[0].eBlock + T[1].eBlock;
    std::printf("bad %lld\n", bad);
    return bad ? 1 : 0;
}
