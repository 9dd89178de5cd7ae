// BranchHeap::fill against pushing the same value key by key: the two heaps
// must then answer the same random operations alike, ties included (keys out
// of range and listed twice among them).  Usage: heap_fill seed capacity
#include "branch_heap.hpp"

#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

int main(int argc, char** argv) {
    if (argc != 3) return 2;
    std::mt19937_64 rng((unsigned)std::atoi(argv[1]));
    const long cap = std::atol(argv[2]);
    long bad = 0;
    for (int round = 0; round < 200; ++round) {
        std::vector<int> keys;
        const long count = (long)(rng() % (unsigned long)(cap + 2));
        for (long i = 0; i < count; ++i) keys.push_back(round % 2 ? (int)i - 1 : (int)(rng() % (unsigned long)(cap + 2)) - 1);
        const double value = round % 3 ? std::numeric_limits<double>::infinity() : 2.0;
        pgc::BranchHeap a(cap), b(cap);
        a.fill(value, keys);
        for (const int k : keys) b.push(value, k);
        for (long op = 0; op < 4 * cap + 8; ++op) {
            const long key = (long)(rng() % (unsigned long)(cap + 2)) - 1;
            const double v = (double)(rng() % 4) * 0.5;
            switch (rng() % 4) {
                case 0: a.push(v, key); b.push(v, key); break;
                case 1: bad += a.decrease(key, v) != b.decrease(key, v); break;
                case 2: bad += a.pop() != b.pop(); break;
                default: bad += a.peakKey(key) != b.peakKey(key); break;
            }
            bad += a.getSize() != b.getSize() || a.peak() != b.peak();
        }
        while (!a.isEmpty() || !b.isEmpty())
            if (a.pop() != b.pop()) {
                ++bad;
                break;
            }
    }
    std::printf("%ld differ\n", bad);
    return bad ? 1 : 0;
}
