// The row-walking recovery's work list: every row of every column once, at most
// the CTAs the device holds, whole CTAs, neighbouring columns in a CTA, and a
// handful of allocations (a moving mesh builds one at every change of its blocks).
#include <cstdio>
#include <cstdlib>
#include <new>
#include <random>

#include "knc_runs.h"

static size_t allocations = 0;
void* operator new(size_t n) {
    ++allocations;
    if (void* p = std::malloc(n ? n : 1)) return p;
    throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }

using Shapes = std::vector<std::pair<int64_t, int64_t>>;
constexpr int WPC = knc::TILE_THREADS / 32;

static int check(const char* name, const Shapes& shapes, int64_t ctas) {
    allocations = 0;
    const knc::RecoveryRuns r = knc::recovery_runs(shapes, ctas);
    const size_t made = allocations;
    const int64_t warps = (int64_t)r.off.size() - 1;
    if (warps % WPC || warps / WPC > std::max<int64_t>(ctas, 2)) return std::printf("FAIL %s: %ld warps\n", name, (long)warps);
    if (made > 64) return std::printf("FAIL %s: %zu allocations\n", name, made);
    std::vector<std::vector<char>> seen;
    for (const auto& s : shapes) seen.emplace_back((size_t)(s.first * ((s.second + 31) / 32)), 0);
    if (r.off.front() != 0 || r.off.back() != (int)r.runs.size()) return std::printf("FAIL %s: offsets\n", name);
    for (int64_t k = 0; k < warps; ++k) {
        if (r.off[k] > r.off[k + 1]) return std::printf("FAIL %s: offsets\n", name);
        for (int p = r.off[k]; p < r.off[k + 1]; ++p) {
            const int4 t = r.runs[p];
            const auto& s = shapes[t.x];
            if (t.w < 1 || t.y < 0 || t.y + t.w > s.first || t.z % 32 || t.z < 0 || t.z >= s.second)
                return std::printf("FAIL %s: run outside its block\n", name);
            for (int i = t.y; i < t.y + t.w; ++i)
                if (seen[t.x][(size_t)i * ((s.second + 31) / 32) + t.z / 32]++) return std::printf("FAIL %s: row twice\n", name);
            // a block whose columns fill CTAs: the CTA's first warp walks the same rows w columns before
            if (((s.second + 31) / 32) % WPC == 0) {
                const int4 f = r.runs[r.off[k - k % WPC] + (p - r.off[k])];
                if (f.x != t.x || f.y != t.y || f.w != t.w || f.z + 32 * (k % WPC) != t.z)
                    return std::printf("FAIL %s: not neighbours\n", name);
            }
        }
    }
    for (const auto& b : seen)
        for (char c : b)
            if (!c) return std::printf("FAIL %s: row missing\n", name);
    return 0;
}

int main() {
    int bad = 0;
    bad += check("none", {}, 456) != 0;
    bad += check("one zone", {{1, 1}}, 456) != 0;
    bad += check("wind", Shapes(64, {64, 1024}), 456) != 0;
    bad += check("jet", Shapes(32, {64, 512}), 456) != 0;
    bad += check("ragged", Shapes(7, {37, 93}), 456) != 0;
    bad += check("polar 97", Shapes(90, {13, 97}), 456) != 0;
    std::mt19937 g(3);
    for (int n = 0; n < 300; ++n) {
        Shapes s;
        const int blocks = 1 + (int)(g() % 96);
        for (int k = 0; k < blocks; ++k) {
            static const int nrs[] = {1, 4, 32, 64, 128, 256, 512}, nqs[] = {1, 16, 64, 97, 128, 256, 300, 512, 1024};
            s.push_back({nrs[g() % 7], nqs[g() % 9]});
        }
        bad += check("drawn", s, n % 3 ? 456 : 1 + (int)(g() % 8)) != 0;
    }
    std::printf(bad ? "%d failed\n" : "ok\n", bad);
    return bad != 0;
}
