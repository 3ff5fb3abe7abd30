// near_plan.h -- which nodes of a case step in passes of several steps.
#pragma once
#include <vector_types.h>

#include <algorithm>
#include <cstdint>
#include <cstdlib>
#include <vector>

namespace lbm {

// A case's nodes near special ones in passes of `lv` steps (Solver::near_plan):
// deep, a word per strip and row, a bit per pair whose nodes are both lv or more
// away from every special node; segs[q], the clean pairs that step q of a pass
// takes one step at a time, as (0, row, first column, a bit per pair of 64 columns).
struct NearPlan {
    int lv = 0;
    std::vector<uint32_t> deep;
    std::vector<std::vector<int4>> segs;
    long long near_pairs = 0;
};

// Bit l of the result: bit 2 l or 2 l + 1 of x (a pair with either node).
inline uint32_t pair_bits(uint64_t x) {
    x = (x | x >> 1) & 0x5555555555555555ull;
    x = (x | x >> 1) & 0x3333333333333333ull;
    x = (x | x >> 2) & 0x0F0F0F0F0F0F0F0Full;
    x = (x | x >> 4) & 0x00FF00FF00FF00FFull;
    x = (x | x >> 8) & 0x0000FFFF0000FFFFull;
    return (uint32_t)(x | x >> 16);
}

// special: the nodes (x & colmask, y), rows ascending, columns ascending in a
// row, whole pairs; halo: columns a strip of 64 gives up on either side. Distance:
// the larger of |dx|, |dy|, wrapped on periodic axes.
// Step q + 1 of the list needs the nodes within 2 lv - (q + 1) of a special one,
// the last every pair that is not deep. Each special row is widened along x into
// words of 64 nodes for each of those distances; a row of the plan gathers the
// words of the 2 (2 lv - 1) + 1 rows around it. So the work goes with the special
// nodes, not with the grid: 4096^2 cavity 25 ms with a byte per node, 3.4 ms this
// way (x86 core).
inline NearPlan make_near_plan(int Nx, int Ny, bool px, bool py, const std::vector<int2> &special, int colmask, int lv,
                               int halo) {
    constexpr int kMaxLevels = 4;
    NearPlan plan;
    plan.lv = lv;
    const int m = 2 * lv - 1, W = (Nx + 63) / 64;
    int radius[kMaxLevels];  // of step q's nodes
    for (int q = 0; q < lv; q++) radius[q] = q == lv - 1 ? lv - 1 : m - q;

    struct Words {
        int w;
        uint64_t self, wide[kMaxLevels];
    };
    std::vector<Words> words;
    std::vector<size_t> first((size_t)Ny + 1, 0);
    std::vector<uint64_t> ext((size_t)W + 3, 0);  // columns -64 .. of one row, with what wraps to the other end
    std::vector<int> hit;
    size_t n = 0;
    for (int j = 0; j < Ny; j++) {
        first[j] = words.size();
        hit.clear();
        auto set = [&](int col) {
            const int k = col + 64;
            ext[k >> 6] |= 1ull << (k & 63);
            if (hit.empty() || hit.back() != k >> 6) hit.push_back(k >> 6);
        };
        for (; n < special.size() && special[n].y == j; n++) {
            const int c = special[n].x & colmask;
            set(c);
            if (px && c >= Nx - m) set(c - Nx);
            if (px && c < m) set(c + Nx);
        }
        if (hit.empty()) continue;
        const size_t set_words = hit.size();
        for (size_t h = 0; h < set_words; h++) {
            const int e = hit[h];
            hit.push_back(e - 1);
            hit.push_back(e + 1);
        }
        std::sort(hit.begin(), hit.end());
        hit.erase(std::unique(hit.begin(), hit.end()), hit.end());
        for (int e : hit) {
            if (e < 1 || e > W) continue;
            const uint64_t a = ext[e - 1], b = ext[e], c = ext[e + 1];
            const uint64_t in = e == W && Nx % 64 ? (1ull << Nx % 64) - 1 : ~0ull;
            Words t;
            t.w = e - 1;
            t.self = b & in;
            uint64_t o = b;
            for (int s = 1; s <= m; s++) {
                o |= b << s | a >> (64 - s) | b >> s | c << (64 - s);
                for (int q = 0; q < lv; q++)
                    if (radius[q] == s) t.wide[q] = o & in;
            }
            if (o & in) words.push_back(t);
        }
        for (int e : hit)
            if (e >= 0 && e < W + 3) ext[e] = 0;
    }
    first[Ny] = words.size();

    // Every pair of the grid is deep, then the near ones are taken out.
    const int width = 64 - 2 * halo, strips = (Nx + width - 1) / width;
    plan.deep.resize((size_t)strips * Ny);
    for (int st = 0; st < strips; st++) {
        uint32_t all = 0;
        for (int c = 0; c < width && st * width + c + 1 < Nx; c += 2) all |= 1u << ((c + halo) / 2);
        std::fill(plan.deep.begin() + (size_t)st * Ny, plan.deep.begin() + (size_t)(st + 1) * Ny, all);
    }
    plan.segs.assign(lv, std::vector<int4>());
    std::vector<uint64_t> self((size_t)W, 0), wide((size_t)W * lv, 0);
    std::vector<uint8_t> seen((size_t)W, 0);
    for (int j = 0; j < Ny; j++) {
        hit.clear();
        for (int dy = -m; dy <= m; dy++) {
            int y = j + dy;
            if (py) y = (y + Ny) % Ny;
            if (y < 0 || y >= Ny) continue;
            for (size_t k = first[y]; k < first[y + 1]; k++) {
                const Words &t = words[k];
                if (!seen[t.w]) {
                    seen[t.w] = 1;
                    hit.push_back(t.w);
                }
                if (dy == 0) self[t.w] |= t.self;
                for (int q = 0; q < lv; q++)
                    if (std::abs(dy) <= radius[q]) wide[(size_t)t.w * lv + q] |= t.wide[q];
            }
        }
        std::sort(hit.begin(), hit.end());
        for (int w : hit) {
            const int cols = std::min(64, Nx - 64 * w);  // an odd last column is special and no pair
            const uint32_t whole = cols / 2 == 32 ? ~0u : (1u << cols / 2) - 1u;
            const uint32_t sp = pair_bits(self[w]);
            for (int q = 0; q < lv; q++) {
                const uint32_t all = pair_bits(wide[(size_t)w * lv + q]) & whole, mask = all & ~sp;
                wide[(size_t)w * lv + q] = 0;
                if (mask) {
                    plan.segs[q].push_back(int4{0, j, 64 * w, (int)mask});
                    plan.near_pairs += __builtin_popcount(mask);
                }
                if (q == lv - 1)
                    for (uint32_t left = all; left; left &= left - 1) {
                        const int i = 64 * w + 2 * __builtin_ctz(left);
                        plan.deep[(size_t)(i / width) * Ny + j] &= ~(1u << ((i % width + halo) / 2));
                    }
            }
            self[w] = 0;
            seen[w] = 0;
        }
    }
    return plan;
}

}  // namespace lbm
