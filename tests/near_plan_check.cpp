// make_near_plan against the distances node by node. near_plan_check COUNT:
// that many random cases; prints "cases wrong", exit status 1 when one differs.
#include <cstdio>
#include <random>

#include "near_plan.h"

using namespace lbm;

// The plan by its definition.
static NearPlan plain(int Nx, int Ny, bool px, bool py, const std::vector<uint8_t> &sp, int lv, int halo) {
    const int m = 2 * lv - 1, width = 64 - 2 * halo, strips = (Nx + width - 1) / width;
    std::vector<int> dist((size_t)Nx * Ny, 1000);
    for (int y = 0; y < Ny; y++)
        for (int x = 0; x < Nx; x++) {
            if (!sp[(size_t)y * Nx + x]) continue;
            for (int dy = -m; dy <= m; dy++)
                for (int dx = -m; dx <= m; dx++) {
                    int i = x + dx, j = y + dy;
                    if (px) i = (i + Nx) % Nx;
                    if (py) j = (j + Ny) % Ny;
                    if (i < 0 || i >= Nx || j < 0 || j >= Ny) continue;
                    int &d = dist[(size_t)j * Nx + i];
                    d = std::min(d, std::max(std::abs(dx), std::abs(dy)));
                }
        }
    NearPlan p;
    p.lv = lv;
    p.deep.assign((size_t)strips * Ny, 0);
    p.segs.assign(lv, std::vector<int4>());
    for (int j = 0; j < Ny; j++)
        for (int s0 = 0; s0 < Nx; s0 += 64) {
            std::vector<uint32_t> mask(lv, 0);
            for (int l = 0; l < 32 && s0 + 2 * l + 1 < Nx; l++) {
                const int i = s0 + 2 * l, d = std::min(dist[(size_t)j * Nx + i], dist[(size_t)j * Nx + i + 1]);
                if (d >= lv) p.deep[(size_t)(i / width) * Ny + j] |= 1u << ((i % width + halo) / 2);
                if (d == 0) continue;
                for (int q = 0; q < lv; q++)
                    if (d < (q == lv - 1 ? lv : 2 * lv - q)) mask[q] |= 1u << l;
            }
            for (int q = 0; q < lv; q++)
                if (mask[q]) {
                    p.segs[q].push_back(int4{0, j, s0, (int)mask[q]});
                    p.near_pairs += __builtin_popcount(mask[q]);
                }
        }
    return p;
}

int main(int, char **argv) {
    std::mt19937 gen(3);
    long wrong = 0;
    const int count = std::atoi(argv[1]);
    for (int n = 0; n < count; n++) {
        auto pick = [&](int a, int b) { return a + (int)(gen() % (unsigned)(b - a + 1)); };
        const int Nx = pick(8, n % 3 ? 70 : 300), Ny = pick(8, 40), lv = n % 2 ? 4 : 2, halo = (lv + 1) / 2 * 2;
        const bool px = gen() & 1, py = gen() & 1;
        std::vector<uint8_t> sp((size_t)Nx * Ny, 0);
        for (int k = pick(0, 6); k > 0; k--) {  // nodes, walls, blocks
            const int x0 = pick(0, Nx - 1), y0 = pick(0, Ny - 1), kind = pick(0, 3);
            const int w = kind == 1 ? Nx : kind == 2 ? 1 : pick(1, 9), h = kind == 2 ? Ny : kind == 1 ? 1 : pick(1, 5);
            for (int y = y0; y < std::min(Ny, y0 + h); y++)
                for (int x = kind == 1 ? 0 : x0; x < std::min(Nx, x0 + w); x++) sp[(size_t)y * Nx + x] = 1;
        }
        std::vector<int2> list;
        for (int y = 0; y < Ny; y++)
            for (int x = 0; x < Nx; x += 2) {  // whole pairs, and an odd last column
                uint8_t *a = &sp[(size_t)y * Nx + x];
                if (x + 1 == Nx) a[0] = 1;
                else if (a[0] | a[1]) a[0] = a[1] = 1;
                if (!a[0]) continue;
                list.push_back(int2{x | (pick(0, 1) << 30), y});
                if (x + 1 < Nx) list.push_back(int2{x + 1, y});
            }
        const NearPlan a = make_near_plan(Nx, Ny, px, py, list, ~(1 << 30), lv, halo), b = plain(Nx, Ny, px, py, sp, lv, halo);
        bool same = a.lv == b.lv && a.deep == b.deep && a.near_pairs == b.near_pairs;
        for (int q = 0; q < lv; q++) {
            same = same && a.segs[q].size() == b.segs[q].size();
            for (size_t k = 0; same && k < a.segs[q].size(); k++) {
                const int4 x = a.segs[q][k], y = b.segs[q][k];
                same = x.x == y.x && x.y == y.y && x.z == y.z && x.w == y.w;
            }
        }
        if (!same && wrong++ < 5) std::printf("%d x %d, periodic %d %d, %d levels\n", Nx, Ny, px, py, lv);
    }
    std::printf("%d %ld\n", count, wrong);
    return wrong != 0;
}
