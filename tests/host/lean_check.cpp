// Walks LORs with the interior (packed, branch-free) slab code and holds every slab to the range-tested
// form: the same offsets and weights to the bit, offsets inside the image, every slab visited once.
#include <cstdio>
#include <cstdlib>
#include <vector>
using namespace srf;

struct Counts { long lors = 0, hot = 0, slabs = 0, outside = 0, differ = 0, missed = 0; };

template <bool TOF, bool QDIV, int G, int U>
static Counts check(const std::vector<float> &lors, const Grid &g, const TofParams &tp) {
    Counts c;
    const int64_t n = (int64_t)g.nx * g.ny * g.nz;
    const int64_t sx[3] = {1, g.nx, (int64_t)g.nx * g.ny}, sy[3] = {g.ny, 1, (int64_t)g.nx * g.ny};
    const GridK k = make_gridk<TOF>(g, tp);
    for (size_t i = 0; 7 * i < lors.size(); ++i) {
        const float *l = &lors[7 * i];
        const LeanRec E = make_lean<TOF, G>(setup_rec<TOF>(l, l[6], 1.0f, g, k), g, k, sx, sy, true, G * U);
        if (!(E.flags & F_VALID) || (E.flags & F_TIE)) continue;
        ++c.lors;
        const LeanAxes ax = lean_axes(E, g);
        std::vector<int> seen(E.hi + 1, 0);
        auto one = [&](int ip, const int32_t *o, const float *w) {
            int32_t eo[3];
            float ew[3];
            lean_slab<TOF, QDIV>(E, ax, std::min(ip, E.hi), ip <= E.hi, eo, ew);
            if (ip <= E.hi) ++seen[ip];
            ++c.slabs;
            for (int s = 0; s < 3; ++s) {
                if (w[s] != 0.0f && (o[s] < 0 || o[s] >= n)) ++c.outside;
                if (w[s] != ew[s] || (w[s] != 0.0f && o[s] != eo[s])) ++c.differ;
            }
        };
        for (int lane = 0; lane < G; ++lane) {
            if (E.flags & F_HOT) {
                const int ng = E.flags >> kHotShift;
                int32_t o[4][3];
                float w[4][3];
                if (ng == 4) interior_groups<TOF, G, QDIV, 4>(E, E.lo, E.hi, lane, o, w);
                else if (ng == 3) interior_groups<TOF, G, QDIV, 3>(E, E.lo, E.hi, lane, o, w);
                else if (ng == 2) interior_groups<TOF, G, QDIV, 2>(E, E.lo, E.hi, lane, o, w);
                else interior_groups<TOF, G, QDIV, 1>(E, E.lo, E.hi, lane, o, w);
                for (int u = 0; u < ng; ++u) one(E.lo + G * u + lane, o[u], w[u]);
                c.hot += lane == 0;
            } else {
                int at = E.lo;
                lean_walk<TOF, U, G, QDIV>(E, ax, E.lo, E.hi, lane, [&](auto &o, auto &w, auto ng) {
                    for (int u = 0; u < decltype(ng)::value; ++u) one(at + G * u + lane, o[u], w[u]);
                    at += G * decltype(ng)::value;
                });
            }
        }
        for (int ip = E.lo; ip <= E.hi; ++ip) c.missed += seen[ip] != 1;
    }
    return c;
}

// argv: file of n x 7 floats, grid, size, TOF (0 / 1), nsigma
int main(int, char **v) {
    std::vector<float> lors;
    FILE *f = fopen(v[1], "rb");
    float row[7];
    while (f && fread(row, 4, 7, f) == 7) lors.insert(lors.end(), row, row + 7);
    const Grid g{atoi(v[2]), atoi(v[3]), atoi(v[4]), 0, 0, 0, (float)atof(v[5]), (float)atof(v[6]), (float)atof(v[7])};
    const TofParams tp{3.66f, 1138.0f, (float)atof(v[9])};
    const bool tof = atoi(v[8]), qdiv = grid_qdiv(g);
    auto show = [](const Counts &c) { printf("%ld %ld %ld %ld %ld %ld\n", c.lors, c.hot, c.slabs, c.outside, c.differ, c.missed); };
#define SRF_RUN(G, U) show(tof ? (qdiv ? check<true, true, G, U>(lors, g, tp) : check<true, false, G, U>(lors, g, tp)) \
                              : (qdiv ? check<false, true, G, U>(lors, g, tp) : check<false, false, G, U>(lors, g, tp)))
    SRF_RUN(32, 4);
    SRF_RUN(32, 2);
    SRF_RUN(8, 4);
    return 0;
}
