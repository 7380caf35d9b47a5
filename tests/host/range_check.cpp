// Offsets of the slots that a traversal visits (non-zero weight) outside the image, over the walks and, for
// LORs that are whole interior chunks, the untested form of the fused step: "LORs visits outside".
#include <cstdio>
#include <cstdlib>
#include <vector>
using namespace srf;

template <bool QDIV>
static void check(const std::vector<float> &lors, const Grid &g) {
    long n = 0, visits = 0, outside = 0;
    const int64_t v = (int64_t)g.nx * g.ny * g.nz, sx[3] = {1, g.nx, (int64_t)g.nx * g.ny}, sy[3] = {g.ny, 1, (int64_t)g.nx * g.ny};
    const GridK k = make_gridk<false>(g, TofParams{0, 0, 0});
    for (size_t i = 0; 6 * i < lors.size(); ++i) {
        const LeanRec E = make_lean<false, 32>(setup_rec<false>(&lors[6 * i], 0.0f, 1.0f, g, k), g, k, sx, sy, true, 128);
        if (!(E.flags & F_VALID) || (E.flags & F_TIE)) continue;
        ++n;
        auto slot = [&](const int32_t *o, const float *w) {
            for (int s = 0; s < 3; ++s)
                if (w[s] != 0.0f) { ++visits; outside += o[s] < 0 || o[s] >= v; }
        };
        for (int lane = 0; lane < 32; ++lane) {
            lean_walk<false, 4, 32, QDIV>(E, lean_axes(E, g), E.lo, E.hi, lane, [&](auto &o, auto &w, auto ng) {
                for (int u = 0; u < decltype(ng)::value; ++u) slot(o[u], w[u]);
            });
            if (E.flags & F_HOT)
                for (int ip = E.lo; ip <= E.hi; ip += 32) {
                    int32_t o[1][3];
                    float w[1][3];
                    interior_groups<false, 32, QDIV, 1>(E, ip, E.hi, lane, o, w);
                    slot(o[0], w[0]);
                }
        }
    }
    printf("%ld %ld %ld\n", n, visits, outside);
}

// argv: file of n x 6 floats, grid, size
int main(int, char **v) {
    std::vector<float> lors;
    FILE *f = fopen(v[1], "rb");
    float row[6];
    while (f && fread(row, 4, 6, f) == 6) lors.insert(lors.end(), row, row + 6);
    const Grid g{atoi(v[2]), atoi(v[3]), atoi(v[4]), 0, 0, 0, (float)atof(v[5]), (float)atof(v[6]), (float)atof(v[7])};
    if (grid_qdiv(g)) check<true>(lors, g);
    else check<false>(lors, g);
    return 0;
}
