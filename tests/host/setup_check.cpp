// The LOR setup's division and its TOF values.
//   division N SEED      div_exact against the host's division over N random operands: "cases differing"
//   tof FILE grid size nsigma   slab weights of the file's LORs (n x 7 floats): "LORs slabs nan nonzero"
#include <cstdio>
#include <cstdlib>
#include <random>
#include <string>
#include <vector>
using namespace srf;

template <bool QDIV>
static void weights(const std::vector<float> &lors, const Grid &g, const TofParams &tp) {
    long n = 0, slabs = 0, nan = 0, nonzero = 0;
    const int64_t sx[3] = {1, g.nx, (int64_t)g.nx * g.ny}, sy[3] = {g.ny, 1, (int64_t)g.nx * g.ny};
    const GridK k = make_gridk<true>(g, tp);
    for (size_t i = 0; 7 * i < lors.size(); ++i) {
        const float *l = &lors[7 * i];
        const LeanRec E = make_lean<true, 32>(setup_rec<true>(l, l[6], 1.0f, g, k), g, k, sx, sy, true, 128);
        ++n;
        if (!(E.flags & F_VALID)) continue;
        for (int lane = 0; lane < 32; ++lane)
            lean_walk<true, 4, 32, QDIV>(E, lean_axes(E, g), E.lo, E.hi, lane, [&](auto &, auto &w, auto ng) {
                for (int u = 0; u < decltype(ng)::value; ++u)
                    for (int s = 0; s < 3; ++s) {
                        ++slabs;
                        nan += w[u][s] != w[u][s];
                        nonzero += w[u][s] == w[u][s] && w[u][s] != 0.0f;
                    }
            });
    }
    printf("%ld %ld %ld %ld\n", n, slabs, nan, nonzero);
}

int main(int, char **v) {
    if (std::string(v[1]) == "division") {
        std::mt19937_64 rng(atoi(v[3]));
        std::uniform_real_distribution<float> mant(1.0f, 2.0f);
        std::uniform_int_distribution<int> ex(-40, 40), one(0, 15);
        const long n = atol(v[2]);
        long differ = 0;
        for (long i = 0; i < n; ++i) {
            float a = std::ldexp(mant(rng), ex(rng)), b = std::ldexp(mant(rng), ex(rng));
            if (rng() & 1) a = -a;
            if (rng() & 1) b = -b;
            const int kind = one(rng);
            if (kind == 0) a = 0.0f;
            if (kind == 1) b = 1.0f;
            if (kind == 2) a = std::nextafterf(b, INFINITY);
            if (kind == 3) b = std::ldexp(std::nextafterf(2.0f, 0.0f), ex(rng));
            differ += !(div_exact(a, b, 1.0f / b) == a / b);
        }
        printf("%ld %ld\n", n, differ);
        return 0;
    }
    std::vector<float> lors;
    FILE *f = fopen(v[2], "rb");
    float row[7];
    while (f && fread(row, 4, 7, f) == 7) lors.insert(lors.end(), row, row + 7);
    const Grid g{atoi(v[3]), atoi(v[4]), atoi(v[5]), 0, 0, 0, (float)atof(v[6]), (float)atof(v[7]), (float)atof(v[8])};
    const TofParams tp{3.66f, 1138.0f, (float)atof(v[9])};
    if (grid_qdiv(g)) weights<true>(lors, g, tp);
    else weights<false>(lors, g, tp);
    return 0;
}
