// Runs the traversal's scatter lane by lane on the host and holds what it adds to the slabs' own visits:
// one addition of value * weight for every slot of non-zero weight, none for any other slot, none outside
// the image, whatever the value (1, infinite, NaN).
#include <cstdio>
#include <cstdlib>
#include <utility>
#include <vector>
using namespace srf;

struct Slots { int32_t o[3]; float w[3]; };
typedef std::vector<std::pair<int64_t, uint32_t>> Adds;

static uint32_t bits_of(float v) { return v != v ? 0x7fc00000u : (uint32_t)__float_as_int(v); }

struct Counts { long lors = 0, adds = 0, unvisited = 0, outside = 0, differ = 0; };

// One scatter call of a group: lane l's slots in at[l]. First pass: each lane's shuffle arguments; second
// pass: what it adds.
template <int G>
static void scatter_group(const std::vector<Slots> &at, float r, int64_t n, float *im, Counts &c) {
    lanes.args.assign(G, {});
    lanes.record = true;
    for (int pass = 0; pass < 2; ++pass, lanes.record = false)
        for (int l = 0; l < G; ++l) {
            lanes.lane = l;
            lanes.next = 0;
            lanes.adds.clear();
            int32_t o[1][3];
            float w[1][3];
            std::memcpy(o, at[l].o, sizeof(o));
            std::memcpy(w, at[l].w, sizeof(w));
            scatter_slots<G, 1>(im, o, w, r, l);
            if (pass)
                for (auto &a : lanes.adds) lanes.all.push_back({a.first - im, bits_of(a.second)});
        }
    Adds want;
    for (auto &s : at)
        for (int k = 0; k < 3; ++k) {
            if (s.w[k] != 0.0f) want.push_back({s.o[k], bits_of(r * s.w[k])});
            else if (s.o[k] < 0 || s.o[k] >= n) ++c.unvisited;
        }
    Adds got;
    got.swap(lanes.all);
    for (auto &a : got) c.outside += a.first < 0 || a.first >= n;
    std::sort(got.begin(), got.end());
    std::sort(want.begin(), want.end());
    c.adds += got.size();
    c.differ += got != want;
}

template <bool TOF, bool QDIV, int G, int U>
static Counts check(const std::vector<float> &lors, const Grid &g, const TofParams &tp, float r) {
    Counts c;
    const int64_t n = (int64_t)g.nx * g.ny * g.nz;
    std::vector<float> image(1);
    const int64_t sx[3] = {1, g.nx, (int64_t)g.nx * g.ny}, sy[3] = {g.ny, 1, (int64_t)g.nx * g.ny};
    const GridK k = make_gridk<TOF>(g, tp);
    for (size_t i = 0; 7 * i < lors.size(); ++i) {
        const float *l = &lors[7 * i];
        const LeanRec E = make_lean<TOF, G>(setup_rec<TOF>(l, l[6], 1.0f, g, k), g, k, sx, sy, true, G * U);
        if (!(E.flags & F_VALID) || (E.flags & F_TIE)) continue;
        ++c.lors;
        const LeanAxes ax = lean_axes(E, g);
        // what the lanes of a walk scatter, call by call; a short LOR also as one range-tested chunk
        std::vector<std::vector<Slots>> calls;
        auto put = [&](size_t call, int lane, const int32_t *o, const float *w) {
            if (calls.size() <= call) calls.resize(call + 1, std::vector<Slots>(G));
            std::memcpy(calls[call][lane].o, o, 12);
            std::memcpy(calls[call][lane].w, w, 12);
        };
        const bool chunk = E.hi - E.lo < G * U;
        for (int lane = 0; lane < G; ++lane) {
            size_t call = 0;
            if (chunk) {
                int32_t o[U][3];
                float w[U][3];
                edge_chunk<TOF, U, G, QDIV>(E, ax, E.lo, E.hi, lane, o, w);
                for (int u = 0; u < U; ++u) put(call++, lane, o[u], w[u]);
            }
            lean_walk<TOF, U, G, QDIV>(E, ax, E.lo, E.hi, lane, [&](auto &o, auto &w, auto ng) {
                for (int u = 0; u < decltype(ng)::value; ++u) put(call++, lane, o[u], w[u]);
            });
        }
        for (auto &at : calls) scatter_group<G>(at, r, n, image.data(), c);
    }
    return c;
}

// argv: file of n x 7 floats, grid, size, TOF (0 / 1), nsigma, value
int main(int, char **v) {
    std::vector<float> lors;
    FILE *f = fopen(v[1], "rb");
    float row[7];
    while (f && fread(row, 4, 7, f) == 7) lors.insert(lors.end(), row, row + 7);
    const Grid g{atoi(v[2]), atoi(v[3]), atoi(v[4]), 0, 0, 0, (float)atof(v[5]), (float)atof(v[6]), (float)atof(v[7])};
    const TofParams tp{3.66f, 1138.0f, (float)atof(v[9])};
    const bool tof = atoi(v[8]), qdiv = grid_qdiv(g);
    const float r = (float)atof(v[10]);
    auto show = [](const Counts &c) { printf("%ld %ld %ld %ld %ld\n", c.lors, c.adds, c.unvisited, c.outside, c.differ); };
#define SRF_RUN(G, U) show(tof ? (qdiv ? check<true, true, G, U>(lors, g, tp, r) : check<true, false, G, U>(lors, g, tp, r)) \
                              : (qdiv ? check<false, true, G, U>(lors, g, tp, r) : check<false, false, G, U>(lors, g, tp, r)))
    SRF_RUN(32, 4);
    SRF_RUN(32, 2);
    SRF_RUN(16, 4);
    SRF_RUN(8, 4);
    return 0;
}
