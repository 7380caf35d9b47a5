// Image layout changes in one pass: dst[0], dst[1] = src[0] (+ src[1]), every array a (nx, ny, nz) image
// with strides of its own. The traversals want x-fastest images with a y-fastest copy beside them, callers
// hold z-fastest ones, and backprojections come back as an x-fastest and a y-fastest half.
//
// A block moves a 16 x 16 x 16 tile through shared memory; each array is read or written with 16 lanes
// along its own unit-stride axis, 64-byte segments whichever axis that is, and every array is touched
// once. Bound by memory: 200 x 200 x 109, one source and two copies 53 MB, two 20-us copies of the framework library -> one 12-us pass.
#include "common.cuh"

namespace srf {

struct Strided {
    float *p;
    int64_t st[3];
    int fast;  // axis of the lanes: the one of unit stride (z if there is none)
};

struct Relayout {
    Strided src[2], dst[2];
};

constexpr int kEdge = 16;

// Tile coordinates of element e (0 .. 4095) of an array whose fastest axis is `fast`.
__device__ __forceinline__ void tile_coord(int e, int fast, int c[3]) {
    const int f = e & 15, a = (e >> 4) & 15, b = e >> 8;
    c[0] = fast == 0 ? f : a;
    c[1] = fast == 1 ? f : (fast == 0 ? a : b);
    c[2] = fast == 2 ? f : b;
}

__global__ void __launch_bounds__(256)
k_relayout(Relayout r, int nx, int ny, int nz) {
    // [x][y][z]; strides 273, 17 and 1 keep 16 lanes along any axis on different banks
    __shared__ float tile[kEdge * 273];
    const int o[3] = {(int)blockIdx.x * kEdge, (int)blockIdx.y * kEdge, (int)blockIdx.z * kEdge};
    const int n[3] = {nx - o[0], ny - o[1], nz - o[2]};
    auto at = [&](const Strided &s, const int c[3]) {
        return s.p + ((o[0] + c[0]) * s.st[0] + (o[1] + c[1]) * s.st[1] + (o[2] + c[2]) * s.st[2]);
    };
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const Strided s = r.src[k];
        if (s.p == nullptr) break;
        float v[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            int c[3];
            tile_coord(threadIdx.x + 256 * i, s.fast, c);
            v[i] = c[0] < n[0] && c[1] < n[1] && c[2] < n[2] ? __ldg(at(s, c)) : 0.0f;
        }
        if (k) __syncthreads();
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            int c[3];
            tile_coord(threadIdx.x + 256 * i, s.fast, c);
            float &t = tile[c[0] * 273 + c[1] * 17 + c[2]];
            t = k ? __fadd_rn(t, v[i]) : v[i];
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const Strided s = r.dst[k];
        if (s.p == nullptr) break;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            int c[3];
            tile_coord(threadIdx.x + 256 * i, s.fast, c);
            if (c[0] < n[0] && c[1] < n[1] && c[2] < n[2]) *at(s, c) = tile[c[0] * 273 + c[1] * 17 + c[2]];
        }
    }
}

}  // namespace srf

using namespace srf;

extern "C" int srf_relayout(const float *src, const int64_t src_strides[3], const float *src2, const int64_t src2_strides[3],
                            float *dst, const int64_t dst_strides[3], float *dst2, const int64_t dst2_strides[3],
                            const int32_t grid[3], void *stream) {
    if (!grid) return fail(SRF_EINVAL, "grid must not be NULL");
    Grid g; int rc;
    const float c[3] = {0, 0, 0}, sz[3] = {1, 1, 1};
    if ((rc = check_geometry(grid, c, sz, g))) return rc;
    Relayout r;
    auto put = [&](const float *p, const int64_t *st, const char *name, bool required, Strided &s) {
        View v;
        if (int e = check_view(p, st, g, name, v, required)) return e;
        s = Strided{v.ptr, {v.st[0], v.st[1], v.st[2]}, v.st[0] == 1 ? 0 : v.st[1] == 1 ? 1 : 2};
        return (int)SRF_OK;
    };
    if ((rc = put(src, src_strides, "src", true, r.src[0]))) return rc;
    if ((rc = put(src2, src2_strides, "src2", false, r.src[1]))) return rc;
    if ((rc = put(dst, dst_strides, "dst", true, r.dst[0]))) return rc;
    if ((rc = put(dst2, dst2_strides, "dst2", false, r.dst[1]))) return rc;
    const dim3 blocks((g.nx + kEdge - 1) / kEdge, (g.ny + kEdge - 1) / kEdge, (g.nz + kEdge - 1) / kEdge);
    k_relayout<<<blocks, 256, 0, (cudaStream_t)stream>>>(r, g.nx, g.ny, g.nz);
    return check_cuda("relayout kernel launch");
}
