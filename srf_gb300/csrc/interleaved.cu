// The batched projector and its exact adjoint on interleaved images: the W = 2, 4 or 8 values of a
// voxel (one per image) stand next to each other, so that a voxel visit is one or two 16-byte loads
// or vector reductions instead of a 4-byte access per image. Each LOR is set up and traversed once for all
// images, as in the separate-image form (k_trace_fused_batch), with the same slabs, voxels and
// weights.
//
// What bounds the separate-image form is its accesses: per slab and slot a warp touches ~11 sectors
// of 32 bytes in each image (32 slabs cross ~14 rows of 8 voxels), 91 for eight images, in eight
// instructions. Interleaved by eight, a voxel is one sector whatever the direction of the LOR: 32
// sectors in two instructions, and projections need no second layout for y-dominant LORs (W = 2 and 4
// keep one). Adjoints keep a second accumulator at every width: with one, a voxel's sum has twice the rms
// rounding error (1.97 times at 1,100 terms a voxel).
// Measured, 8 images 128 x 128 x 64, 5e6 TOF LORs at 3 sigma, projection + adjoint with the loss between
// them: 21.7 -> 7.6 ms (8.0 ms with one accumulator).
#include "common.cuh"
#include "fused.cuh"
#include "lean.cuh"

namespace srf {

template <int W>
struct Vals {
    float2 v[W / 2];
};

template <int W>
__device__ __forceinline__ Vals<W> load_vals(const float *__restrict__ p) {
    Vals<W> r;
    if constexpr (W == 2) {
        r.v[0] = __ldg(reinterpret_cast<const float2 *>(p));
    } else {
#pragma unroll
        for (int k = 0; k < W / 4; ++k) {
            const float4 q = __ldg(reinterpret_cast<const float4 *>(p) + k);
            r.v[2 * k] = make_float2(q.x, q.y);
            r.v[2 * k + 1] = make_float2(q.z, q.w);
        }
    }
    return r;
}

// p[0 .. W) += v, as vector reductions (no order among or within them, as scalar atomicAdd)
template <int W>
__device__ __forceinline__ void red_vals(float *p, const Vals<W> &a) {
    if constexpr (W == 2) {
        asm volatile("red.relaxed.gpu.global.add.v2.f32 [%0], {%1, %2};" ::"l"(p), "f"(a.v[0].x), "f"(a.v[0].y) : "memory");
    } else {
#pragma unroll
        for (int k = 0; k < W / 4; ++k)
            asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p + 4 * k), "f"(a.v[2 * k].x),
                         "f"(a.v[2 * k].y), "f"(a.v[2 * k + 1].x), "f"(a.v[2 * k + 1].y)
                         : "memory");
    }
}

template <int W>
__device__ __forceinline__ Vals<W> times(const Vals<W> &a, float w) {
    Vals<W> r;
#pragma unroll
    for (int k = 0; k < W / 2; ++k) r.v[k] = __fmul2_rn(a.v[k], make_float2(w, w));
    return r;
}

// Sums the lanes' W partial values: halves are exchanged until each lane holds one image's sum over
// a set of lanes (W - 1 shuffles), then the sets are added. Lanes whose low bits are 0 return the sum
// of image `which`.
template <int W>
__device__ __forceinline__ float sum_vals(const Vals<W> &a, int lane, int &which) {
    float x[W];
#pragma unroll
    for (int k = 0; k < W / 2; ++k) { x[2 * k] = a.v[k].x; x[2 * k + 1] = a.v[k].y; }
    which = 0;
    int mask = 16;
#pragma unroll
    for (int h = W / 2; h > 0; h /= 2, mask /= 2) {
        const bool upper = lane & mask;
        which += upper ? h : 0;
#pragma unroll
        for (int k = 0; k < h; ++k) {
            const float send = upper ? x[k] : x[k + h];
            x[k] = (upper ? x[k + h] : x[k]) + __shfl_xor_sync(0xffffffffu, send, mask);
        }
    }
    for (; mask > 0; mask /= 2) x[0] += __shfl_xor_sync(0xffffffffu, x[0], mask);
    return x[0];
}

constexpr int kIlBlock = 128;
constexpr int kIlSlabs = 2;  // slabs per lane and chunk: offsets and weights are used at once, so few are held

// ADJ: values -> images; else images -> out. LORs, batches and rows as k_trace_fused_batch.
template <bool TOF, int W, bool ADJ, bool QDIV>
__global__ void __launch_bounds__(kIlBlock, 5)
k_trace_il(const float *__restrict__ lors, int64_t n, int stride, const float *__restrict__ tof, int tof_stride, Grid g,
           TofParams tp, int nb, float *__restrict__ rows, int64_t rstride, View v, View vt, int batch) {
    constexpr int U = kIlSlabs;
    __shared__ LeanRec s_rec[kIlBlock / 32][32];
    __shared__ __align__(16) float s_val[kIlBlock / 32][32][W];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    LeanRec *rec = s_rec[wib];
    float(*val)[W] = s_val[wib];
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const bool have_t = vt.ptr != nullptr;
    const GridK k = make_gridk<TOF>(g, tp);
    for (int64_t base = warp * batch; base < n; base += nwarps * batch) {
        const int64_t il = base + lane;
        const bool mine = il < n && lane < batch;
        {
            LeanRec E = {};
            E.lo = 1;
            if (mine) {
                const float *l = lors + il * stride;
                float lv[6];
#pragma unroll
                for (int c = 0; c < 6; ++c) lv[c] = __ldg(l + c);
                const float tv = TOF ? __ldg(tof + il * tof_stride) : 0.0f;
                E = make_lean<TOF, 32>(setup_rec<TOF>(lv, tv, 1.0f, g, k), g, k, v.st, vt.st, have_t, 0);
            }
            store_lean(&rec[lane], E);
#pragma unroll
            for (int b = 0; b < W; ++b) val[lane][b] = ADJ && mine && b < nb ? __ldg(rows + b * rstride + il) : 0.0f;
        }
        __syncwarp();
        for (int j = 0; j < batch; ++j) {
            const LeanRec E = load_lean(&rec[j]);
            Vals<W> a;  // ADJ: the LOR's values, else its partial sums
            bool any = false;
#pragma unroll
            for (int b = 0; b < W / 2; ++b) {
                a.v[b] = ADJ ? *reinterpret_cast<const float2 *>(&val[j][2 * b]) : make_float2(0.0f, 0.0f);
                any = any || a.v[b].x != 0.0f || a.v[b].y != 0.0f;
            }
            const bool tie = !TOF && (E.flags & F_TIE);
            if ((!ADJ || any) && tie) {  // the non-TOF projector's own axis: generic slabs
                const float *l = lors + (base + j) * stride;
                LorSetup S;
                if (setup_lor<TOF, RULES_PROJ>(__ldg(l), __ldg(l + 1), __ldg(l + 2), __ldg(l + 3), __ldg(l + 4), __ldg(l + 5),
                                               0.0f, g, tp, v.st, vt.st, have_t, S)) {
                    float *im = (!S.xdom && have_t) ? vt.ptr : v.ptr;
                    for (int ip = S.lo + lane; ip <= S.hi; ip += 32)
                        slab<TOF, RULES_PROJ>(S, ip, [&](int32_t off, float w) {
                            if (ADJ) {
                                red_vals<W>(im + off, times<W>(a, w));
                            } else {
                                const Vals<W> x = load_vals<W>(im + off);
#pragma unroll
                                for (int b = 0; b < W / 2; ++b) a.v[b] = __ffma2_rn(x.v[b], make_float2(w, w), a.v[b]);
                            }
                        });
                }
            } else if ((!ADJ || any) && (E.flags & F_VALID) && (E.flags & F_PROJ)) {
                float *im = (!(E.flags & F_XDOM) && have_t) ? vt.ptr : v.ptr;
                if (ADJ) a = times<W>(a, E.invL2);
                lean_walk<TOF, U, 32, QDIV>(E, lean_axes(E, g), E.plo, E.phi, lane, [&](auto &o, auto &w, auto ng) {
#pragma unroll
                    for (int u = 0; u < decltype(ng)::value; ++u) {
                        if (ADJ) {
#pragma unroll
                            for (int c = 0; c < 3; ++c)
                                if (w[u][c] != 0.0f) red_vals<W>(im + o[u][c], times<W>(a, w[u][c]));
                        } else {
                            Vals<W> x[3] = {};
#pragma unroll
                            for (int c = 0; c < 3; ++c)
                                if (w[u][c] != 0.0f) x[c] = load_vals<W>(im + o[u][c]);
#pragma unroll
                            for (int c = 0; c < 3; ++c)
#pragma unroll
                                for (int b = 0; b < W / 2; ++b)
                                    a.v[b] = __ffma2_rn(x[c].v[b], make_float2(w[u][c], w[u][c]), a.v[b]);
                        }
                    }
                });
                if (!ADJ) a = times<W>(a, E.invL2);
            }
            if (!ADJ) {
                int which;
                const float p = sum_vals<W>(a, lane, which);
                if ((lane & (32 / W - 1)) == 0) val[j][which] = p;
            }
        }
        __syncwarp();
        if (!ADJ && mine)
#pragma unroll
            for (int b = 0; b < W; ++b)
                if (b < nb) rows[b * rstride + il] = val[lane][b];
        __syncwarp();
    }
}

// ---------------------------------------------------------------- layouts
// Images b < nb of any strides (sb, s[]) into dst, W values per voxel (0 for b >= nb), x-fastest, and
// into dst_t (when given), y-fastest. A block moves a 32 x 32 tile of (a, c): c the axis of unit stride
// in the source, a the fastest axis of the destination; both sides are coalesced.
struct IlSrc {
    const float *p;
    int64_t sb, st[3];
};

template <int W, bool TO>
__global__ void __launch_bounds__(256)
k_il_tile(IlSrc src, int nb, float *__restrict__ il, float *__restrict__ flat, const float *__restrict__ il_t, int na, int nm,
          int nc, int64_t ta, int64_t tm, int64_t tc, int64_t da, int64_t dm, int64_t dc) {
    // element (a, m, c): source strides (ta, tm, tc) per image, interleaved strides (da, dm, dc) in voxels
    __shared__ float tile[32][32 * W + 1];
    const int a0 = blockIdx.x * 32, c0 = blockIdx.y * 32;
    const int lane = threadIdx.x & 31, row = threadIdx.x >> 5;
    for (int m = blockIdx.z; m < nm; m += gridDim.z) {
        if (TO) {
            for (int b = 0; b < W; ++b)
                for (int r = row; r < 32; r += 8) {
                    const int a = a0 + r, c = c0 + lane;
                    tile[lane][r * W + b] = b < nb && a < na && c < nc ? src.p[b * src.sb + a * ta + m * tm + c * tc] : 0.0f;
                }
            __syncthreads();
            for (int r = row; r < 32; r += 8) {
                const int c = c0 + r;
                for (int e = lane; e < 32 * W; e += 32)
                    if (c < nc && a0 + e / W < na) il[((int64_t)a0 * da + m * dm + c * dc) * W + e] = tile[r][e];
            }
        } else {
            for (int r = row; r < 32; r += 8) {
                const int c = c0 + r;
                for (int e = lane; e < 32 * W; e += 32)
                    tile[r][e] = c < nc && a0 + e / W < na ? il[((int64_t)a0 * da + m * dm + c * dc) * W + e] : 0.0f;
            }
            __syncthreads();
            for (int b = 0; b < nb; ++b)
                for (int r = row; r < 32; r += 8) {
                    const int a = a0 + r, c = c0 + lane;
                    if (a >= na || c >= nc) continue;
                    const int64_t o = b * src.sb + a * ta + m * tm + c * tc;
                    const float x = tile[lane][r * W + b];
                    flat[o] = il_t != nullptr ? __fadd_rn(flat[o], x) : x;
                }
        }
        __syncthreads();
    }
}

template <bool TO>
static int il_tiles(int W, const IlSrc &src, int nb, float *il, float *flat, bool y_fast, bool add, const Grid &g, cudaStream_t s) {
    // a: fastest axis of the interleaved layout (x, or y for the y-fastest one); c: z when it has unit stride
    // in the flat images (or by default), else the other transaxial axis is as good
    const int a = y_fast ? 1 : 0, m = y_fast ? 0 : 1, n[3] = {g.nx, g.ny, g.nz};
    const int64_t dst[3] = {y_fast ? (int64_t)g.ny : 1, y_fast ? 1 : (int64_t)g.nx, (int64_t)g.nx * g.ny};
    const dim3 blocks((n[a] + 31) / 32, (g.nz + 31) / 32, n[m] < 65535 ? n[m] : 65535);
    const float *flag = add ? il : nullptr;
#define SRF_IL(w) k_il_tile<w, TO><<<blocks, 256, 0, s>>>(src, nb, il, flat, flag, n[a], n[m], g.nz, src.st[a], src.st[m], src.st[2], dst[a], dst[m], dst[2])
    if (W == 2) SRF_IL(2);
    else if (W == 4) SRF_IL(4);
    else SRF_IL(8);
#undef SRF_IL
    return check_cuda("interleave kernel launch");
}

template <bool TOF, int W, bool ADJ>
static int launch_il(const float *lors, int64_t n, int stride, const float *tof, int tof_stride, const Grid &g,
                     const TofParams &tp, int nb, float *rows, int64_t rstride, const View &v, const View &vt, cudaStream_t s) {
    auto kern = grid_qdiv(g) ? k_trace_il<TOF, W, ADJ, true> : k_trace_il<TOF, W, ADJ, false>;
    const LorSplit d = split_lors(kern, n, 1, kIlBlock);
    kern<<<d.blocks, kIlBlock, 0, s>>>(lors, n, stride, tof, tof_stride, g, tp, nb, rows, rstride, v, vt, d.batch);
    return check_cuda("interleaved projector kernel launch");
}

template <bool ADJ>
static int project_il(const float *lors, int64_t n, int32_t lor_stride, const float *tof, int32_t tof_stride, float tof_bin,
                      float tof_sigma2, float tof_nsigma, int32_t nb, int32_t width, const float *images,
                      const float *images_t, const int32_t grid[3], const float center[3], const float size[3],
                      const float *rows, int64_t rstride, cudaStream_t s) {
    Grid g; int rc;
    if ((rc = check_lors(lors, n, lor_stride))) return rc;
    if ((rc = check_geometry(grid, center, size, g))) return rc;
    if (width != 2 && width != 4 && width != 8) return fail(SRF_EINVAL, "width must be 2, 4 or 8");
    if (nb < 1 || nb > width) return fail(SRF_EINVAL, "n_images must be 1..width");
    if (rstride < n) return fail(SRF_EINVAL, "row stride of the LOR values is below n");
    if (n > 0 && !rows) return fail(SRF_EINVAL, "LOR values must not be NULL");
    if (((uintptr_t)images | (uintptr_t)images_t) & (4 * width - 1)) return fail(SRF_EINVAL, "interleaved images must be aligned to a voxel");
    const int64_t w = width, xs[3] = {w, w * g.nx, w * g.nx * g.ny}, ys[3] = {w * g.ny, w, w * g.nx * g.ny};
    View v, vt;
    if ((rc = check_view(images, xs, g, "images", v, true))) return rc;
    if ((rc = check_view(images_t, ys, g, "images_t", vt, false))) return rc;
    TofParams tp{0, 0, 0};
    if (tof && (rc = check_tof(tof, n, tof_stride, tof_bin, tof_sigma2, tof_nsigma, tp))) return rc;
    if (n == 0) return ok();
    float *r = const_cast<float *>(rows);
#define SRF_IL(w) (tof ? launch_il<true, w, ADJ>(lors, n, lor_stride, tof, tof_stride, g, tp, nb, r, rstride, v, vt, s) \
                       : launch_il<false, w, ADJ>(lors, n, lor_stride, nullptr, 1, g, tp, nb, r, rstride, v, vt, s))
    return width == 2 ? SRF_IL(2) : width == 4 ? SRF_IL(4) : SRF_IL(8);
#undef SRF_IL
}

static int layout_args(const void *images, int64_t batch_stride, const int64_t st[3], int32_t nb, int32_t width, const void *il,
                       const int32_t grid[3], Grid &g, IlSrc &src) {
    if (!images || !st || !il || !grid) return fail(SRF_EINVAL, "NULL argument");
    const float c[3] = {0, 0, 0}, sz[3] = {1, 1, 1};
    int rc;
    if ((rc = check_geometry(grid, c, sz, g))) return rc;
    if (width != 2 && width != 4 && width != 8) return fail(SRF_EINVAL, "width must be 2, 4 or 8");
    if (nb < 1 || nb > width) return fail(SRF_EINVAL, "n_images must be 1..width");
    src = IlSrc{static_cast<const float *>(images), batch_stride, {st[0], st[1], st[2]}};
    return SRF_OK;
}

}  // namespace srf

using namespace srf;

extern "C" {

int srf_interleave(const float *images, int64_t batch_stride, const int64_t image_strides[3], int32_t n_images, int32_t width,
                   const int32_t grid[3], float *il, float *il_t, void *stream) {
    Grid g; IlSrc src; int rc;
    if ((rc = layout_args(images, batch_stride, image_strides, n_images, width, il, grid, g, src))) return rc;
    if ((rc = il_tiles<true>(width, src, n_images, il, nullptr, false, false, g, (cudaStream_t)stream))) return rc;
    return il_t ? il_tiles<true>(width, src, n_images, il_t, nullptr, true, false, g, (cudaStream_t)stream) : rc;
}

int srf_deinterleave(const float *il, const float *il_t, int32_t n_images, int32_t width, const int32_t grid[3], float *images,
                     int64_t batch_stride, const int64_t image_strides[3], void *stream) {
    Grid g; IlSrc src; int rc;
    if ((rc = layout_args(images, batch_stride, image_strides, n_images, width, il, grid, g, src))) return rc;
    if ((rc = il_tiles<false>(width, src, n_images, const_cast<float *>(il), images, false, false, g, (cudaStream_t)stream))) return rc;
    return il_t ? il_tiles<false>(width, src, n_images, const_cast<float *>(il_t), images, true, true, g, (cudaStream_t)stream) : rc;
}

int srf_projection_il(const float *lors, int64_t n, int32_t lor_stride, const float *tof, int32_t tof_stride, float tof_bin,
                      float tof_sigma2, float tof_nsigma, int32_t n_images, int32_t width, const float *il, const float *il_t,
                      const int32_t grid[3], const float center[3], const float size[3], float *out, int64_t out_stride,
                      void *stream) {
    return project_il<false>(lors, n, lor_stride, tof, tof_stride, tof_bin, tof_sigma2, tof_nsigma, n_images, width, il, il_t,
                             grid, center, size, out, out_stride, (cudaStream_t)stream);
}

int srf_projection_adjoint_il(const float *lors, int64_t n, int32_t lor_stride, const float *tof, int32_t tof_stride,
                              float tof_bin, float tof_sigma2, float tof_nsigma, int32_t n_images, int32_t width,
                              const float *values, int64_t values_stride, float *il, float *il_t, const int32_t grid[3],
                              const float center[3], const float size[3], void *stream) {
    return project_il<true>(lors, n, lor_stride, tof, tof_stride, tof_bin, tof_sigma2, tof_nsigma, n_images, width, il, il_t,
                            grid, center, size, values, values_stride, (cudaStream_t)stream);
}

}  // extern "C"
