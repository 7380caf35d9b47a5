// Sensitivity image over all ordered crystal pairs, with the LORs generated on the device.
//
// srfnef's EcatEmapGenerator('block-full') (srfnef/functions/emap_generator.py:77-111) builds, for
// each of nb x nb block columns, an M^2-row LOR array on the host with numpy and launches the
// non-TOF backprojector on it (2304 launches and 1.05e9 LORs for a 48-block, 676-crystal-column
// scanner). Here LOR k = ((i*nb + j)*M + a)*M + b takes endpoint 1 from table row i*M + a and
// endpoint 2 from row j*M + b of a crystal table that holds exactly the float32 positions the
// reference computes (srf_gb300.geometry.block_full_crystal_table). Two forms:
//
//  * by column pairs (k_emap_columns, srf_emap_block_full_ws): the crystals of a cylindrical scanner
//    stand in axial columns, rows of the table with the same (x, y) to the bit. All c1 x c2 lines
//    between two columns share their transaxial geometry: the dominant axis, the slabs, the in-plane
//    faces and crossings. Only their axial coordinate and length differ.
//  * line by line (k_emap_fused in osem.cu, srf_emap_block_full): every LOR through the fused
//    kernel's backprojector traversal with value 1; also for tables without such columns.
#include "common.cuh"
#include "fused.cuh"
#include "lean.cuh"

namespace srf {

// ---------------------------------------------------------------- columns of the table
// Work area of srf_emap_block_full_ws, in 4-byte words: a hash table of (x, y) keys, then per row.
struct EmapCols {
    unsigned long long *keys;  // [slots] bit patterns of (x, y); ~0 = free
    int *slot_n, *slot_col;    // [slots] members, column index
    int *row_slot;             // [rows] hash slot, or -1 (a non-finite row contributes nothing)
    int *off;                  // [rows + 1] first member of each column
    int *fill;                 // [rows]
    float2 *xy;                // [rows] (x, y) of each column
    float *zu, *z;             // [rows] members' z, as collected and sorted by column
    int *meta;                 // [0] number of columns, [1] 1: the column form runs
};

inline int64_t emap_slots(int64_t rows) {
    int64_t h = 64;
    while (h < 2 * rows) h *= 2;
    return h;
}

inline int64_t emap_words(int64_t rows) { return emap_slots(rows) * 4 + rows * 8 + 16; }

static EmapCols emap_cols(int32_t *ws, int64_t rows) {
    const int64_t h = emap_slots(rows);
    EmapCols c;
    c.keys = reinterpret_cast<unsigned long long *>(ws); ws += 2 * h;
    c.xy = reinterpret_cast<float2 *>(ws); ws += 2 * rows;
    c.slot_n = ws; ws += h;
    c.slot_col = ws; ws += h;
    c.row_slot = ws; ws += rows;
    c.off = ws; ws += rows + 1;
    c.fill = ws; ws += rows;
    c.zu = reinterpret_cast<float *>(ws); ws += rows;
    c.z = reinterpret_cast<float *>(ws); ws += rows;
    c.meta = ws;
    return c;
}

__global__ void k_cols_clear(EmapCols c, int slots, int rows) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < slots; i += gridDim.x * blockDim.x) {
        c.keys[i] = ~0ull;
        c.slot_n[i] = 0;
        if (i < rows) c.fill[i] = 0;
    }
}

__global__ void k_cols_insert(const float *__restrict__ table, EmapCols c, int slots, int rows) {
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += gridDim.x * blockDim.x) {
        const float x = table[3 * (int64_t)r], y = table[3 * (int64_t)r + 1], z = table[3 * (int64_t)r + 2];
        if (!(isfinite(x) && isfinite(y) && isfinite(z))) {
            c.row_slot[r] = -1;
            continue;
        }
        const unsigned long long key = ((unsigned long long)__float_as_uint(x) << 32) | __float_as_uint(y);
        unsigned h = (unsigned)((key * 0x9E3779B97F4A7C15ull) >> 40) & (unsigned)(slots - 1);
        for (int t = 0; t < slots; ++t, h = (h + 1) & (unsigned)(slots - 1)) {  // half the slots stay free
            const unsigned long long old = atomicCAS(c.keys + h, ~0ull, key);
            if (old == ~0ull || old == key) break;
        }
        c.row_slot[r] = (int)h;
        atomicAdd(c.slot_n + h, 1);
    }
}

// One block: the columns in slot order and their member offsets.
__global__ void __launch_bounds__(1024) k_cols_offsets(EmapCols c, int slots, int rows, int min_members) {
    __shared__ int s_c[32], s_n[32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int cols = 0, members = 0;  // totals of the slots before this round
    for (int base = 0; base < slots; base += 1024) {
        const int i = base + threadIdx.x;
        const int n = i < slots ? c.slot_n[i] : 0;
        int pc = n > 0 ? 1 : 0, pn = n;  // inclusive scans over the block
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int a = __shfl_up_sync(0xffffffffu, pc, o), b = __shfl_up_sync(0xffffffffu, pn, o);
            if (lane >= o) { pc += a; pn += b; }
        }
        if (lane == 31) { s_c[w] = pc; s_n[w] = pn; }
        __syncthreads();
        int bc = 0, bn = 0, tc = 0, tn = 0;
        for (int k = 0; k < 32; ++k) {
            if (k < w) { bc += s_c[k]; bn += s_n[k]; }
            tc += s_c[k]; tn += s_n[k];
        }
        if (n > 0) {
            const int col = cols + bc + pc - 1;
            const unsigned long long key = c.keys[i];
            c.slot_col[i] = col;
            c.off[col] = members + bn + pn - n;
            c.xy[col] = make_float2(__uint_as_float((unsigned)(key >> 32)), __uint_as_float((unsigned)key));
        }
        cols += tc; members += tn;
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        c.off[cols] = members;
        c.meta[0] = cols;
        c.meta[1] = (int64_t)min_members * cols <= members ? 1 : 0;
    }
}

__global__ void k_cols_collect(const float *__restrict__ table, EmapCols c, int rows) {
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += gridDim.x * blockDim.x) {
        const int s = c.row_slot[r];
        if (s < 0) continue;
        const int col = c.slot_col[s];
        c.zu[c.off[col] + atomicAdd(c.fill + col, 1)] = table[3 * (int64_t)r + 2];
    }
}

// Each column's members by z, ascending (rank by counting; the order of equal values is free).
__global__ void k_cols_sort(EmapCols c) {
    if (!c.meta[1]) return;
    const int cols = c.meta[0];
    for (int col = blockIdx.x; col < cols; col += gridDim.x) {
        const int lo = c.off[col], n = c.off[col + 1] - lo;
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            const float z = c.zu[lo + i];
            int rank = 0;
            for (int j = 0; j < n; ++j) {
                const float v = c.zu[lo + j];
                rank += (v < z || (v == z && j < i)) ? 1 : 0;
            }
            c.z[lo + rank] = z;
        }
    }
}

// ---------------------------------------------------------------- lines between two columns
constexpr int kParams = 64;  // members of the second column whose line constants are held at a time

// The lines from one member (axial face coordinate zA) to `cnt` members of the other column, on one
// slab per lane. prm[j] = (D, wc, 1 / |axial step per slab|): D the axial extent in voxels, wc the
// weight of a whole slab. ta, tb: the slab's two faces along the line (0 at zA, 1 at the other end),
// the one with the lower axial coordinate first. fq: fraction of the slab before its in-plane
// crossing. Cell (a, c): lane's word at s[(c + row) * 32], rows from row a of the two in-plane cells.
// Slots and weights as lean_slab's; RANGE adds its axial range tests (the in-plane ones are per
// slab and decided when the cells are written out).
template <bool RANGE>
__device__ __forceinline__ void column_lines(float *s, const float4 *prm, int j0, int cnt, float zA, float ta, float tb,
                                             float fq, int nz) {
    const unsigned cA = 0u - (unsigned)kFloorBits * 32u, cB = cA + (unsigned)nz * 32u;
    constexpr int K = 4;  // lines whose arithmetic is interleaved before their additions run in order
    for (int j = j0; j < cnt; j += K) {
        unsigned i0[K], i1[K], i2[K];
        float w0[K], w1[K], w2[K];
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const float4 p = prm[min(j + k, cnt - 1)];
            const float wc = j + k < cnt ? p.y : 0.0f;
            float z1 = fmaf(p.x, ta, zA), z2 = fmaf(p.x, tb, zA);
            if (RANGE) {
                z1 = fminf(fmaxf(z1, -2097152.0f), 2097152.0f);
                z2 = fminf(fmaxf(z2, -2097152.0f), 2097152.0f);
            }
            const float f1 = __fadd_rd(z1, kFloorMagic), f2 = __fadd_rd(z2, kFloorMagic);
            const unsigned b1 = (unsigned)__float_as_int(f1), b2 = (unsigned)__float_as_int(f2);
            const float fz = b1 != b2 ? ((f2 - kFloorMagic) - z1) * p.z : 1.0f;
            const bool qfirst = fq > fz;
            w0[k] = fminf(fq, fz) * wc;
            w1[k] = fabsf(fq - fz) * wc;
            w2[k] = fmaf(-fmaxf(fq, fz), wc, wc);
            i0[k] = b1 * 32u + cA;
            i1[k] = (qfirst ? b2 : b1) * 32u + (qfirst ? cA : cB);
            i2[k] = b2 * 32u + cB;
            if (RANGE) {
                const int c1 = (int)b1 - kFloorBits, c2 = (int)b2 - kFloorBits;
                const bool B = (unsigned)c1 < (unsigned)nz, D = (unsigned)c2 < (unsigned)nz && c1 >= -1;
                const bool v1 = qfirst ? D : B;
                w0[k] = B ? w0[k] : 0.0f; i0[k] = B ? i0[k] : 0u;
                w1[k] = v1 ? w1[k] : 0.0f; i1[k] = v1 ? i1[k] : (unsigned)nz * 32u;
                w2[k] = D ? w2[k] : 0.0f; i2[k] = D ? i2[k] : 0u;
            }
        }
#pragma unroll
        for (int k = 0; k < K; ++k) {
            if (RANGE) {  // dropped slots add zero to some cell, so the additions keep their order
                s[i0[k]] += w0[k];
                s[i1[k]] += w1[k];
                s[i2[k]] += w2[k];
                continue;
            }
            // slots 0 and 1 are different cells, and slot 2 (both coordinates cross) a third
            const float a = s[i0[k]], b = s[i1[k]];
            if (w2[k] != 0.0f) s[i2[k]] += w2[k];
            s[i0[k]] = a + w0[k];
            s[i1[k]] = b + w1[k];
        }
    }
}

// One warp (= one block) takes one pair of columns A < B and one tile of 32 slabs; each lane owns a
// slab: two in-plane cells (before and after its crossing) of nz voxels each in shared memory, private
// to the lane, so the c1 c2 lines accumulate there without atomics. The cells then go to the image
// with one reduction per voxel, times two: the line from B to A is the line from A to B, and both
// are in the sum (a column with itself has no transaxial extent and is skipped by the short-LOR rule).
// Bound: instruction issue of the loop over the lines, ~32 instructions per line and 32 slabs against
// ~120 of the line-by-line form and half the lines; shared memory (2 nz words per lane, 28 KB at
// nz = 109) allows 7 warps per SM, whose additions' latency the K = 4 interleaving covers.
// Measured, 32,448 crystals (624 columns of 52) on 200 x 200 x 109: 121.6 ms against 308 ms line by line.
__global__ void __launch_bounds__(32)
k_emap_columns(EmapCols c, Grid g, View v, View vt, int tiles) {
    extern __shared__ float s_cells[];                      // [2 nz][32]
    __shared__ float4 prm[kParams];
    if (!c.meta[1]) return;
    const int lane = threadIdx.x;
    const int cols = c.meta[0];
    const int64_t items = (int64_t)cols * (cols - 1) / 2 * tiles;
    const TofParams tp{0, 0, 0};
    const GridK k = make_gridk<false>(g, tp);
    const int nz = g.nz;
    float *s = s_cells + lane;
    for (int r = 0; r < 2 * nz; ++r) s[r * 32] = 0.0f;
    for (int64_t it = blockIdx.x; it < items; it += gridDim.x) {
        const int64_t pair = it / tiles;
        // pair = B (B - 1) / 2 + A, A < B
        int B = (int)((1.0 + sqrt(1.0 + 8.0 * (double)pair)) * 0.5);
        while ((int64_t)B * (B - 1) / 2 > pair) --B;
        while ((int64_t)(B + 1) * B / 2 <= pair) ++B;
        const int A = (int)(pair - (int64_t)B * (B - 1) / 2);
        const float2 pa = c.xy[A], pb = c.xy[B];
        const float x1 = __fdiv_rn(__fsub_rn(pa.x, g.cx), k.dx_), y1 = __fdiv_rn(__fsub_rn(pa.y, g.cy), k.dx_);
        const float x2 = __fdiv_rn(__fsub_rn(pb.x, g.cx), k.dx_), y2 = __fdiv_rn(__fsub_rn(pb.y, g.cy), k.dx_);
        const float xd = __fsub_rn(x2, x1), yd = __fsub_rn(y2, y1);
        const float t2d = __fadd_rn(__fmul_rn(xd, xd), __fmul_rn(yd, yd));
        if (!isfinite(t2d) || __fsqrt_rn(t2d) < 10.0f) continue;
        const bool xdom = absr(xd) > absr(yd);
        const float p1 = xdom ? x1 : y1, q1 = xdom ? y1 : x1, pd = xdom ? xd : yd;
        const float kq = __fdiv_rn(xdom ? yd : xd, pd);
        const int np = xdom ? g.nx : g.ny, nq = xdom ? g.ny : g.nx;
        const float np2 = xdom ? k.nx2 : k.ny2, nq2 = xdom ? k.ny2 : k.nx2, dq = xdom ? k.dy : 1.0f;
        int lo = 0, hi = np - 1;
        clip_linear(__fadd_rn(__fdiv_rn(__fsub_rn(q1, __fmul_rn(kq, p1)), dq), nq2), kq / dq, -1.0f, (float)nq + 1.0f,
                    np2, lo, hi);
        lo = max(lo, 0);
        hi = min(hi, np - 1);
        const int first = lo + 32 * (int)(it - pair * tiles);
        if (first > hi) continue;
        const int ip = min(first + lane, hi);
        const bool act = first + lane <= hi;
        const float pp1 = __fsub_rn((float)ip, np2), pp2 = __fadd_rn(pp1, 1.0f);
        const bool q_one = dq == 1.0f;
        const float ua = bcoord(q1, kq, pp1, p1, dq, nq2, q_one), ub = bcoord(q1, kq, pp2, p1, dq, nq2, q_one);
        const float qq1 = kq >= 0.0f ? ua : ub, qq2 = kq >= 0.0f ? ub : ua;
        const int cq1 = ifloor(qq1), cq2 = ifloor(qq2);
        const float fq = cq1 != cq2 ? ((float)cq2 - qq1) / (qq2 - qq1) : 1.0f;
        const bool okA = act && 0 <= cq1 && cq1 < nq, okB = act && 0 <= cq2 && cq2 < nq && cq1 >= -1;
        if (!__any_sync(0xffffffffu, okA || okB)) continue;
        const float t_lo = __fdiv_rn(__fsub_rn(pp1, p1), pd), t_hi = __fdiv_rn(__fsub_rn(pp2, p1), pd);
        const int a0 = c.off[A], na = c.off[A + 1] - a0, b0 = c.off[B], nb = c.off[B + 1] - b0;
        auto face_z = [&](float z) { return __fdiv_rn(__fdiv_rn(__fsub_rn(z, g.cz), k.dx_), k.dz) + k.nz2; };
        // members are sorted: inside the box by a margin when the first and the last of both columns are
        // (and the slab lies between the columns, so that every axial coordinate does too)
        const float zlo = fminf(face_z(c.z[a0]), face_z(c.z[b0])), zhi = fmaxf(face_z(c.z[a0 + na - 1]), face_z(c.z[b0 + nb - 1]));
        const bool between = __all_sync(0xffffffffu, t_lo >= 0.0f && t_lo <= 1.0f && t_hi >= 0.0f && t_hi <= 1.0f);
        const bool inside = between && zlo >= kInteriorMargin && zhi <= (float)nz - kInteriorMargin;
        const float ku = 1.0f + kq * kq, ipd = 1.0f / pd;
        for (int jb = 0; jb < nb; jb += kParams) {
            const int cnt = min(kParams, nb - jb);
            for (int ia = 0; ia < na; ++ia) {
                const float zA = face_z(__ldg(c.z + a0 + ia));
                __syncwarp();
                int down = 0;  // members below A's: D < 0 (they come first)
                for (int j = lane; j < kParams; j += 32) {
                    float D = 0.0f, wc = 0.0f, iz = 0.0f;
                    if (j < cnt) {
                        D = face_z(__ldg(c.z + b0 + jb + j)) - zA;
                        const float kz = D * k.dz * ipd;
                        wc = isfinite(D) ? sqrtf(ku + kz * kz) * k.dx_ : 0.0f;
                        D = isfinite(D) ? D : 0.0f;
                        iz = fabsf(pd) / fabsf(D);
                    }
                    prm[j] = make_float4(D, wc, iz, 0.0f);
                    down += __popc(__ballot_sync(0xffffffffu, D < 0.0f));
                }
                __syncwarp();
                // the face with the lower axial coordinate: the lower slab face when the line rises with p
                const bool up = pd > 0.0f;
                if (inside) {
                    column_lines<false>(s, prm, 0, down, zA, up ? t_hi : t_lo, up ? t_lo : t_hi, fq, nz);
                    column_lines<false>(s, prm, down, cnt, zA, up ? t_lo : t_hi, up ? t_hi : t_lo, fq, nz);
                } else {
                    column_lines<true>(s, prm, 0, down, zA, up ? t_hi : t_lo, up ? t_lo : t_hi, fq, nz);
                    column_lines<true>(s, prm, down, cnt, zA, up ? t_lo : t_hi, up ? t_hi : t_lo, fq, nz);
                }
            }
        }
        // the cells into the image, and back to zero
        const bool tview = !xdom && vt.ptr != nullptr;
        const int64_t st_p = tview ? vt.st[1] : (xdom ? v.st[0] : v.st[1]);
        const int64_t st_q = tview ? vt.st[0] : (xdom ? v.st[1] : v.st[0]);
        const int64_t st_z = tview ? vt.st[2] : v.st[2];
        float *im = tview ? vt.ptr : v.ptr;
        float *imA = im + ip * st_p + (int64_t)(okA ? cq1 : 0) * st_q, *imB = im + ip * st_p + (int64_t)(okB ? cq2 : 0) * st_q;
        for (int r = 0; r < nz; ++r) {
            const float a = s[r * 32], b = s[(nz + r) * 32];
            s[r * 32] = 0.0f;
            s[(nz + r) * 32] = 0.0f;
            if (okA && a != 0.0f) atomicAdd(imA + r * st_z, 2.0f * a);
            if (okB && b != 0.0f) atomicAdd(imB + r * st_z, 2.0f * b);
        }
    }
}

// Columns shorter than this on average go line by line: a column pair costs a tile ~1,300 instructions
// to write its cells out, as much as ~11 lines of the line-by-line form.
constexpr int kMinMembers = 4;
constexpr int64_t kMaxRows = 1 << 20;
constexpr int kMaxCellBytes = 224 * 1024;

static int emap_args(const float *table, int32_t n_blocks, int32_t m, float *emap, const int64_t st[3], float *emap_t,
                     const int64_t st_t[3], const int32_t grid[3], const float center[3], const float size[3], Grid &g,
                     View &v, View &vt) {
    int rc;
    if (!table) return fail(SRF_EINVAL, "crystal_table must not be NULL");
    if (n_blocks <= 0 || m <= 0) return fail(SRF_EINVAL, "n_blocks and m must be positive");
    if ((rc = check_geometry(grid, center, size, g))) return rc;
    if ((rc = check_view(emap, st, g, "emap", v, true))) return rc;
    return check_view(emap_t, st_t, g, "emap_t", vt, false);
}

}  // namespace srf

using namespace srf;

extern "C" int srf_emap_block_full(const float *crystal_table, int32_t n_blocks, int32_t m,
                                   float *emap, const int64_t emap_strides[3], float *emap_t,
                                   const int64_t emap_t_strides[3], const int32_t grid[3],
                                   const float center[3], const float size[3], void *stream) {
    Grid g; View v, vt; int rc;
    if ((rc = emap_args(crystal_table, n_blocks, m, emap, emap_strides, emap_t, emap_t_strides, grid, center, size, g, v, vt))) return rc;
    return fused_emap(crystal_table, n_blocks, m, g, v, vt, nullptr, (cudaStream_t)stream);
}

extern "C" int64_t srf_emap_workspace(int32_t n_blocks, int32_t m, const int32_t grid[3]) {
    const int64_t rows = (int64_t)(n_blocks > 0 ? n_blocks : 0) * (m > 0 ? m : 0);
    if (rows < 1 || rows > kMaxRows || !grid || (int64_t)grid[2] * 256 > kMaxCellBytes) return 0;
    return emap_words(rows) * 4;
}

extern "C" int srf_emap_block_full_ws(const float *crystal_table, int32_t n_blocks, int32_t m,
                                      float *emap, const int64_t emap_strides[3], float *emap_t,
                                      const int64_t emap_t_strides[3], const int32_t grid[3], const float center[3],
                                      const float size[3], void *workspace, int64_t workspace_bytes, void *stream) {
    Grid g; View v, vt; int rc;
    if ((rc = emap_args(crystal_table, n_blocks, m, emap, emap_strides, emap_t, emap_t_strides, grid, center, size, g, v, vt))) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    const int64_t need = srf_emap_workspace(n_blocks, m, grid);
    if (need == 0) return fused_emap(crystal_table, n_blocks, m, g, v, vt, nullptr, s);  // a size the columns do not serve
    if (!workspace) return fail(SRF_EINVAL, "workspace must not be NULL");
    if ((uintptr_t)workspace & 7) return fail(SRF_EINVAL, "workspace must be 8-byte aligned");
    if (workspace_bytes < need) return fail(SRF_ERANGE, "workspace of %lld bytes, %lld are needed", (long long)workspace_bytes, (long long)need);
    const int rows = n_blocks * m, slots = (int)emap_slots(rows);
    EmapCols c = emap_cols(static_cast<int32_t *>(workspace), rows);
    k_cols_clear<<<grid_for(k_cols_clear, slots, 256), 256, 0, s>>>(c, slots, rows);
    k_cols_insert<<<grid_for(k_cols_insert, rows, 256), 256, 0, s>>>(crystal_table, c, slots, rows);
    k_cols_offsets<<<1, 1024, 0, s>>>(c, slots, rows, kMinMembers);
    k_cols_collect<<<grid_for(k_cols_collect, rows, 256), 256, 0, s>>>(crystal_table, c, rows);
    k_cols_sort<<<grid_for(k_cols_sort, rows, 1, 0, 64), 64, 0, s>>>(c);
    if ((rc = check_cuda("emap column launches"))) return rc;
    const int smem = g.nz * 256;
    if (smem > 32 * 1024) cudaFuncSetAttribute(k_emap_columns, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    const int tiles = ((g.nx > g.ny ? g.nx : g.ny) + 31) / 32;
    // at most rows (rows - 1) / 2 column pairs; the kernel reads how many there are
    const int64_t items = (int64_t)rows * (rows - 1) / 2 * tiles;
    k_emap_columns<<<grid_for(k_emap_columns, items, 1, smem, 32), 32, smem, s>>>(c, g, v, vt, tiles);
    if ((rc = check_cuda("emap column kernel launch"))) return rc;
    return fused_emap(crystal_table, n_blocks, m, g, v, vt, c.meta + 1, s);
}
