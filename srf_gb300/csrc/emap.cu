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
    float *zu, *fz;            // [rows] members' z as collected, and their axial coordinates (voxels) sorted by column
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
    c.fz = reinterpret_cast<float *>(ws); ws += rows;
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

// Each column's members by z, ascending (rank by counting), as axial coordinates in voxels.
__global__ void k_cols_sort(EmapCols c, Grid g) {
    if (!c.meta[1]) return;
    const GridK k = make_gridk<false>(g, TofParams{0, 0, 0});
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
            c.fz[lo + rank] = __fdiv_rn(__fdiv_rn(__fsub_rn(z, g.cz), k.dx_), k.dz) + k.nz2;
        }
    }
}

// ---------------------------------------------------------------- lines between two columns
constexpr int kParams = 64;  // members of the second column whose line constants are held at a time
constexpr int kWindow = 56;  // axial voxels of a lane's cells

// Line constants: D the axial extent in voxels, wc the weight of a whole slab, iz = 1 / |axial step per
// slab|, nwc = -wc. Lines that rise and lines that fall with the slab's first face are two runs; a
// run of cnt lines, ascending in D, is dealt to groups of four, line j to place 4 (j mod q) + j / q,
// q = cnt / 4, so that a group's lines end a quarter of the run apart; the last cnt mod 4 lines form
// a group of their own, padded with lines of weight 0.
struct LineParams {
    float D[kParams + 8], wc[kParams + 8], iz[kParams + 8], nwc[kParams + 8];
};

// The lines of one run (groups of four from place g0) from one member (axial face coordinate zA,
// relative to the lane's window), on one slab per lane. ta, tb: the slab's two faces along the line (0
// at zA, 1 at the other end), the one with the lower axial coordinate first. fq: fraction of the slab
// before its in-plane crossing. Cells: the lane's words s[c * 32] of the first in-plane cell and
// s[(kWindow + c) * 32] of the second. Slots and weights as lean_slab's, without its range tests:
// every voxel lies in the window, and what lies outside the image is not written out.
__device__ __forceinline__ void column_lines(float *s, const LineParams &prm, int g0, int groups, float zA, float ta,
                                             float tb, float fq) {
    constexpr unsigned cA = 0u - (unsigned)kFloorBits * 32u, dB = (unsigned)kWindow * 32u;
    const float2 one_m = make_float2(-1.0f, -1.0f), magic = make_float2(kFloorMagic, kFloorMagic);
    const float2 magic_m = make_float2(-kFloorMagic, -kFloorMagic);
    const float2 zA2 = make_float2(zA, zA), ta2 = make_float2(ta, ta), tb2 = make_float2(tb, tb), fq2 = make_float2(fq, fq);
    for (int g = 0; g < groups; ++g) {
        const int at = g0 + 4 * g;
        const float4 D4 = *reinterpret_cast<const float4 *>(prm.D + at), wc4 = *reinterpret_cast<const float4 *>(prm.wc + at);
        const float4 iz4 = *reinterpret_cast<const float4 *>(prm.iz + at), nw4 = *reinterpret_cast<const float4 *>(prm.nwc + at);
        const float2 D_[2] = {{D4.x, D4.y}, {D4.z, D4.w}}, wc_[2] = {{wc4.x, wc4.y}, {wc4.z, wc4.w}};
        const float2 iz_[2] = {{iz4.x, iz4.y}, {iz4.z, iz4.w}}, nw_[2] = {{nw4.x, nw4.y}, {nw4.z, nw4.w}};
        unsigned i0[4], i1[4], i2[4];
        float w0[4], w1[4], w2[4];
        int b1[4], b2[4];
#pragma unroll
        for (int h = 0; h < 2; ++h) {  // two lines at a time in packed FP32 arithmetic
            const float2 z1 = __ffma2_rn(D_[h], ta2, zA2), z2 = __ffma2_rn(D_[h], tb2, zA2);
            const float2 f1 = __fadd2_rd(z1, magic), f2 = __fadd2_rd(z2, magic);
            const float2 fr = __fmul2_rn(__ffma2_rn(z1, one_m, __fadd2_rn(f2, magic_m)), iz_[h]);
            b1[2 * h] = __float_as_int(f1.x); b1[2 * h + 1] = __float_as_int(f1.y);
            b2[2 * h] = __float_as_int(f2.x); b2[2 * h + 1] = __float_as_int(f2.y);
            const float2 fz = make_float2(f1.x != f2.x ? fr.x : 1.0f, f1.y != f2.y ? fr.y : 1.0f);
            const float2 a0 = __fmul2_rn(make_float2(fminf(fq, fz.x), fminf(fq, fz.y)), wc_[h]);
            const float2 a1 = __fmul2_rn(__ffma2_rn(fz, one_m, fq2), wc_[h]);  // > 0: the in-plane crossing is later
            const float2 a2 = __ffma2_rn(make_float2(fmaxf(fq, fz.x), fmaxf(fq, fz.y)), nw_[h], wc_[h]);
            w0[2 * h] = a0.x; w0[2 * h + 1] = a0.y;
            w1[2 * h] = a1.x; w1[2 * h + 1] = a1.y;
            w2[2 * h] = a2.x; w2[2 * h + 1] = a2.y;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            i0[k] = (unsigned)b1[k] * 32u + cA;
            i2[k] = (unsigned)b2[k] * 32u + (cA + dB);
            i1[k] = w1[k] > 0.0f ? i2[k] - dB : i0[k] + dB;
        }
        // A line's slots 0 and 1 are different cells, and slot 2 (both coordinates cross) a third. When
        // the group's lines use different voxels too, their additions overlap; else they run in order.
        if (__all_sync(0xffffffffu, b1[1] > b2[0] && b1[2] > b2[1] && b1[3] > b2[2])) {
            float a[4], b[4], c[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                a[k] = s[i0[k]];
                b[k] = s[i1[k]];
                c[k] = w2[k] != 0.0f ? s[i2[k]] : 0.0f;
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                s[i0[k]] = a[k] + w0[k];
                s[i1[k]] = b[k] + fabsf(w1[k]);
                if (w2[k] != 0.0f) s[i2[k]] = c[k] + w2[k];
            }
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float a = s[i0[k]], b = s[i1[k]];
                if (w2[k] != 0.0f) s[i2[k]] += w2[k];
                s[i0[k]] = a + w0[k];
                s[i1[k]] = b + fabsf(w1[k]);
            }
        }
    }
}

// The same lines straight into the image (imA, imB: the slab's two in-plane cells, null outside the
// image), with every range test: steep lines, and slabs beyond the columns.
__device__ __forceinline__ void column_lines_direct(const LineParams &prm, int g0, int groups, float zA, float ta, float tb,
                                                    float fq, int nz, int64_t st_z, float *imA, float *imB) {
    for (int j = g0; j < g0 + 4 * groups; ++j) {
        const float D = prm.D[j], wc = 2.0f * prm.wc[j];
        if (wc == 0.0f) continue;
        const float z1 = fminf(fmaxf(fmaf(D, ta, zA), -2097152.0f), 2097152.0f);
        const float z2 = fminf(fmaxf(fmaf(D, tb, zA), -2097152.0f), 2097152.0f);
        const float f1 = __fadd_rd(z1, kFloorMagic), f2 = __fadd_rd(z2, kFloorMagic);
        const int c1 = __float_as_int(f1) - kFloorBits, c2 = __float_as_int(f2) - kFloorBits;
        const float fz = c1 != c2 ? ((f2 - kFloorMagic) - z1) * prm.iz[j] : 1.0f;
        const bool qfirst = fq > fz;
        const bool B = (unsigned)c1 < (unsigned)nz, C = (unsigned)c2 < (unsigned)nz && c1 >= -1;
        const float w0 = fminf(fq, fz) * wc, w1 = fabsf(fq - fz) * wc, w2 = fmaf(-fmaxf(fq, fz), wc, wc);
        if (imA && B && w0 != 0.0f) atomicAdd(imA + c1 * st_z, w0);
        if (imA && qfirst && C && w1 != 0.0f) atomicAdd(imA + c2 * st_z, w1);
        if (imB && !qfirst && B && w1 != 0.0f) atomicAdd(imB + c1 * st_z, w1);
        if (imB && C && w2 != 0.0f) atomicAdd(imB + c2 * st_z, w2);
    }
}

// Last member (exclusive) of the piece that starts at member i: at most kParams members within `ext`
// axial voxels of it (z ascending).
__device__ __forceinline__ int piece_end(const float *fz, int i, int n, float ext, int lane) {
    const float z0 = fz[i];
    int e = i;
#pragma unroll
    for (int r = 0; r < kParams / 32; ++r) {
        const int j = i + lane + 32 * r;
        e += __popc(__ballot_sync(0xffffffffu, j < n && fz[min(j, n - 1)] - z0 <= ext));
    }
    return max(e, i + 1);
}

// One warp (= one block) takes one pair of columns A < B and one tile of 32 slabs, and of each column
// a piece at a time (at most kWindow - 4 voxels long). A line between two points lies between the
// lines through the pieces' ends, so on any slab the pieces' lines use at most kWindow voxels along
// the axis, from a first voxel of the slab's own: each lane owns a slab and holds its two in-plane
// cells (before and after the crossing) over that window in shared memory. The lines accumulate there
// without atomics, then the cells go to the image with one reduction per voxel, times two: the line
// from B to A is the line from A to B, and both are in the sum (a column with itself has no
// transaxial extent and is skipped by the short-LOR rule).
// Bound: instruction issue of column_lines, ~35 instructions per line and 32 slabs against ~120 of the
// line-by-line form, and half the lines. The window sets the warps an SM can hold: whole columns of
// cells (109 voxels: 28 KB a warp, 7 warps) ran at 51 % of the issue slots, 115 ms; kWindow 56 (14 KB,
// 13 warps) at 66 %, 85 ms, all on 32,448 crystals (624 columns of 52) and 200 x 200 x 109; line by line 308 ms.
__global__ void __launch_bounds__(32)
k_emap_columns(EmapCols c, Grid g, View v, View vt, int tiles) {
    __shared__ float s_cells[2 * kWindow * 32];
    __shared__ __align__(16) LineParams prm;
    if (!c.meta[1]) return;
    const int lane = threadIdx.x;
    const int cols = c.meta[0];
    const int64_t items = (int64_t)cols * (cols - 1) / 2 * tiles;
    const TofParams tp{0, 0, 0};
    const GridK k = make_gridk<false>(g, tp);
    const int nz = g.nz;
    const double rdx = (double)g.nx / g.sx, dx_dy = (double)g.ny / g.sy / rdx;  // 1 / voxel size, x per y voxel size
    float *s = s_cells + lane;
    for (int r = 0; r < 2 * kWindow; ++r) s[r * 32] = 0.0f;
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
        // The fraction before the crossing, from the lower face in 64 bits; the floors are the reference's. In FP32
        // its rounding was the image's error: line by line the two orders of a pair round independently, here one
        // counts twice (40 clinical columns: 1.29e-5 from 64 bits, line by line 1.19e-5, with this 1.5e-6). Once per
        // slab and column pair: 84.5 ms before, 84.3 ms with it. (The axial coordinate stays in FP32: on
        // steep lines the reference jumps at voxel faces, and its error does not show beside the fraction's.)
        float fq = 1.0f;
        if (cq1 != cq2) {
            const double u1 = ((double)(xdom ? pa.x : pa.y) - (xdom ? g.cx : g.cy)) * rdx;
            const double v1 = ((double)(xdom ? pa.y : pa.x) - (xdom ? g.cy : g.cx)) * rdx;
            const double k64 = ((double)(xdom ? pb.y : pb.x) - (xdom ? pa.y : pa.x)) / ((double)(xdom ? pb.x : pb.y) - (xdom ? pa.x : pa.y));
            const double lower = (v1 + k64 * ((double)(kq >= 0.0f ? pp1 : pp2) - u1)) * (xdom ? dx_dy : 1.0) + 0.5 * nq;
            fq = fminf(fmaxf((float)((double)cq2 - lower) * fabsf(dq / kq), 0.0f), 1.0f);
        }
        const bool okA = act && 0 <= cq1 && cq1 < nq, okB = act && 0 <= cq2 && cq2 < nq && cq1 >= -1;
        if (!__any_sync(0xffffffffu, okA || okB)) continue;
        const float t_lo = __fdiv_rn(__fsub_rn(pp1, p1), pd), t_hi = __fdiv_rn(__fsub_rn(pp2, p1), pd);
        const bool between = __all_sync(0xffffffffu, t_lo >= 0.0f && t_lo <= 1.0f && t_hi >= 0.0f && t_hi <= 1.0f);
        const int a0 = c.off[A], na = c.off[A + 1] - a0, b0 = c.off[B], nb = c.off[B + 1] - b0;
        const float *zA_ = c.fz + a0, *zB_ = c.fz + b0;
        // pieces of equal length, as few as fit
        const float extA = zA_[na - 1] - zA_[0], extB = zB_[nb - 1] - zB_[0];
        const float lenA = extA / fmaxf(ceilf(extA / (kWindow - 5.0f)), 1.0f) + 0.5f;
        const float lenB = extB / fmaxf(ceilf(extB / (kWindow - 5.0f)), 1.0f) + 0.5f;
        const float ku = 1.0f + kq * kq, ipd = 1.0f / pd;
        const bool up = pd > 0.0f;  // a line with D > 0 has its lower axial coordinate at the slab's lower face
        // views: cells (ip, cq1) and (ip, cq2)
        const bool tview = !xdom && vt.ptr != nullptr;
        const int64_t st_p = tview ? vt.st[1] : (xdom ? v.st[0] : v.st[1]);
        const int64_t st_q = tview ? vt.st[0] : (xdom ? v.st[1] : v.st[0]);
        const int64_t st_z = tview ? vt.st[2] : v.st[2];
        float *im = tview ? vt.ptr : v.ptr;
        float *imA = okA ? im + ip * st_p + (int64_t)cq1 * st_q : nullptr, *imB = okB ? im + ip * st_p + (int64_t)cq2 * st_q : nullptr;
        for (int ja = 0, ea; ja < na; ja = ea) {
            ea = piece_end(zA_, ja, na, lenA, lane);
            for (int jb = 0, eb; jb < nb; jb = eb) {
                eb = piece_end(zB_, jb, nb, lenB, lane);
                const int cnt = eb - jb;
                // the window's first voxel, and whether the window holds the pieces' lines: slabs between the
                // columns, at most one voxel of axial step per slab
                const float zA0 = zA_[ja], zB0 = zB_[jb], zA1 = zA_[ea - 1], zB1 = zB_[eb - 1];
                const float m = fminf(fmaf(zB0 - zA0, t_lo, zA0), fmaf(zB0 - zA0, t_hi, zA0));
                // (coordinates and extents below 2^13 keep their rounding far below the margin of 0.01)
                const float rise = fmaxf(fabsf(zB1 - zA0), fabsf(zB0 - zA1));
                const float base = floorf(m - 0.01f);
                const bool fast = between && __all_sync(0xffffffffu, rise * fabsf(ipd) <= 1.0f && rise < 8192.0f && fabsf(base) < 8192.0f);
                for (int ia = ja; ia < ea; ++ia) {
                    const float zA = zA_[ia];
                    __syncwarp();
                    // constants of the lines to this lane's members; falling lines (D < 0) come first
                    float D[kParams / 32], wc[kParams / 32];
                    int n_down = 0;
#pragma unroll
                    for (int r = 0; r < kParams / 32; ++r) {
                        const int j = lane + 32 * r;
                        D[r] = wc[r] = 0.0f;
                        if (j < cnt) {
                            const float d = zB_[jb + j] - zA;
                            const float kz = d * k.dz * ipd;
                            if (isfinite(d)) { D[r] = d; wc[r] = sqrtf(ku + kz * kz) * k.dx_; }
                        }
                        n_down += __popc(__ballot_sync(0xffffffffu, D[r] < 0.0f));
                    }
                    const int n_up = cnt - n_down, g_down = (n_down + 3) >> 2, g_up = (n_up + 3) >> 2;
#pragma unroll
                    for (int r = 0; r < kParams / 32; ++r) {
                        const int j = lane + 32 * r;
                        if (j < cnt) {
                            const bool first_run = j < n_down;
                            const int i = first_run ? j : j - n_down, q = (first_run ? n_down : n_up) >> 2;
                            const int quarter = (i >= q) + (i >= 2 * q) + (i >= 3 * q);
                            const int at = (first_run ? 0 : 4 * g_down) + (i < 4 * q ? 4 * (i - quarter * q) + quarter : i);
                            prm.D[at] = D[r];
                            prm.wc[at] = wc[r];
                            prm.nwc[at] = -wc[r];
                            prm.iz[at] = fabsf(pd) / fabsf(D[r]);
                        }
                    }
                    __syncwarp();
                    if (lane < 8) {  // the padding of both runs' last groups: the run's last line, weightless
                        const int n_run = lane < 4 ? n_down : n_up, rem = n_run & 3, run = lane < 4 ? 0 : 4 * g_down;
                        const int at = run + (n_run & ~3) + (lane & 3);
                        if (rem != 0 && (lane & 3) >= rem) {
                            prm.D[at] = prm.D[run + n_run - 1];
                            prm.wc[at] = prm.nwc[at] = prm.iz[at] = 0.0f;
                        }
                    }
                    __syncwarp();
                    const float t_dn = up ? t_hi : t_lo, t_up = up ? t_lo : t_hi;
                    if (fast) {
                        column_lines(s, prm, 0, g_down, zA - base, t_dn, t_up, fq);
                        column_lines(s, prm, 4 * g_down, g_up, zA - base, t_up, t_dn, fq);
                    } else {
                        column_lines_direct(prm, 0, g_down, zA, t_dn, t_up, fq, nz, st_z, imA, imB);
                        column_lines_direct(prm, 4 * g_down, g_up, zA, t_up, t_dn, fq, nz, st_z, imA, imB);
                    }
                }
                if (!fast) continue;
                // the cells into the image, and back to zero
                const int z0 = (int)base;
#pragma unroll 4
                for (int r = 0; r < kWindow; ++r) {
                    const float a = s[r * 32], b = s[(kWindow + r) * 32];
                    s[r * 32] = 0.0f;
                    s[(kWindow + r) * 32] = 0.0f;
                    const int z = z0 + r;
                    if ((unsigned)z >= (unsigned)nz) continue;
                    if (imA && a != 0.0f) atomicAdd(imA + z * st_z, 2.0f * a);
                    if (imB && b != 0.0f) atomicAdd(imB + z * st_z, 2.0f * b);
                }
            }
        }
    }
}

// Columns shorter than this on average go line by line: a column pair costs a tile ~1,300 instructions
// to set up and to write its cells out, as much as ~11 lines of the line-by-line form.
constexpr int kMinMembers = 4;
constexpr int64_t kMaxRows = 1 << 20;

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

extern "C" int64_t srf_emap_workspace(int32_t n_blocks, int32_t m) {
    const int64_t rows = (int64_t)(n_blocks > 0 ? n_blocks : 0) * (m > 0 ? m : 0);
    if (rows < 1 || rows > kMaxRows) return 0;
    return emap_words(rows) * 4;
}

extern "C" int srf_emap_block_full_ws(const float *crystal_table, int32_t n_blocks, int32_t m,
                                      float *emap, const int64_t emap_strides[3], float *emap_t,
                                      const int64_t emap_t_strides[3], const int32_t grid[3], const float center[3],
                                      const float size[3], void *workspace, int64_t workspace_bytes, void *stream) {
    Grid g; View v, vt; int rc;
    if ((rc = emap_args(crystal_table, n_blocks, m, emap, emap_strides, emap_t, emap_t_strides, grid, center, size, g, v, vt))) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    const int64_t need = srf_emap_workspace(n_blocks, m);
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
    k_cols_sort<<<grid_for(k_cols_sort, rows, 1, 0, 64), 64, 0, s>>>(c, g);
    if ((rc = check_cuda("emap column launches"))) return rc;
    const int tiles = ((g.nx > g.ny ? g.nx : g.ny) + 31) / 32;
    // at most rows (rows - 1) / 2 column pairs; the kernel reads how many there are
    const int64_t items = (int64_t)rows * (rows - 1) / 2 * tiles;
    k_emap_columns<<<grid_for(k_emap_columns, items, 1, 0, 32), 32, 0, s>>>(c, g, v, vt, tiles);
    if ((rc = check_cuda("emap column kernel launch"))) return rc;
    return fused_emap(crystal_table, n_blocks, m, g, v, vt, c.meta + 1, s);
}
