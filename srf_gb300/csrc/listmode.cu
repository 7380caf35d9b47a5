// List-mode ingestion on the GPU: crystal index <-> position, endpoint snapping, and
// histogramming into the triangular crystal-pair sinogram.
//
// * crystal index of a position: srfnef/functions/geometry/pet_ecat_scanner.py:15-60
//   (EcatCrystalPosToIndex): iblock = round(atan2(y, x) / angle_per_block) mod nb,
//   iring = floor((z + axial/2) / (gap + block_z)), iy = round(y_corr / unit_y - 0.5),
//   iz = round(z_corr / unit_z - 0.5); index = iy + iz*s1 + iblock*per_block + iring*per_ring.
//   With float32 positions numpy evaluates atan2, the block division and the ring floor in
//   float32 (Python scalars do not promote), the in-block offsets in float64 (int64 index times
//   a Python float), and rounds half to even; this code follows the same promotions.
// * position of an index: pet_ecat_scanner.py:63-89 (EcatIndexToCrystalPos), float64 then
//   rounded to float32, with numpy's floor-division/modulo semantics for the digit split.
// * snapping: srfnef/functions/data_transform/pet_ecat.py:43-60 (PetEcatListmodeTrans), TOF
//   column kept.
// * sinogram: srfnef/corrections/scattering/listmode2sinogram.py:17-23, 76-85 (change_id +
//   cal_sinogram): bin (hi - 1) * hi / 2 + lo of the ordered pair, float64 weights.
#include "common.cuh"

namespace srf {

struct EcatK {
    double avg_radius, angle_per_block, axial_length, gap, block_y, block_z, unit_y, unit_z;
    int64_t s1, s2, nb, per_block, per_ring, nb_crystals;
};

__device__ __forceinline__ int64_t floordiv(int64_t a, int64_t b) {
    int64_t q = a / b;
    if ((a % b != 0) && ((a < 0) != (b < 0))) --q;
    return q;
}

__device__ __forceinline__ int64_t pymod(int64_t a, int64_t b) { return a - floordiv(a, b) * b; }

__device__ __forceinline__ int64_t crystal_index(const EcatK &s, float x, float y, float z) {
    const float bq = __fdiv_rn(atan2f(y, x), (float)s.angle_per_block);
    const int64_t iblock = pymod((int64_t)rintf(bq), s.nb);
    const float zr = __fdiv_rn(__fadd_rn(z, (float)(s.axial_length / 2)), (float)(s.gap + s.block_z));
    const int64_t iring = (int64_t)floorf(zr);
    const double ang = (double)iblock * s.angle_per_block;
    const double y_corr = -(double)x * sin(ang) + (double)y * cos(ang) + s.block_y / 2;
    const int64_t iy = (int64_t)rint(y_corr / s.unit_y - 0.5);
    const double z_corr = (double)__fadd_rn(z, (float)(s.axial_length / 2)) - (double)iring * (s.block_z + s.gap);
    const int64_t iz = (int64_t)rint(z_corr / s.unit_z - 0.5);
    return iy + iz * s.s1 + iblock * s.per_block + iring * s.per_ring;
}

__device__ __forceinline__ void crystal_position(const EcatK &s, int64_t ind, float out[3]) {
    const int64_t iy = pymod(ind, s.s1);
    const int64_t iz = pymod(floordiv(ind, s.s1), s.s2);
    const int64_t iblock = pymod(floordiv(floordiv(ind, s.s1), s.s2), s.nb);
    const int64_t iring = floordiv(floordiv(floordiv(ind, s.s1), s.s2), s.nb);
    const double x0 = s.avg_radius;
    const double y0 = ((double)iy + 0.5) * s.unit_y - s.block_y / 2;
    const double th = s.angle_per_block * (double)iblock;
    out[0] = (float)(x0 * cos(th) - y0 * sin(th));
    out[1] = (float)(x0 * sin(th) + y0 * cos(th));
    out[2] = (float)(((double)iz + 0.5) * s.unit_z + (double)iring * (s.gap + s.block_z) - s.axial_length / 2);
}

// Per-block tables of the scanner in shared memory: sin and cos of every block's angle in double (the
// values crystal_index computes per event), their float roundings for the fast index, and the crystal
// centres: (x, y) of each (block, iy) and z of each (ring, iz), as crystal_position rounds them.
//
// What bounds the snap is FP64: this part issues about two FP64 lanes per clock and SM, and the direct
// form (sin, cos and two divisions per endpoint, then sin and cos again for the centre, and 64-bit
// integer divisions) took 942 us for 2e6 events, 56 times the 17 us their 112 MB need at the measured
// copy rate. The angles of a ring are nb values, so every block tabulates them once (one block of 32
// warps per SM: the prologue's FP64 is paid per block), endpoints are indexed in FP32 with a bound on
// the rounding and only the undecided ones (about 3e-4 of them) and the ones outside the detector
// take the direct form. Measured, 2e6 events on the clinical scanner: 945 -> 31 us a call (3.6 TB/s);
// 3,000 events 26.5 -> 24.8 us, most of it the call itself.
constexpr int kSnapBlock = 1024;
constexpr int kMaxTabFloats = 4608;  // 18 KB beside the 28 KB of staged rows (48 KB in all); clinical size needs 1,588

struct EcatTab {
    const double2 *sc;   // (sin, cos) of block b
    const float2 *scf;
    const float2 *xy;    // [iblock * s1 + iy]
    const float *z;      // [iring * s2 + iz]
    float apb, half_ax, pitch, block_y2, unit_y, unit_z, ru_y, ru_z;
    int s1, s2, nb, rings;
};

inline int64_t tab_floats(const EcatK &s, int64_t rings) {
    return s.nb * (4 + 2 + 2 * s.s1) + rings * s.s2;
}

// Every thread of the block takes part; ends with a block barrier.
__device__ __forceinline__ EcatTab build_tab(const EcatK &s, int rings, double2 *buf, bool centres) {
    EcatTab T;
    T.s1 = (int)s.s1; T.s2 = (int)s.s2; T.nb = (int)s.nb; T.rings = rings;
    T.apb = (float)s.angle_per_block;
    T.half_ax = (float)(s.axial_length / 2);
    T.pitch = (float)(s.gap + s.block_z);
    T.block_y2 = (float)(s.block_y / 2);
    T.unit_y = (float)s.unit_y;
    T.unit_z = (float)s.unit_z;
    T.ru_y = 1.0f / T.unit_y;
    T.ru_z = 1.0f / T.unit_z;
    float2 *scf = reinterpret_cast<float2 *>(buf + T.nb), *xy = scf + T.nb;
    float *z = reinterpret_cast<float *>(xy + T.nb * T.s1);
    for (int b = threadIdx.x; b < T.nb; b += blockDim.x) {
        const double ang = (double)b * s.angle_per_block;
        const double sn = sin(ang), cs = cos(ang);
        buf[b] = make_double2(sn, cs);
        scf[b] = make_float2((float)sn, (float)cs);
    }
    __syncthreads();
    if (centres) {
        for (int k = threadIdx.x; k < T.nb * T.s1; k += blockDim.x) {
            const int b = k / T.s1;
            const double2 t = buf[b];
            const double y0 = ((double)(k - b * T.s1) + 0.5) * s.unit_y - s.block_y / 2;
            xy[k] = make_float2((float)(s.avg_radius * t.y - y0 * t.x), (float)(s.avg_radius * t.x + y0 * t.y));
        }
        for (int k = threadIdx.x; k < rings * T.s2; k += blockDim.x) {
            const int r = k / T.s2;
            z[k] = (float)(((double)(k - r * T.s2) + 0.5) * s.unit_z + (double)r * (s.gap + s.block_z) - s.axial_length / 2);
        }
        __syncthreads();
    }
    T.sc = buf; T.scf = scf; T.xy = xy; T.z = z;
    return T;
}

// Digits (iblock, iy, iring, iz) of a position, or false when crystal_index has to be asked: a hit
// outside the detector (a gap, beyond the ends, not finite), or within the FP32 error of the border
// between two crystals. Block and ring follow crystal_index's float32 arithmetic operation for
// operation. The in-block offsets are FP32 here and double there: y_corr sums three terms of
// magnitude |x|, |y| and block_y / 2, each within 2^-23 relative of the double value (float sin / cos,
// one rounding per product and sum), so t = y_corr / unit - 0.5 is within 4 * 2^-23 (|x| + |y| +
// block_y / 2) / unit plus its own two roundings of the double one; the margin is twice that. z_corr
// alike with its two terms.
__device__ __forceinline__ bool fast_digits(const EcatTab &T, float x, float y, float z, int &ib, int &iy, int &ir, int &iz) {
    constexpr float kEps = 9.6e-7f;  // 8 * 2^-23
    const float bf = rintf(__fdiv_rn(atan2f(y, x), T.apb));
    if (!(fabsf(bf) < 1.0e6f)) return false;
    ib = (int)bf;
    ib += ib < 0 ? T.nb : 0;
    if (ib < 0 || ib > T.nb) return false;
    ib = ib == T.nb ? 0 : ib;
    const float zc = __fadd_rn(z, T.half_ax);
    const float rf = floorf(__fdiv_rn(zc, T.pitch));
    if (!(rf >= 0.0f && rf < (float)T.rings)) return false;
    ir = (int)rf;
    const float2 sc = T.scf[ib];
    const float ty = (-x * sc.x + y * sc.y + T.block_y2) * T.ru_y - 0.5f;
    const float tz = (zc - rf * T.pitch) * T.ru_z - 0.5f;
    const float qy = rintf(ty), qz = rintf(tz);
    const float my = kEps * ((fabsf(x) + fabsf(y) + T.block_y2) * T.ru_y + 1.0f + fabsf(ty));
    const float mz = kEps * ((fabsf(zc) + rf * T.pitch) * T.ru_z + 1.0f + fabsf(tz));
    if (!(fabsf(ty - qy) < 0.5f - my && fabsf(tz - qz) < 0.5f - mz)) return false;
    if (!(qy >= 0.0f && qy < (float)T.s1 && qz >= 0.0f && qz < (float)T.s2)) return false;
    iy = (int)qy;
    iz = (int)qz;
    return true;
}

__device__ __forceinline__ int64_t digits_index(const EcatK &s, int ib, int iy, int ir, int iz) {
    return iy + iz * s.s1 + ib * s.per_block + ir * s.per_ring;
}

// Index and (when POS) centre of an endpoint.
template <bool POS>
__device__ __forceinline__ int64_t snap_point(const EcatK &s, const EcatTab &T, float x, float y, float z, float p[3]) {
    int ib, iy, ir, iz;
    if (fast_digits(T, x, y, z, ib, iy, ir, iz)) {
        if (POS) {
            const float2 xy = T.xy[ib * T.s1 + iy];
            p[0] = xy.x; p[1] = xy.y; p[2] = T.z[ir * T.s2 + iz];
        }
        return digits_index(s, ib, iy, ir, iz);
    }
    const int64_t ind = crystal_index(s, x, y, z);
    if (POS) crystal_position(s, ind, p);
    return ind;
}

// PACKED: rows of exactly seven floats, 16-byte aligned, in and out. A warp moves its 32 rows (896
// bytes) as 56 16-byte accesses through shared memory, the next rows' loads issued before it works on
// the current ones; seven 4-byte accesses at a 28-byte stride per lane would cost the load-store
// unit as much time as DRAM. Lane l's row starts at word 7 l, which is free of bank conflicts.
template <bool PACKED>
__global__ void __launch_bounds__(kSnapBlock, 1)
k_snap(const float *__restrict__ lors, int64_t n, int stride, EcatK s, int rings, float *__restrict__ out, int out_stride,
       int64_t *__restrict__ ids) {
    extern __shared__ double2 s_tab[];
    __shared__ float4 s_rows[PACKED ? kSnapBlock / 32 : 1][56];
    const EcatTab T = build_tab(s, rings, s_tab, out != nullptr);
    const int lane = threadIdx.x & 31;
    auto put_ids = [&](int64_t i, int64_t a, int64_t b) {
        if (ids) {
            ids[2 * i] = a;
            ids[2 * i + 1] = b;
        }
    };
    if (PACKED) {
        float4 *buf = s_rows[threadIdx.x >> 5];
        float *row = reinterpret_cast<float *>(buf) + 7 * lane;
        const int64_t warps = (int64_t)gridDim.x * (kSnapBlock / 32);
        const int64_t full = n / 32;  // the last n % 32 rows are taken by the loop below
        const float4 *src = reinterpret_cast<const float4 *>(lors);
        float4 *dst = reinterpret_cast<float4 *>(out);
        int64_t w = (int64_t)(threadIdx.x >> 5) * gridDim.x + blockIdx.x;
        float4 v0 = {}, v1 = {};
        if (w < full) {
            v0 = src[w * 56 + lane];
            if (lane < 24) v1 = src[w * 56 + 32 + lane];
        }
        while (w < full) {
            buf[lane] = v0;
            if (lane < 24) buf[32 + lane] = v1;
            const int64_t nw = w + warps;
            if (nw < full) {
                v0 = src[nw * 56 + lane];
                if (lane < 24) v1 = src[nw * 56 + 32 + lane];
            }
            __syncwarp();
            float pa[3], pb[3];
            const int64_t a = snap_point<true>(s, T, row[0], row[1], row[2], pa);
            const int64_t b = snap_point<true>(s, T, row[3], row[4], row[5], pb);
            put_ids(w * 32 + lane, a, b);
            row[0] = pa[0]; row[1] = pa[1]; row[2] = pa[2];
            row[3] = pb[0]; row[4] = pb[1]; row[5] = pb[2];
            __syncwarp();
            dst[w * 56 + lane] = buf[lane];
            if (lane < 24) dst[w * 56 + 32 + lane] = buf[32 + lane];
            __syncwarp();
            w = nw;
        }
    }
    const int64_t first = PACKED ? n / 32 * 32 : 0;
    for (int64_t i = first + blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const float *l = lors + i * stride;
        float pa[3], pb[3];
        if (!out) {
            put_ids(i, snap_point<false>(s, T, l[0], l[1], l[2], pa), snap_point<false>(s, T, l[3], l[4], l[5], pb));
            continue;
        }
        const int64_t a = snap_point<true>(s, T, l[0], l[1], l[2], pa);
        const int64_t b = snap_point<true>(s, T, l[3], l[4], l[5], pb);
        put_ids(i, a, b);
        float *o = out + i * out_stride;
        o[0] = pa[0]; o[1] = pa[1]; o[2] = pa[2];
        o[3] = pb[0]; o[4] = pb[1]; o[5] = pb[2];
        for (int c = 6; c < out_stride && c < stride; ++c) o[c] = l[c];
    }
}

// The direct form of the snap, for scanners whose tables would not fit in shared memory.
__global__ void k_snap_direct(const float *__restrict__ lors, int64_t n, int stride, EcatK s,
                              float *__restrict__ out, int out_stride, int64_t *__restrict__ ids) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        const float *l = lors + i * stride;
        const int64_t a = crystal_index(s, l[0], l[1], l[2]);
        const int64_t b = crystal_index(s, l[3], l[4], l[5]);
        if (ids) {
            ids[2 * i] = a;
            ids[2 * i + 1] = b;
        }
        if (out) {
            float pa[3], pb[3];
            crystal_position(s, a, pa);
            crystal_position(s, b, pb);
            float *o = out + i * out_stride;
            o[0] = pa[0]; o[1] = pa[1]; o[2] = pa[2];
            o[3] = pb[0]; o[4] = pb[1]; o[5] = pb[2];
            for (int c = 6; c < out_stride && c < stride; ++c) o[c] = l[c];
        }
    }
}

// TAB: the endpoints are indexed as in k_snap (tables without the centres); else in the direct form.
template <bool TAB>
__global__ void k_lm2sino(const float *__restrict__ lors, int64_t n, int stride,
                          const float *__restrict__ values, EcatK s, int rings, double *__restrict__ sino,
                          int64_t n_bins, unsigned long long *__restrict__ dropped) {
    extern __shared__ double2 s_tab[];
    EcatTab T = {};
    if (TAB) T = build_tab(s, rings, s_tab, false);
    float unused[3];
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        const float *l = lors + i * stride;
        const int64_t a = TAB ? snap_point<false>(s, T, l[0], l[1], l[2], unused) : crystal_index(s, l[0], l[1], l[2]);
        const int64_t b = TAB ? snap_point<false>(s, T, l[3], l[4], l[5], unused) : crystal_index(s, l[3], l[4], l[5]);
        const int64_t hi = a > b ? a : b, lo = a > b ? b : a;
        const int64_t bin = (hi - 1) * hi / 2 + lo;
        if (lo >= 0 && hi < s.nb_crystals && bin >= 0 && bin < n_bins)
            atomicAdd(sino + bin, (double)(values ? values[i] : 1.0f));
        else if (dropped)
            atomicAdd(dropped, 1ULL);
    }
}

inline int make_ecat(const double p[8], const int64_t shape[3], EcatK &s) {
    for (int k = 0; k < 8; ++k)
        if (!std::isfinite(p[k])) return fail(SRF_ENONFINITE, "scanner parameter %d is not finite", k);
    if (shape[0] <= 0 || shape[1] <= 0 || shape[2] <= 0) return fail(SRF_EGRID, "bad scanner shape");
    s.avg_radius = p[0]; s.angle_per_block = p[1]; s.axial_length = p[2]; s.gap = p[3];
    s.block_y = p[4]; s.block_z = p[5]; s.unit_y = p[6]; s.unit_z = p[7];
    if (!(s.angle_per_block > 0) || !(s.unit_y > 0) || !(s.unit_z > 0) || !(s.gap + s.block_z > 0))
        return fail(SRF_EGRID, "scanner sizes must be positive");
    s.s1 = shape[0]; s.s2 = shape[1]; s.nb = shape[2];
    s.per_block = s.s1 * s.s2;
    s.per_ring = s.per_block * s.nb;
    return SRF_OK;
}

// Whether the tables of build_tab fit (the digits are then small integers too).
inline bool tables_fit(const EcatK &s, int64_t rings) {
    return rings > 0 && rings <= kMaxTabFloats && s.nb <= kMaxTabFloats && s.s1 <= kMaxTabFloats && s.s2 <= kMaxTabFloats &&
           tab_floats(s, rings) <= kMaxTabFloats;
}

}  // namespace srf

using namespace srf;

extern "C" {

int srf_listmode_snap(const float *lors, int64_t n, int32_t lor_stride, const double scanner[8],
                      const int64_t scanner_shape[4], float *out, int32_t out_stride,
                      int64_t *crystal_ids, void *stream) {
    int rc;
    if ((rc = check_lors(lors, n, lor_stride))) return rc;
    if (!scanner || !scanner_shape) return fail(SRF_EINVAL, "scanner must not be NULL");
    if (out && out_stride < 6) return fail(SRF_EINVAL, "out_stride %d < 6", out_stride);
    EcatK s;
    if ((rc = make_ecat(scanner, scanner_shape, s))) return rc;
    s.nb_crystals = s.per_ring * scanner_shape[3];
    if (n == 0) return ok();
    cudaStream_t st = (cudaStream_t)stream;
    if (!tables_fit(s, scanner_shape[3])) {
        unsigned blocks = grid_for(k_snap_direct, n, kBlock);
        k_snap_direct<<<blocks, kBlock, 0, st>>>(lors, n, lor_stride, s, out, out_stride, crystal_ids);
        return check_cuda("snap kernel launch");
    }
    const int smem = (int)tab_floats(s, scanner_shape[3]) * 4, rings = (int)scanner_shape[3];
    // one block of 32 warps per SM; fewer events get one warp per 32 of them, spread over the SMs
    const int64_t need = (n + 31) / 32;
    const unsigned blocks = (unsigned)(need < num_sms() ? need : num_sms());
    const bool packed = lor_stride == 7 && out_stride == 7 && out && (((uintptr_t)lors | (uintptr_t)out) & 15) == 0;
    if (packed) k_snap<true><<<blocks, kSnapBlock, smem, st>>>(lors, n, lor_stride, s, rings, out, out_stride, crystal_ids);
    else k_snap<false><<<blocks, kSnapBlock, smem, st>>>(lors, n, lor_stride, s, rings, out, out_stride, crystal_ids);
    return check_cuda("snap kernel launch");
}

int srf_lm2sino(const float *lors, int64_t n, int32_t lor_stride, const float *values,
                const double scanner[8], const int64_t scanner_shape[4], double *sino,
                int64_t n_bins, unsigned long long *dropped, void *stream) {
    int rc;
    if ((rc = check_lors(lors, n, lor_stride))) return rc;
    if (!scanner || !scanner_shape || !sino) return fail(SRF_EINVAL, "NULL argument");
    EcatK s;
    if ((rc = make_ecat(scanner, scanner_shape, s))) return rc;
    s.nb_crystals = s.per_ring * scanner_shape[3];
    if (n_bins < 0) return fail(SRF_EINVAL, "negative bin count");
    if (n == 0) return ok();
    cudaStream_t st = (cudaStream_t)stream;
    if (tables_fit(s, scanner_shape[3])) {
        const int smem = (int)tab_floats(s, scanner_shape[3]) * 4, rings = (int)scanner_shape[3];
        unsigned blocks = grid_for(k_lm2sino<true>, n, kBlock, smem);
        k_lm2sino<true><<<blocks, kBlock, smem, st>>>(lors, n, lor_stride, values, s, rings, sino, n_bins, dropped);
    } else {
        unsigned blocks = grid_for(k_lm2sino<false>, n, kBlock);
        k_lm2sino<false><<<blocks, kBlock, 0, st>>>(lors, n, lor_stride, values, s, 0, sino, n_bins, dropped);
    }
    return check_cuda("lm2sino kernel launch");
}

}  // extern "C"
