// Lean slab loop of the fused traversal: per-LOR constants folded so that a slab costs a few
// dozen instructions, and the image-box range tests run only for slabs near the box's faces.
//
// A LOR's slab ip is evaluated from its relative index pp = ip - ic (ic: the middle of the LOR's
// slab range). The in-plane coordinate q at the slab's two faces follows the reference's operand
// order (srfnef/cc/siddon/siddon.cu.cc:59-73; siddon_tof.cu.cc:77-90), so its floors and crossing
// fractions are the reference's. The axial coordinate z uses the linear form
//   z at the near / far face (ordered, zz1 <= zz2) = fma(Bz, pp, Z1) / fma(Bz, pp, Z2)
// with the reference's per-slab division folded into the constants (siddon.cu.cc:74-84), one FMA
// per face instead of an IEEE division. Floors come from
// one round-down add of 1.5 * 2^23: the sum's bit pattern is 0x4B400000 + floor(v) for
// |v| < 2^22, which feeds the offset multiply-adds directly (the bias is folded into the LOR's
// base offset) and compares for the crossing tests.
//
// The slab's (up to) three voxels, with fq, fz the fractions of the slab before the q and z
// crossings (1 when that coordinate does not cross):
//   slot 0  (cq1, cz1)                                   weight min(fq, fz)
//   slot 1  (cq1, cz2) if fq > fz else (cq2, cz1)          weight |fq - fz|
//   slot 2  (cq2, cz2)                                   weight 1 - max(fq, fz)
// Slot 1 is the far voxel when one coordinate crosses and the middle voxel when both do; slot 2
// is non-zero only when both cross. This is the reference's case analysis (siddon.cu.cc:86-189)
// without branches: its weights are ry/rz, (ry - rz) or (rz - ry), 1 - ry or 1 - rz.
//
// Exactness. The linear z form differs from the reference's value by a few units in the last
// place. A z floor can therefore differ when a face coordinate lies within ~1e-5 of an integer;
// the weight that moves between the two neighbouring voxels is then of the same order (the slab
// weight is continuous in the face coordinates), far below the 1e-5 relative L2 parity bound.
// (With the linear form for q as well, the fractions of LORs nearly parallel to the dominant axis
// carried that rounding divided by the small slope: the clinical backprojection drifted to
// 1.2e-5 relative L2 from the oracle.) Everything discontinuous
// is decided exactly, per LOR, in the reference's arithmetic: the skip rules, the dominant axis,
// the projector's endpoint slab range and the truncated TOF window (t2 <= nsigma^2).
//
// Range tests. Per LOR, [ilo, ihi] is the slab range whose face coordinates all lie at least
// kInteriorMargin inside the image box, so every candidate voxel is inside. Groups of slabs entirely
// within it skip the reference's range tests (siddon.cu.cc:88-189) and run up to four at a time
// without a branch between them, so that their instruction chains interleave; other groups run the
// tests one group at a time. A LOR whose coordinates step more than one voxel per slab (non-square
// voxels, steep LORs) has no interior, nor has one whose first endpoint lies more than kInteriorReach voxels
// away: its q faces round by 2^-24 of that distance in each of about five operations, a quarter of the margin
// at 8192 and an offset outside the image from about 1e6 on. Gathers and reductions are predicated on a
// non-zero weight.
//
// Interior groups work on two slabs per lane at a time in packed FP32 (one instruction, two
// independent roundings, each that of the scalar operation): the loop is bound by instruction issue.
// Their voxels follow from the first one by per-LOR strides, because a floor moves by at most one.
#pragma once
#include "fused.cuh"

namespace srf {

constexpr float kFloorMagic = 12582912.0f;   // 1.5 * 2^23
constexpr int kFloorBits = 0x4B400000;       // bit pattern of kFloorMagic
constexpr float kInteriorMargin = 0.01f;     // voxel units
constexpr float kInteriorReach = 8192.0f;    // voxel units

struct __align__(16) LeanRec {
    float invq, invz, Bz, Z1;     // 1/|q step|, 1/|z step| per slab; z faces: fma(Bz, pp, Z1 or Z2)
    float Z2, tS, tT, wc;         // TOF: exponent -(fma(tS, pp, tT))^2 in log2 units; wc with amplitude
    float invL2, yv, ad, nq2;
    float p1, q1, kq, dq;         // the q face coordinate in the reference's operand order
    float rdq, c1, c2, neg_zero;  // rdq = RN(1 / dq); pp + c1, pp + c2: faces of the lower and upper q (exact)
    int lo, hi, ic, flags;        // flags: F_VALID | F_PROJ | F_XDOM | F_TIE | F_HOT, its groups << kHotShift
    int ilo, ihi, plo, phi;       // interior slabs; the projector's slabs (empty when it skips the LOR)
    int base, sp, sq, sz;         // element offset of slab ic at the floor-bit origin (mod 2^32); strides
};
// F_HOT: the projector's slabs are all of the LOR's, interior, and fit one chunk of the kernel.
constexpr int F_HOT = 16, kHotShift = 8;
constexpr int kLeanVec = sizeof(LeanRec) / 16;
static_assert(sizeof(LeanRec) == 128, "LeanRec is eight 16-byte vectors");

__device__ __forceinline__ LeanRec load_lean(const LeanRec *src) {
    LeanRec R;
    const float4 *s4 = reinterpret_cast<const float4 *>(src);
    float4 *d4 = reinterpret_cast<float4 *>(&R);
#pragma unroll
    for (int c = 0; c < kLeanVec; ++c) d4[c] = s4[c];
    return R;
}

__device__ __forceinline__ void store_lean(LeanRec *dst, const LeanRec &R) {
    const float4 *s4 = reinterpret_cast<const float4 *>(&R);
    float4 *d4 = reinterpret_cast<float4 *>(dst);
#pragma unroll
    for (int c = 0; c < kLeanVec; ++c) d4[c] = s4[c];
}

// The truncated TOF kernel keeps slab ip when t2 <= nsigma^2, t2 in the reference's arithmetic
// (siddon_tof.cu.cc:55-58: xc, d2_tof, t2), as the oracle applies it.
__device__ __forceinline__ bool tof_keep(const LorRec &R, const GridK &k, int ip, int np_half, float dpc) {
    const float pc = __fmul_rn(__fadd_rn((float)(ip - np_half), 0.5f), dpc);
    const float d2 = __fmul_rn(__fsub_rn(div_exact(__fsub_rn(pc, R.p1), R.pd, R.rpd), R.ratio1), R.L);
    const float t2 = div_exact(__fmul_rn(d2, d2), k.expand, k.rexp);
    return t2 <= k.nsig2;
}

// [a, b] of real face positions f where A + B f stays within [m, n - m] (its FP32 rounding is far
// inside the margin m); rB = 1 / B.
__device__ __forceinline__ void face_interval(float A, float B, float rB, float n, float m, float &a, float &b) {
    if (B == 0.0f) {
        if (A >= m && A <= n - m) { a = -1e30f; b = 1e30f; } else { a = 1e30f; b = -1e30f; }
        return;
    }
    const float t1 = (m - A) * rB, t2 = (n - m - A) * rB;
    a = fminf(t1, t2);
    b = fmaxf(t1, t2);
}

// Lean record of a LOR from its setup record (lane-parallel, once per LOR). hot: slabs of one chunk of
// the kernel that walks it (0: no F_HOT), G: its lanes per LOR.
template <bool TOF, int G>
__device__ __forceinline__ LeanRec make_lean(const LorRec &R, const Grid &g, const GridK &k,
                                             const int64_t stx[3], const int64_t sty[3], bool have_t, int hot) {
    LeanRec E = {};
    E.flags = R.flags;
    E.yv = R.yv;
    E.ad = R.ad;
    E.invL2 = R.invL2;
    E.lo = R.lo;
    E.hi = R.hi;
    E.plo = 1;
    if (!(R.flags & F_VALID) || (R.flags & F_TIE)) return E;
    const bool xdom = R.flags & F_XDOM;
    const int np = xdom ? g.nx : g.ny, nq = xdom ? g.ny : g.nx;
    const float np2 = xdom ? k.nx2 : k.ny2;
    const int np_half = np / 2;
    const float dpc = xdom ? 1.0f : k.dy;
    // d(ip) = ((pc(ip) - p1) / pd - ratio1) L with pc(ip) = (ip - np/2 + 0.5) dpc is linear in ip
    const float tA = div_exact(dpc, R.pd, R.rpd) * R.L;
    int lo = R.lo, hi = R.hi;
    if (TOF && k.nsig2 > 0.0f && lo <= hi) {
        // exact truncated window: t2 <= nsigma^2 keeps an interval of slabs; estimate it (to a
        // slab) and settle both ends with the predicate itself
        const float tB = (((0.5f - (float)np_half) * dpc - R.p1) * R.rpd - R.ratio1) * R.L;
        const float rtA = __fdividef(1.0f, tA);
        const float half = k.nsw * fabsf(rtA);
        const float c = -tB * rtA;
        int a = (int)fmaxf(fminf(ceilf(c - half), (float)hi + 1.0f), (float)lo - 1.0f);
        int b = (int)fmaxf(fminf(floorf(c + half), (float)hi + 1.0f), (float)lo - 1.0f);
        for (int t = 0; t < 6 && a > lo && tof_keep(R, k, a - 1, np_half, dpc); ++t) --a;
        for (int t = 0; t < 6 && a <= b && !tof_keep(R, k, a, np_half, dpc); ++t) ++a;
        for (int t = 0; t < 6 && b < hi && tof_keep(R, k, b + 1, np_half, dpc); ++t) ++b;
        for (int t = 0; t < 6 && b >= a && !tof_keep(R, k, b, np_half, dpc); ++t) --b;
        lo = max(lo, a);
        hi = min(hi, b);
    }
    if (lo > hi) {
        E.flags = 0;
        return E;
    }
    E.lo = lo;
    E.hi = hi;
    const int ic = (lo + hi) >> 1;
    E.ic = ic;
    // z at face f (slab ip has faces ip and ip + 1): Az + Bz (f - np/2); at pp = ip - ic the
    // lower face is f = ip + (Bz < 0), the upper one f = ip + (Bz >= 0)
    const float icnp = __fsub_rn((float)ic, np2);  // exact
    const float s_lo = R.Bz < 0.0f ? 1.0f : 0.0f;
    E.Bz = R.Bz;
    E.Z1 = fmaf(R.Bz, icnp + s_lo, R.Az);
    E.Z2 = fmaf(R.Bz, icnp + (1.0f - s_lo), R.Az);
    E.invq = fabsf(R.rBq);
    E.invz = fabsf(R.rBz);
    E.wc = R.wc;
    E.p1 = R.p1;
    E.q1 = R.q1;
    E.kq = R.kq;
    E.dq = xdom ? k.dy : 1.0f;
    E.rdq = xdom ? k.rdy : 1.0f;
    E.c1 = icnp + (R.kq >= 0.0f ? 0.0f : 1.0f);
    E.c2 = icnp + (R.kq >= 0.0f ? 1.0f : 0.0f);
    E.nq2 = xdom ? k.ny2 : k.nx2;
    E.neg_zero = -0.0f;
    if (TOF) {
        // exponent of the Gaussian in log2 units: d(ip)^2 k2 = -(s d(ip))^2, s = sqrt(-k2), with
        // d = tA pp + d(ic), d(ic) in the reference's operand order
        const float s = sqrtf(-k.k2);
        const float pc = __fmul_rn(__fadd_rn((float)(ic - np_half), 0.5f), dpc);
        const float dic = __fmul_rn(__fsub_rn(div_exact(__fsub_rn(pc, R.p1), R.pd, R.rpd), R.ratio1), R.L);
        E.tS = tA * s;
        // NaN: a finite TOF value whose quotient by the voxel size overflowed (infinite in IEEE division); it lies
        // infinitely far from every slab
        E.tT = dic == dic ? dic * s : INFINITY;
    }
    // interior slabs: both faces of every slab within the box by the margin, in q and in z
    float qa, qb, za, zb;
    face_interval(R.Aq - R.Bq * np2, R.Bq, R.rBq, (float)nq, kInteriorMargin, qa, qb);
    face_interval(R.Az - R.Bz * np2, R.Bz, R.rBz, (float)g.nz, kInteriorMargin, za, zb);
    const float fa = fmaxf(qa, za), fb = fminf(qb, zb);   // faces f in [fa, fb]
    const float il = fmaxf(ceilf(fa), (float)lo), ih = fminf(floorf(fb) - 1.0f, (float)hi);
    // (an endpoint far away: the q faces of its LOR round by more than the margin)
    const bool inner = il <= ih && fabsf(R.Bq) <= 1.0f + 1e-5f && fabsf(R.Bz) <= 1.0f + 1e-5f &&
                       fmaxf(fabsf(R.p1), fabsf(R.q1)) * E.rdq <= kInteriorReach;
    E.ilo = inner ? (int)il : 1;
    E.ihi = inner ? (int)ih : 0;
    E.plo = (R.flags & F_PROJ) ? max(lo, R.pmlo) : 1;
    E.phi = (R.flags & F_PROJ) ? min(hi, R.pmhi) : 0;
    if (E.plo == lo && E.phi == hi && lo >= E.ilo && hi <= E.ihi && hi - lo < hot)
        E.flags |= F_HOT | (((hi - lo) / G + 1) << kHotShift);
    // element offset of (slab ic, floor bits 0x4B400000 + cq, 0x4B400000 + cz), modulo 2^32
    const int64_t *st = (!xdom && have_t) ? sty : stx;
    const uint32_t sp = (uint32_t)(xdom ? st[0] : st[1]);
    const uint32_t sq = (uint32_t)(xdom ? st[1] : st[0]);
    const uint32_t sz = (uint32_t)st[2];
    E.base = (int)((uint32_t)ic * sp - (uint32_t)kFloorBits * (sq + sz));
    E.sp = (int)sp;
    E.sq = (int)sq;
    E.sz = (int)sz;
    return E;
}

// Extents of the LOR's in-plane secondary and axial directions (the range tests').
struct LeanAxes {
    int32_t nq, nz;
};

__device__ __forceinline__ LeanAxes lean_axes(const LeanRec &E, const Grid &g) {
    return LeanAxes{(E.flags & F_XDOM) ? g.ny : g.nx, g.nz};
}

// float and float2 (two slabs, packed instructions) forms of the slab arithmetic
__device__ __forceinline__ float f_add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float f_mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float f_fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float f_add_rd(float a, float b) { return __fadd_rd(a, b); }
__device__ __forceinline__ float2 f_add(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 f_mul(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 f_fma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 f_add_rd(float2 a, float2 b) { return __fadd2_rd(a, b); }
template <typename T> __device__ __forceinline__ T f_all(float a);
template <> __device__ __forceinline__ float f_all<float>(float a) { return a; }
template <> __device__ __forceinline__ float2 f_all<float2>(float a) { return make_float2(a, a); }
template <typename T> constexpr int kParts = sizeof(T) / sizeof(float);
__device__ __forceinline__ float part(float a, int) { return a; }
__device__ __forceinline__ float part(float2 a, int i) { return i ? a.y : a.x; }
__device__ __forceinline__ void set_part(float &a, int, float v) { a = v; }
__device__ __forceinline__ void set_part(float2 &a, int i, float v) { if (i) a.y = v; else a.x = v; }
// A product that a following sum must not absorb: the compiler fuses a packed product and sum even where
// both are rounded explicitly (seen as q faces off by one rounding), so the packed product is an FMA with
// a -0 that the compiler cannot see.
__device__ __forceinline__ float f_mul_rounded(float a, float b, float) { return __fmul_rn(a, b); }
__device__ __forceinline__ float2 f_mul_rounded(float2 a, float2 b, float neg_zero) {
    return __ffma2_rn(a, b, make_float2(neg_zero, neg_zero));
}

// The slab's q face coordinate at pp + c in the reference's operand order (siddon.cu.cc:59-73:
// (q1 + kq (pp - p1)) / dq + nq2 at pp = ip - np/2 or ip - np/2 + 1), so that the q floors and crossing
// fractions are the reference's. QDIV: dq != 1 (non-square transaxial voxels, x-dominant LORs); the
// division is one Newton step from rdq = RN(1 / dq) (Markstein; a / 1 returns a unchanged).
template <bool QDIV, typename T>
__device__ __forceinline__ T q_face(const LeanRec &E, T pp, float c) {
    T t = f_add(f_all<T>(E.q1), f_mul_rounded(f_all<T>(E.kq), f_add(f_add(pp, f_all<T>(c)), f_all<T>(-E.p1)), E.neg_zero));
    if (QDIV) {
        const T q0 = f_mul(t, f_all<T>(E.rdq));
        const T r = f_fma(q0, f_all<T>(-E.dq), t);
        t = f_fma(r, f_all<T>(E.rdq), q0);
    }
    return f_add(t, f_all<T>(E.nq2));
}

// One slab near the image faces: the three slots' element offsets and weights (zero for a voxel the
// slab does not visit) under the reference's range tests. ipc = min(ip, hi); act = ip <= hi (an
// inactive lane contributes zero weight).
template <bool TOF, bool QDIV>
__device__ __forceinline__ void lean_slab(const LeanRec &E, const LeanAxes &ax, int ipc, bool act, int32_t o[3], float w[3]) {
    const float pp = (float)(ipc - E.ic);
    float wt = E.wc;
    if (TOF) {
        const float d = fmaf(E.tS, pp, E.tT);
        float ex;
        asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(ex) : "f"(-d * d));
        wt *= ex;
    }
    wt = act ? wt : 0.0f;
    const float qq1 = q_face<QDIV>(E, pp, E.c1), qq2 = q_face<QDIV>(E, pp, E.c2);
    const float zz1 = fmaf(E.Bz, pp, E.Z1), zz2 = fmaf(E.Bz, pp, E.Z2);
    const float fq1 = __fadd_rd(qq1, kFloorMagic), fq2 = __fadd_rd(qq2, kFloorMagic);
    const float fz1 = __fadd_rd(zz1, kFloorMagic), fz2 = __fadd_rd(zz2, kFloorMagic);
    const int bq1 = __float_as_int(fq1), bq2 = __float_as_int(fq2);
    const int bz1 = __float_as_int(fz1), bz2 = __float_as_int(fz2);
    const bool dq = bq1 != bq2, dz = bz1 != bz2;
    const float fq = dq ? ((fq2 - kFloorMagic) - qq1) * E.invq : 1.0f;
    const float fz = dz ? ((fz2 - kFloorMagic) - zz1) * E.invz : 1.0f;
    const bool qfirst = fq > fz;
    const float mn = fminf(fq, fz), mx = fmaxf(fq, fz);
    const float w0 = mn * wt, w1 = fabsf(fq - fz) * wt, w2 = fmaf(-mx, wt, wt);
    const uint32_t base = (uint32_t)E.base + (uint32_t)(ipc - E.ic) * (uint32_t)E.sp;
    const uint32_t t1 = (uint32_t)bz1 * (uint32_t)E.sz + base;
    const uint32_t t2 = (uint32_t)bz2 * (uint32_t)E.sz + base;
    const uint32_t oa = (uint32_t)bq2 * (uint32_t)E.sq + t1;   // (cq2, cz1)
    const uint32_t ob = (uint32_t)bq1 * (uint32_t)E.sq + t2;   // (cq1, cz2)
    // the reference's range tests (cq1 <= cq2, cz1 <= cz2): c in [0, n) as one unsigned compare
    const bool A = (unsigned)(bq1 - kFloorBits) < (unsigned)ax.nq;
    const bool B = (unsigned)(bz1 - kFloorBits) < (unsigned)ax.nz;
    const bool C = (unsigned)(bq2 - kFloorBits) < (unsigned)ax.nq;
    const bool D = (unsigned)(bz2 - kFloorBits) < (unsigned)ax.nz;
    const bool qm = bq1 >= kFloorBits - 1, zm = bz1 >= kFloorBits - 1;
    w[0] = A && B ? w0 : 0.0f;
    w[1] = (qfirst ? (A && D && zm) : (C && B && qm)) ? w1 : 0.0f;
    w[2] = C && D && qm && zm ? w2 : 0.0f;
    o[0] = (int32_t)((uint32_t)bq1 * (uint32_t)E.sq + t1);
    o[1] = (int32_t)(qfirst ? ob : oa);
    o[2] = (int32_t)((uint32_t)bq2 * (uint32_t)E.sq + t2);
}

// kParts<T> interior slabs of this lane (both faces inside the box, floors that move by at most one):
// pp and the element offset at the floor-bit origin of each; act_last: whether the last is the LOR's.
template <bool TOF, bool QDIV, typename T>
__device__ __forceinline__ void interior_slabs(const LeanRec &E, T pp, const uint32_t *base, bool act_last,
                                               int32_t (*o)[3], float (*w)[3]) {
    constexpr int P = kParts<T>;
    T wt = f_all<T>(E.wc);
    if (TOF) {
        const T d = f_fma(f_all<T>(E.tS), pp, f_all<T>(E.tT));
        const T dd = f_mul(d, d);
        T ex;
#pragma unroll
        for (int i = 0; i < P; ++i) {
            float v;
            asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(v) : "f"(-part(dd, i)));
            set_part(ex, i, v);
        }
        wt = f_mul(wt, ex);
    }
    set_part(wt, P - 1, act_last ? part(wt, P - 1) : 0.0f);
    const T qq1 = q_face<QDIV>(E, pp, E.c1), qq2 = q_face<QDIV>(E, pp, E.c2);
    const T zz1 = f_fma(f_all<T>(E.Bz), pp, f_all<T>(E.Z1)), zz2 = f_fma(f_all<T>(E.Bz), pp, f_all<T>(E.Z2));
    const T M = f_all<T>(kFloorMagic), Mn = f_all<T>(-kFloorMagic), one_m = f_all<T>(-1.0f);
    const T fq1 = f_add_rd(qq1, M), fq2 = f_add_rd(qq2, M), fz1 = f_add_rd(zz1, M), fz2 = f_add_rd(zz2, M);
    const T rq = f_mul(f_fma(qq1, one_m, f_add(fq2, Mn)), f_all<T>(E.invq));
    const T rz = f_mul(f_fma(zz1, one_m, f_add(fz2, Mn)), f_all<T>(E.invz));
    T fq, fz, mn, mx;
    uint32_t step_q[P], step_z[P];  // from the first voxel across the crossings there are
#pragma unroll
    for (int i = 0; i < P; ++i) {
        const bool dq = part(fq1, i) != part(fq2, i), dz = part(fz1, i) != part(fz2, i);
        const float a = dq ? part(rq, i) : 1.0f, b = dz ? part(rz, i) : 1.0f;
        step_q[i] = dq ? (uint32_t)E.sq : 0u;
        step_z[i] = dz ? (uint32_t)E.sz : 0u;
        set_part(fq, i, a);
        set_part(fz, i, b);
        set_part(mn, i, fminf(a, b));
        set_part(mx, i, fmaxf(a, b));
    }
    const T w0 = f_mul(mn, wt), w2 = f_fma(mx, f_mul(wt, one_m), wt);
    const T w1 = f_mul(f_fma(fz, one_m, fq), wt);  // > 0: slot 1 is (cq1, cz2), else (cq2, cz1)
#pragma unroll
    for (int i = 0; i < P; ++i) {
        const uint32_t o0 = (uint32_t)__float_as_int(part(fq1, i)) * (uint32_t)E.sq +
                            ((uint32_t)__float_as_int(part(fz1, i)) * (uint32_t)E.sz + base[i]);
        o[i][0] = (int32_t)o0;
        // a fraction can round to just above 1 (a crossing at the slab's far face): slot 1 or 2 then has a
        // weight of the order of that rounding, at a voxel that the slab touches
        o[i][1] = (int32_t)(o0 + (part(w1, i) > 0.0f ? step_z[i] : step_q[i]));
        o[i][2] = (int32_t)(o0 + step_z[i] + step_q[i]);
        w[i][0] = part(w0, i);
        w[i][1] = fabsf(part(w1, i));
        w[i][2] = part(w2, i);
    }
}

// N interior groups of G slabs from slab c0, the last one cut at whi (the others are whole).
template <bool TOF, int G, bool QDIV, int N>
__device__ __forceinline__ void interior_groups(const LeanRec &E, int c0, int whi, int lane, int32_t (*o)[3], float (*w)[3]) {
    const int ip = c0 + lane, last = ip + G * (N - 1);
    const bool act = last <= whi;
    const float pp0 = (float)(ip - E.ic);
    uint32_t base[N];
#pragma unroll
    for (int u = 0; u < N; ++u)
        base[u] = (uint32_t)E.base + (uint32_t)((u == N - 1 ? min(last, whi) : ip + G * u) - E.ic) * (uint32_t)E.sp;
    const float pp_last = fminf(pp0 + (float)(G * (N - 1)), (float)(whi - E.ic));
#pragma unroll
    for (int u = 0; u + 1 < N; u += 2) {
        const float2 pp = make_float2(pp0 + (float)(G * u), u + 2 == N ? pp_last : pp0 + (float)(G * (u + 1)));
        interior_slabs<TOF, QDIV, float2>(E, pp, base + u, u + 2 == N ? act : true, o + u, w + u);
    }
    if (N & 1) interior_slabs<TOF, QDIV, float>(E, pp_last, base + N - 1, act, o + N - 1, w + N - 1);
}

template <int N> struct Groups { static constexpr int value = N; };

// A walk over slabs [lo, hi] of a LOR with G lanes: f(o, w, Groups<N>) for every run of N <= U interior
// groups and every edge group.
template <bool TOF, int U, int G, bool QDIV, typename F>
__device__ __forceinline__ void lean_walk(const LeanRec &E, const LeanAxes &ax, int lo, int hi, int lane, F &&f) {
    static_assert(U >= 1 && U <= 4, "1 to 4 groups per run");
    int32_t o[U][3];
    float w[U][3];
    for (int c = lo; c <= hi;) {
        // whole interior groups from c (the last one may be cut at hi)
        const int n = c < E.ilo ? 0 : E.ihi >= hi ? (hi - c) / G + 1 : (E.ihi - c + 1) / G;
        if (n >= U) {
            interior_groups<TOF, G, QDIV, U>(E, c, hi, lane, o, w);
            f(o, w, Groups<U>());
            c += G * U;
        } else if (U > 3 && n == 3) {
            interior_groups<TOF, G, QDIV, (U > 3 ? 3 : 1)>(E, c, hi, lane, o, w);
            f(o, w, Groups<(U > 3 ? 3 : 1)>());
            c += G * 3;
        } else if (U > 2 && n == 2) {
            interior_groups<TOF, G, QDIV, (U > 2 ? 2 : 1)>(E, c, hi, lane, o, w);
            f(o, w, Groups<(U > 2 ? 2 : 1)>());
            c += G * 2;
        } else if (U > 1 && n == 1) {
            interior_groups<TOF, G, QDIV, 1>(E, c, hi, lane, o, w);
            f(o, w, Groups<1>());
            c += G;
        } else {
            const int ip = c + lane;
            lean_slab<TOF, QDIV>(E, ax, min(ip, hi), ip <= hi, o[0], w[0]);
            f(o, w, Groups<1>());
            c += G;
        }
    }
}

// The groups of one chunk [c0, whi] (whi - c0 < G U) with their range tests: offsets and weights of all
// at once, for a caller that needs them twice; groups past whi have zero weights.
template <bool TOF, int U, int G, bool QDIV>
__device__ __forceinline__ void edge_chunk(const LeanRec &E, const LeanAxes &ax, int c0, int whi, int lane,
                                           int32_t (&o)[U][3], float (&w)[U][3]) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int ip = c0 + G * u + lane;
        if (c0 + G * u > whi) {  // uniform over the group
            w[u][0] = w[u][1] = w[u][2] = 0.0f;
            o[u][0] = o[u][1] = o[u][2] = 0;
            continue;
        }
        lean_slab<TOF, QDIV>(E, ax, min(ip, whi), ip <= whi, o[u], w[u]);
    }
}

// Sum of im * w over the slots of N groups.
template <int N>
__device__ __forceinline__ float gather_slots(const float *__restrict__ im, const int32_t (*o)[3], const float (*w)[3], float acc) {
    float x[N][3];
#pragma unroll
    for (int u = 0; u < N; ++u)
#pragma unroll
        for (int c = 0; c < 3; ++c) x[u][c] = w[u][c] != 0.0f ? __ldg(im + o[u][c]) : 0.0f;
#pragma unroll
    for (int u = 0; u < N; ++u)
#pragma unroll
        for (int c = 0; c < 3; ++c) acc = fmaf(x[u][c], w[u][c], acc);
    return acc;
}

// *p += v in global memory. atomicAdd on a pointer whose address space the compiler cannot see (the
// several-study kernel reads its views from shared memory) tests the space of every reduction: 24 studies,
// 3.2e7 events, 4 subsets in the persistent kernel 26.7 -> 19.7 ms with this form; kernels that get their
// views as parameters are as before.
__device__ __forceinline__ void red_add(float *p, float v) {
#ifdef __CUDA_ARCH__
    asm volatile("red.global.add.f32 [%0], %1;" ::"l"(__cvta_generic_to_global(p)), "f"(v) : "memory");
#else
    atomicAdd(p, v);
#endif
}

// red_add where w != 0 (or NaN). Predicated: as a branch around the product and the reduction the compiler
// serialises a lane's slots (2e6 non-TOF LORs 1,705 us, TOF OSEM pass of 2e7 events 13.9 ms), with the
// products in front of the branches 1,335 us and 10.82 ms, predicated 1,323 us and 10.73 ms.
__device__ __forceinline__ void red_add_where(float w, float *p, float v) {
#ifdef __CUDA_ARCH__
    asm volatile("{.reg .pred q; setp.neu.f32 q, %2, 0f00000000; @q red.global.add.f32 [%0], %1;}"
                 ::"l"(__cvta_generic_to_global(p)), "f"(v), "f"(w) : "memory");
#else
    if (w != 0.0f) atomicAdd(p, v);
#endif
}

// Slots 0 and 1 of a group's G slabs go out as two accesses of G lanes, the first with both slots of the
// lower G / 2 slabs, the second with those of the upper ones: the slab after an in-plane crossing continues
// the row that the crossing slab's slot 1 begins, so that one instruction carries both into one
// 32-byte sector. As separate slot 0 and slot 1 accesses the L2's reduction sectors were the bound (181 M
// per 2e6 TOF LORs, 1.0 ms at the rate of coalesced ones): non-TOF backprojection of 2e6 LORs
// 2,136 -> 1,422 us. Gathers are not dealt anew: projection alone was 6 % slower with the two shuffles.
// The weight decides whether a slot is added, never the product: r may be infinite or NaN, and the offset
// of a slot without weight can lie outside the image. (Deciding by a product that is 0 for weight 0 was as
// sound and slower: 1,369 us and 11.16 ms; by an offset of -1 1,377 us and 11.06 ms.)
template <int G, int N>
__device__ __forceinline__ void scatter_slots(float *im, const int32_t (*o)[3], const float (*w)[3], float r, int lane) {
    const bool upper = lane & (G / 2);
    const unsigned m = group_mask<G>();
#pragma unroll
    for (int u = 0; u < N; ++u) {
        const int32_t ox = __shfl_xor_sync(m, o[u][1], G / 2, G);
        const float wx = __shfl_xor_sync(m, w[u][1], G / 2, G);
        const float wa = upper ? wx : w[u][0], wb = upper ? w[u][0] : wx;
        red_add_where(wa, im + (upper ? ox : o[u][0]), r * wa);
        red_add_where(wb, im + (upper ? o[u][0] : ox), r * wb);
        if (w[u][2] != 0.0f) red_add(im + o[u][2], r * w[u][2]);  // rare: both coordinates cross
    }
}

}  // namespace srf
