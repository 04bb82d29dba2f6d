// fix.cuh -- 3x3 complex arithmetic of unitary matrices in 60-bit fixed point
// on the integer multiply-add pipe.
//
// Why: an SM of this chip retires 2 FP64 multiply-adds per clock but 32
// integer ones of 32x32+64 bits (mad.wide.s32).  The entries of SU(3) matrices
// and of their products are bounded by 1, so a fixed-point number needs no
// exponent, and a real product is three integer multiply-adds.  With three
// real products a complex one instead of four (fx_dot), a matrix product takes
// 243 of them, 7.6 clocks of an SM a thread, against 108 FP64 multiply-adds,
// 54 clocks.
//
// Format: Fx = (h, l), both signed 32-bit, value h 2^-29 + l 2^-60, |value| < 4;
// l is balanced (-2^30 <= l < 2^30), which leaves a bit for the sum of two.
// Products: sum h h' accumulates in one 64-bit integer of unit 2^-58, the
// cross terms sum (h l' + l h') in another of unit 2^-89; l l' (below 2^-60 a
// term, of either sign) is dropped.  A matrix product is off by about 2e-18 an
// entry; its FP64 form by about 5e-17 where the entries are of order 1.
// Bounds: with a = |row of A| and b = |column of B| (Euclidean norms) the cross
// sums stay below 2.96 (a + b) 2^60 (Cauchy over the three terms of each of
// its four parts, the limbs of a sum of two counted twice), that is in 64 bits
// for a + b <= 2.70.  Every use below names the norms of its operands where
// they are not 1.
//
// Validity: the caller's matrices are only supposed to be unitary.  Whoever
// converts links counts those that are not (link_state) in a FixGate; kernels
// that follow run in fixed point when the gate is open and in FP64 otherwise,
// so any field gives the result it always gave.
#pragma once
#include "flue_common.cuh"

namespace flue {

using i64 = long long;
using u32 = unsigned int;

struct Fx {
    int h, l;
};

// an accumulator: hi of unit 2^-58, cr of unit 2^-89
struct FxAcc {
    i64 hi, cr;
};
// Starting value of a sum that becomes limbs: 2^28 of the main sum makes h round
// to nearest and l balanced, 2^30 of the cross sum rounds what the fold drops.
constexpr i64 FX_HI0 = (i64)1 << 28, FX_CR0 = (i64)1 << 30;

__device__ __forceinline__ void fx_mad(FxAcc& s, const Fx& a, const Fx& b) {
    s.hi += (i64)a.h * b.h;
    s.cr += (i64)a.h * b.l;
    s.cr += (i64)a.l * b.h;
}
// the sum of unit 2^-58 (its cross part holds the rounding)
__device__ __forceinline__ i64 fx_fold(const FxAcc& s) { return s.hi + (s.cr >> 31); }

// limbs of t - 2^28, t of unit 2^-58
__device__ __forceinline__ Fx fx_split(i64 t) {
    Fx r;
    r.h = (int)__funnelshift_r((u32)t, (u32)((unsigned long long)t >> 32), 29);
    r.l = (int)(((u32)t << 3) + 0x80000000u) >> 1;
    return r;
}
// limbs of a sum that started from (FX_HI0, FX_CR0)
__device__ __forceinline__ Fx fx_limbs(const FxAcc& s) { return fx_split(fx_fold(s)); }
// a 64-bit integer of unit 2^-58 as limbs (|value| < 4)
__device__ __forceinline__ Fx fx_of58(i64 s) { return fx_split(s + FX_HI0); }
// the same integer read in units of 2^-61: limbs of value / 8 (the last bit dropped)
__device__ __forceinline__ Fx fx_of61(i64 s) {
    Fx r;
    r.l = (int)(u32)s >> 1;
    r.h = (int)(s >> 32) + (int)((u32)s >> 31);
    return r;
}

// the value as one integer of unit 2^-60
__device__ __forceinline__ i64 fx_int60(const Fx& a) { return ((i64)a.h << 31) + a.l; }

// double to Fx, |x| < 2: the 53-bit significand shifted to unit 2^-60
// (truncated below it).  In integer instructions: every conversion from or to
// FP64 runs on the FP64 pipe, 64 cycles a warp.
__device__ __forceinline__ Fx fx_of(double x) {
    const u32 hw = (u32)__double2hiint(x), lw = (u32)__double2loint(x);
    // significand with its leading 1 at bit 63, then right by 1025 - exponent
    // (2 for |x| in [1, 2); the shift clamps at 64)
    const u32 mh = __funnelshift_l(lw, hw, 11) | 0x80000000u, ml = lw << 11;
    const u32 sh = (0x401fffffu - (hw & 0x7fffffffu)) >> 20;
    unsigned long long m = ((unsigned long long)mh << 32) | ml;
    asm("shr.u64 %0, %0, %1;" : "+l"(m) : "r"(sh));
    const i64 s = (i64)((int)hw >> 31);
    return fx_of61(((i64)m ^ s) - s);
}
// whether fx_of takes x: |x| < 2 (not for infinities and NaN)
__device__ __forceinline__ bool fx_takes(double x) {
    return ((u32)__double2hiint(x) & 0x7fffffffu) < 0x40000000u;
}

using M3F = M3<Fx>;   // a matrix in limbs
using M3S = M3<i64>;  // a sum of products, unit 2^-58

__device__ __forceinline__ M3F fx_of(const M3<double>& u) {
    M3F m;
#pragma unroll
    for (int k = 0; k < 9; ++k) m.r[k] = fx_of(u.r[k]), m.i[k] = fx_of(u.i[k]);
    return m;
}

__device__ __forceinline__ M3F fx_shfl_down(const M3F& p, int off) {
    M3F q;
#pragma unroll
    for (int e = 0; e < 9; ++e) {
        q.r[e] = {__shfl_down_sync(0xffffffffu, p.r[e].h, off), __shfl_down_sync(0xffffffffu, p.r[e].l, off)};
        q.i[e] = {__shfl_down_sync(0xffffffffu, p.i[e].h, off), __shfl_down_sync(0xffffffffu, p.i[e].l, off)};
    }
    return q;
}
__device__ __forceinline__ M3S s_zero() {
    M3S m;
#pragma unroll
    for (int k = 0; k < 9; ++k) m.r[k] = m.i[k] = 0;
    return m;
}
__device__ __forceinline__ M3F fx_of58(const M3S& s) {
    M3F m;
#pragma unroll
    for (int k = 0; k < 9; ++k) m.r[k] = fx_of58(s.r[k]), m.i[k] = fx_of58(s.i[k]);
    return m;
}
__device__ __forceinline__ M3F fx_of61(const M3S& s) {
    M3F m;
#pragma unroll
    for (int k = 0; k < 9; ++k) m.r[k] = fx_of61(s.r[k]), m.i[k] = fx_of61(s.i[k]);
    return m;
}

__device__ __forceinline__ Fx fx_add(const Fx& a, const Fx& b) { return {a.h + b.h, a.l + b.l}; }
__device__ __forceinline__ Fx fx_sub(const Fx& a, const Fx& b) { return {a.h - b.h, a.l - b.l}; }
__device__ __forceinline__ Fx fx_neg(const Fx& a) { return {-a.h, -a.l}; }

// One row of op(A) and the sums its complex products take.  With
// op(A) = ar + i sa ai and op(B) = br + i sb bi (sa, sb = -1 for a dagger),
//     k1 = ar (br + sb bi),  k2 = br (sa ai - ar),  k3 = -sb bi (ar + sa ai)
// give the real part k1 + k3 and the imaginary part k1 + k2: three real
// products, and both parts start from the shared sum of k1.
struct FxRow {
    Fx r[3], d[3], n[3];  // ar, sa ai - ar, -sb (ar + sa ai)
};
template <bool DA, bool DB>
__device__ __forceinline__ FxRow fx_row(const M3F& A, int a) {
    FxRow x;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const Fx re = DA ? A.r[3 * k + a] : A.r[3 * a + k], im = DA ? A.i[3 * k + a] : A.i[3 * a + k];
        x.r[k] = re;
        x.d[k] = DA ? fx_neg(fx_add(im, re)) : fx_sub(im, re);
        x.n[k] = DA == DB ? (DA ? fx_sub(re, im) : fx_neg(fx_add(re, im))) : (DA ? fx_sub(im, re) : fx_add(re, im));
    }
    return x;
}
// br + sb bi of every element
template <bool DB>
__device__ __forceinline__ void fx_sums(const M3F& B, Fx s[9]) {
#pragma unroll
    for (int k = 0; k < 9; ++k) s[k] = DB ? fx_sub(B.r[k], B.i[k]) : fx_add(B.r[k], B.i[k]);
}
// Real and imaginary part of column b of op(B) against the row; they start
// from cr0 and from hr, hi.
template <bool DB>
__device__ __forceinline__ void fx_dot(FxAcc& sr, FxAcc& si, const FxRow& x, const M3F& B, const Fx bs[9], int b,
                                       i64 hr, i64 hi, i64 cr0) {
    FxAcc k1 = {0, cr0};
#pragma unroll
    for (int k = 0; k < 3; ++k) fx_mad(k1, x.r[k], bs[DB ? 3 * b + k : 3 * k + b]);
    sr = {k1.hi + hr, k1.cr};
    si = {k1.hi + hi, k1.cr};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int e = DB ? 3 * b + k : 3 * k + b;
        fx_mad(sr, x.n[k], B.i[e]);
        fx_mad(si, x.d[k], B.r[e]);
    }
}

// op(A) op(B)
template <bool DA, bool DB>
__device__ __forceinline__ M3F fx_mm(const M3F& A, const M3F& B) {
    M3F C;
    Fx bs[9];
    fx_sums<DB>(B, bs);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const FxRow x = fx_row<DA, DB>(A, a);
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            FxAcc k1 = {FX_HI0, FX_CR0}, sr, si;
#pragma unroll
            for (int k = 0; k < 3; ++k) fx_mad(k1, x.r[k], bs[DB ? 3 * b + k : 3 * k + b]);
            sr = si = k1;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const int e = DB ? 3 * b + k : 3 * k + b;
                fx_mad(sr, x.n[k], B.i[e]);
                fx_mad(si, x.d[k], B.r[e]);
            }
            C.r[3 * a + b] = fx_limbs(sr);
            C.i[3 * a + b] = fx_limbs(si);
        }
    }
    return C;
}

// S += op(A) op(B)
template <bool DA, bool DB>
__device__ __forceinline__ void fx_mac(M3S& S, const M3F& A, const M3F& B) {
    Fx bs[9];
    fx_sums<DB>(B, bs);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const FxRow x = fx_row<DA, DB>(A, a);
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            FxAcc sr, si;
            fx_dot<DB>(sr, si, x, B, bs, b, S.r[3 * a + b], S.i[3 * a + b], FX_CR0);
            S.r[3 * a + b] = fx_fold(sr);
            S.i[3 * a + b] = fx_fold(si);
        }
    }
}

// a times the real number w 2^-29 (an exact limb)
__device__ __forceinline__ Fx fx_scaled(const Fx& a, int w) {
    const FxAcc s = {FX_HI0 + (i64)a.h * w, FX_CR0 + (i64)a.l * w};
    return fx_limbs(s);
}

// ---------------------------------------------------------------------------
// Columns.  Every chain of the 5-loop kernels is a product of matrices onto a
// column, so a thread carries one column b of a site (three threads a site, in
// three warps of a block): 3 of the 9 entries of each running product, a third
// of the registers, and matrices that are read a row at a time.
// ---------------------------------------------------------------------------
struct FxV {  // a column in limbs
    Fx r[3], i[3];
};
struct FxVS {  // a sum of columns, unit 2^-58
    i64 r[3], i[3];
};
__device__ __forceinline__ FxVS vs_zero() {
    FxVS v;
#pragma unroll
    for (int k = 0; k < 3; ++k) v.r[k] = v.i[k] = 0;
    return v;
}
__device__ __forceinline__ FxV fx_of58(const FxVS& s) {
    FxV v;
#pragma unroll
    for (int k = 0; k < 3; ++k) v.r[k] = fx_of58(s.r[k]), v.i[k] = fx_of58(s.i[k]);
    return v;
}
__device__ __forceinline__ FxV fx_scaled(const FxV& a, int w) {
    FxV v;
#pragma unroll
    for (int k = 0; k < 3; ++k) v.r[k] = fx_scaled(a.r[k], w), v.i[k] = fx_scaled(a.i[k], w);
    return v;
}
// A column ready to be multiplied by rows of op(M): with m = mr + i sm mi,
//     k1 = vr (mr + sm mi),  k2 = mr (vi - vr),  k3 = -sm mi (vr + vi)
// give the real part k1 + k3 and the imaginary part k1 + k2 of m v.
struct FxVP {
    Fx r[3], d[3], n[3];  // vr, vi - vr, -sm (vr + vi)
};
template <bool DM>
__device__ __forceinline__ FxVP fx_prep(const FxV& v) {
    FxVP x;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        x.r[k] = v.r[k];
        x.d[k] = fx_sub(v.i[k], v.r[k]);
        const Fx s = fx_add(v.r[k], v.i[k]);
        x.n[k] = DM ? s : fx_neg(s);
    }
    return x;
}
struct FxR {  // a row of op(M): mr, mi, mr + sm mi
    Fx r[3], i[3], s[3];
};
template <bool DM>
__device__ __forceinline__ void fx_row_sums(FxR& m) {
#pragma unroll
    for (int k = 0; k < 3; ++k) m.s[k] = DM ? fx_sub(m.r[k], m.i[k]) : fx_add(m.r[k], m.i[k]);
}
// (row) . (column), the main sums starting from hr and hi
__device__ __forceinline__ void fx_rdot(FxAcc& sr, FxAcc& si, const FxR& m, const FxVP& v, i64 hr, i64 hi) {
    FxAcc k1 = {0, FX_CR0};
#pragma unroll
    for (int k = 0; k < 3; ++k) fx_mad(k1, v.r[k], m.s[k]);
    sr = {k1.hi + hr, k1.cr};
    si = {k1.hi + hi, k1.cr};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        fx_mad(sr, v.n[k], m.i[k]);
        fx_mad(si, v.d[k], m.r[k]);
    }
}
// the same into limbs: both parts start from FX_HI0
__device__ __forceinline__ void fx_rdot_limbs(Fx& re, Fx& im, const FxR& m, const FxVP& v) {
    FxAcc sr = {FX_HI0, FX_CR0}, si;
#pragma unroll
    for (int k = 0; k < 3; ++k) fx_mad(sr, v.r[k], m.s[k]);
    si = sr;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        fx_mad(sr, v.n[k], m.i[k]);
        fx_mad(si, v.d[k], m.r[k]);
    }
    re = fx_limbs(sr);
    im = fx_limbs(si);
}
__device__ __forceinline__ void fx_rdot_add(FxVS& S, int a, const FxR& m, const FxVP& v) {
    FxAcc sr, si;
    fx_rdot(sr, si, m, v, S.r[a], S.i[a]);
    S.r[a] = fx_fold(sr);
    S.i[a] = fx_fold(si);
}

// Re Tr(op(A) op(B)), unit 2^-58; one cross sum per row of A
template <bool DA, bool DB>
__device__ __forceinline__ i64 fx_retr(const M3F& A, const M3F& B) {
    i64 t = 0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        FxAcc s = {0, FX_CR0};
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const int ea = DA ? 3 * k + a : 3 * a + k, eb = DB ? 3 * a + k : 3 * k + a;
            fx_mad(s, A.r[ea], B.r[eb]);
            fx_mad(s, (DA == DB) ? fx_neg(A.i[ea]) : A.i[ea], B.i[eb]);
        }
        t += fx_fold(s);
    }
    return t;
}
// Re (u . conj v) of two columns, unit 2^-58
__device__ __forceinline__ i64 fx_rezdot(const FxV& u, const FxV& v) {
    FxAcc s = {0, FX_CR0};
#pragma unroll
    for (int k = 0; k < 3; ++k) fx_mad(s, u.r[k], v.r[k]), fx_mad(s, u.i[k], v.i[k]);
    return fx_fold(s);
}
// Sum over a warp of integers |t| < 2^60 of unit 2^-58, in units of 2^-54
// (rounded once): three 22-bit parts by the warp's integer reduction.
__device__ __forceinline__ i64 warp_sum_fix54(i64 t) {
    const u32 m = (1u << 22) - 1;
    const u32 s0 = __reduce_add_sync(0xffffffffu, (u32)t & m);
    const u32 s1 = __reduce_add_sync(0xffffffffu, (u32)(t >> 22) & m);
    const int s2 = __reduce_add_sync(0xffffffffu, (int)(t >> 44));
    return ((i64)s2 << 40) + ((i64)s1 << 18) + ((s0 + 8) >> 4);
}

// ---------------------------------------------------------------------------
// the gate between the fixed-point and the FP64 kernels
// ---------------------------------------------------------------------------
struct FixGate {
    u32* p = nullptr;  // [0]: links not unitary or in a patch close to 1, [1]: links away from 1, [2]: blocks done
    u32 need = 0;      // open when [0] is 0 and [1] is at least this
    __device__ __forceinline__ bool open() const {
        return *(volatile const u32*)p == 0 && ((volatile const u32*)p)[1] >= need;
    }
};
// whether the FP64 kernels behind a gate have nothing to do (without a gate
// they always run)
__device__ __forceinline__ bool gate_shut(const FixGate& gt) { return gt.p && gt.open(); }
// A quarter of the links has to be further than 1/16 from 1 (Frobenius norm):
// closer to 1 the FP64 products keep more bits of the small off-diagonal and
// imaginary parts than fixed point does.  (A quarter: a gauge fixed along one
// direction has a quarter of its links at 1.)  And no four plaquettes around a
// site may lie within 1/16 (near_patch): F there is small, and its error absolute
// in fixed point.  Error of F in a region at a distance of 0.2 / 0.1 / 0.06 / 0.04 /
// 0.02 from 1, the rest of the field rough, in 2^-53 of its rms there: 5-loop 1.2 /
// 2.0 / 3.2 / 4.7 / 9.4 against 3.1 in FP64, clover 0.48 / 0.61 / 0.87 / 1.3 / 2.4
// against 1.8.
constexpr float FIX_FAR2 = 1.f / 256.f;
constexpr int GATE_WORDS = 3;  // zeroed before the counts

// |u - 1|^2 (Frobenius)
__device__ __forceinline__ float dist2_one(const float r[9], const float i[9]) {
    float d2 = 0.f;
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        const float x = r[k] - (k % 4 == 0 ? 1.f : 0.f);
        d2 = fmaf(x, x, d2);
        d2 = fmaf(i[k], i[k], d2);
    }
    return d2;
}

// what the counts of one link are: bit 0 = not unitary (or not finite), bit 1 =
// away from 1; f = fx_of(u)
__device__ __forceinline__ u32 link_state(const M3<double>& u, const M3F& f) {
    float r[9], i[9];
    bool ok = true;
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        ok = ok && fx_takes(u.r[k]) && fx_takes(u.i[k]);
        r[k] = (float)f.r[k].h * 0x1p-29f, i[k] = (float)f.i[k].h * 0x1p-29f;
    }
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = a; b < 3; ++b) {
            float re = 0.f, im = 0.f;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                re = fmaf(r[3 * a + k], r[3 * b + k], re);
                re = fmaf(i[3 * a + k], i[3 * b + k], re);
                im = fmaf(i[3 * a + k], r[3 * b + k], im);
                im = fmaf(-r[3 * a + k], i[3 * b + k], im);
            }
            // |U U^+ - 1| <= 2^-16 an element (fields stored in single precision
            // pass): the norm of a product of n links is then within n 2.3e-5 of 1
            ok = ok && fabsf(re - (a == b ? 1.f : 0.f)) <= 0x1p-16f && (a == b || fabsf(im) <= 0x1p-16f);
        }
    return (ok ? 0u : 1u) | (dist2_one(r, i) > FIX_FAR2 ? 2u : 0u);
}

__device__ __forceinline__ bool is_one(const M3<double>& u) {
    bool one = true;
#pragma unroll
    for (int k = 0; k < 9; ++k) one = one && u.r[k] == (k % 4 == 0 ? 1.0 : 0.0) && u.i[k] == 0.0;
    return one;
}

// Whether the twelve links of the four plaquettes in the plane (d, e) around the
// site at coordinates c are all close to 1.  For sites whose link along d is,
// rare in a rough field; most calls end with the first link, the one along e.
__device__ __forceinline__ bool near_patch(const FullLinks<double>& U, const Geom& g, const int c[4], int d, int e) {
    int64_t s = 0, fd = 0, bd = 0, fe = 0, be = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        s += c[k] * g.st[k];
        const int64_t f = c[k] + 1 == g.n[k] ? -(int64_t)(g.n[k] - 1) * g.st[k] : g.st[k];
        const int64_t b = c[k] == 0 ? (int64_t)(g.n[k] - 1) * g.st[k] : -g.st[k];
        if (k == d) fd = f, bd = b;
        if (k == e) fe = f, be = b;
    }
#pragma unroll 1
    for (int i = 0; i < 12; ++i) {
        const int k = (7 + 5 * i) % 12, j = k % 6;  // 6 links along d, 6 along e
        const bool along_e = k >= 6;
        const int back = j / 3, side = j % 3 - 1;
        const int64_t f = along_e ? fd : fe, b = along_e ? bd : be;
        const int64_t z = s + (back ? (along_e ? be : bd) : 0) + (side < 0 ? b : side > 0 ? f : 0);
        const M3F m = fx_of(U.load(z, along_e ? e : d));
        float re[9], im[9];
#pragma unroll
        for (int q = 0; q < 9; ++q) re[q] = (float)m.r[q].h * 0x1p-29f, im[q] = (float)m.i[q].h * 0x1p-29f;
        if (dist2_one(re, im) > FIX_FAR2) return false;
    }
    return true;
}

// add one warp's link states to the gate (all 32 lanes call; st = 0 for idle
// lanes); integer counts, so the result does not depend on the order.  Returns
// the lanes of bit 0 and of bit 1.
__device__ __forceinline__ uint2 gate_count(const FixGate& gt, u32 st) {
    const u32 bad = __ballot_sync(0xffffffffu, st & 1u), far = __ballot_sync(0xffffffffu, st & 2u);
    if ((threadIdx.x & 31) == 0) {
        if (bad) atomicAdd(gt.p, (u32)__popc(bad));
        if (far) atomicAdd(gt.p + 1, (u32)__popc(far));
    }
    return make_uint2(bad, far);
}

// Whether a warp has met something that shuts the gate, whatever the others find:
// what this one would still do is for nothing.  (The same answer in a whole warp.)
__device__ __forceinline__ bool gate_lost(const FixGate& gt) {
    return __any_sync(0xffffffffu, *(volatile const u32*)gt.p != 0);
}

// Whether this block is the last of n to come here (p[2] of the gate counts
// them); its partial sums and the others' are then visible to it.
__device__ __forceinline__ bool gate_last_block(const FixGate& gt, u32 n) {
    __shared__ bool last;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicAdd(gt.p + 2, 1u) == n - 1;
    }
    __syncthreads();
    if (last) __threadfence();
    return last;
}

// ---------------------------------------------------------------------------
// links and intermediates
// ---------------------------------------------------------------------------
// One matrix per (plane k, site s): 9 int4 units (h, l of the real and the
// imaginary part), 144 bytes, in tiles of 32 sites with the units unit-major
// (unit u of site s at tile + 32 u + s % 32), so that a warp's load of one
// unit is 512 contiguous bytes.
struct MatFix {
    int4* __restrict__ p;
    int64_t V;
    int nk = 0;  // planes, checked when > 0 (bounds-checked build)
    __device__ __forceinline__ bool ok(int64_t s, int k) const {
        return FLUE_INB(s >= 0 && s < V && k >= 0 && (nk == 0 || k < nk));
    }
    __device__ __forceinline__ int64_t unit0(int64_t s, int k) const {
        return ((int64_t)k * ((V + 31) >> 5) + (s >> 5)) * 288 + (s & 31);
    }
    __device__ __forceinline__ u32 unit0(u32 s, int k) const {
        return ((u32)k * (u32)((V + 31) >> 5) + (s >> 5)) * 288u + (s & 31u);
    }
    template <typename I>
    __device__ __forceinline__ M3F load(I s, int k) const {
        M3F m;
        if (!ok((int64_t)s, k)) {
#pragma unroll
            for (int e = 0; e < 9; ++e) m.r[e] = m.i[e] = {0, 0};
            return m;
        }
        const int4* q = p + unit0(s, k);
#pragma unroll
        for (int e = 0; e < 9; ++e) {
            const int4 v = q[32 * e];
            m.r[e] = {v.x, v.y};
            m.i[e] = {v.z, v.w};
        }
        return m;
    }
    // row a of op(M) with its sums, or column b (warp-uniform) of op(M)
    template <bool DM, typename I>
    __device__ __forceinline__ FxR row(I s, int k, int a) const {
        FxR m;
        const bool in = ok((int64_t)s, k);
        const int4* q = p + unit0(s, k);
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const int4 v = in ? q[32 * (DM ? 3 * j + a : 3 * a + j)] : make_int4(0, 0, 0, 0);
            m.r[j] = {v.x, v.y};
            m.i[j] = {v.z, v.w};
        }
        fx_row_sums<DM>(m);
        return m;
    }
    template <bool DM, typename I>
    __device__ __forceinline__ FxV col(I s, int k, int b) const {
        FxV c;
        const bool in = ok((int64_t)s, k);
        const int4* q = p + unit0(s, k) + 32 * (DM ? 3 * b : b);
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const int4 v = in ? q[32 * (DM ? j : 3 * j)] : make_int4(0, 0, 0, 0);
            c.r[j] = {v.x, v.y};
            c.i[j] = DM ? Fx{-v.z, -v.w} : Fx{v.z, v.w};
        }
        return c;
    }
    // op(M) v in limbs, and S += op(M) v
    template <bool DM, typename I>
    __device__ __forceinline__ FxV mul(I s, int k, const FxV& v) const {
        const FxVP x = fx_prep<DM>(v);
        FxV y;
#pragma unroll
        for (int a = 0; a < 3; ++a) fx_rdot_limbs(y.r[a], y.i[a], row<DM>(s, k, a), x);
        return y;
    }
    template <bool DM, typename I>
    __device__ __forceinline__ void mac(FxVS& S, I s, int k, const FxV& v) const {
        const FxVP x = fx_prep<DM>(v);
#pragma unroll
        for (int a = 0; a < 3; ++a) fx_rdot_add(S, a, row<DM>(s, k, a), x);
    }
    __device__ __forceinline__ void store(int64_t s, int k, const M3F& m) const {
        if (!ok(s, k)) return;
        int4* q = p + unit0(s, k);
#pragma unroll
        for (int e = 0; e < 9; ++e) q[32 * e] = make_int4(m.r[e].h, m.r[e].l, m.i[e].h, m.i[e].l);
    }
    __device__ __forceinline__ void store_el(int64_t s, int k, int e, const Fx& re, const Fx& im) const {
        if (ok(s, k)) p[unit0(s, k) + 32 * e] = make_int4(re.h, re.l, im.h, im.l);
    }
    static bool fits32(int64_t V, int64_t nk) { return (uint64_t)nk * (uint64_t)((V + 31) >> 5) * 288u < (1ull << 31); }
    static size_t bytes(int64_t V, int64_t nk) { return (size_t)nk * (size_t)((V + 31) >> 5) * 4608; }
};

// Anti-Hermitian K: 9 integers of unit 2^-61 in the order of AHAoS (Im K00,
// Im K11, Im K22, K01, K02, K12), as 4 units of two and 1 of one (72 bytes) in
// tiles of 32 sites; loaded as the limbs of K 2^ks
struct AHFix {
    longlong2* __restrict__ p;
    int64_t V;
    int nk = 0;
    __device__ __forceinline__ bool ok(int64_t s, int k) const {
        return FLUE_INB(s >= 0 && s < V && k >= 0 && (nk == 0 || k < nk));
    }
    __device__ __forceinline__ int64_t tile0(int64_t s, int k) const {
        return ((int64_t)k * ((V + 31) >> 5) + (s >> 5)) * 144;
    }
    __device__ __forceinline__ u32 tile0(u32 s, int k) const { return ((u32)k * (u32)((V + 31) >> 5) + (s >> 5)) * 144u; }
    template <typename I>
    __device__ __forceinline__ void load(I s, int k, int ks, Fx v[9]) const {
        if (!ok((int64_t)s, k)) {
            for (int e = 0; e < 9; ++e) v[e] = {0, 0};
            return;
        }
        const auto t = tile0(s, k);
        const longlong2* q = p + t + (s & 31);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const longlong2 x = q[32 * u];
            v[2 * u] = fx_of61(x.x << ks);
            v[2 * u + 1] = fx_of61(x.y << ks);
        }
        v[8] = fx_of61(reinterpret_cast<const i64*>(p + t + 128)[s & 31] << ks);
    }
    __device__ __forceinline__ void store(int64_t s, int k, const i64 v[9]) const {
        if (!ok(s, k)) return;
        const int64_t t = tile0(s, k);
        longlong2* q = p + t + (s & 31);
#pragma unroll
        for (int u = 0; u < 4; ++u) q[32 * u] = make_longlong2(v[2 * u], v[2 * u + 1]);
        reinterpret_cast<i64*>(p + t + 128)[s & 31] = v[8];
    }
    static bool fits32(int64_t V, int64_t nk) { return (uint64_t)nk * (uint64_t)((V + 31) >> 5) * 144u < (1ull << 31); }
    static size_t bytes(int64_t V, int64_t nk) { return (size_t)nk * (size_t)((V + 31) >> 5) * 2304; }
};

// row a of the anti-Hermitian K (its diagonal is imaginary)
__device__ __forceinline__ FxR ah_row(const Fx v[9], int a) {
    FxR m;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const Fx re = (a + c) == 1 ? v[3] : (a + c) == 2 ? v[5] : v[7];
        m.i[c] = (a == c) ? v[a] : (a + c) == 1 ? v[4] : (a + c) == 2 ? v[6] : v[8];
        m.r[c] = (a == c) ? Fx{0, 0} : a < c ? re : fx_neg(re);
    }
    fx_row_sums<false>(m);
    return m;
}
// column b (the same in a whole warp) of K
__device__ __forceinline__ FxV ah_col(const Fx v[9], int b) {
    FxV x;
    x.i[0] = b == 0 ? v[0] : b == 1 ? v[4] : v[6];
    x.i[1] = b == 0 ? v[4] : b == 1 ? v[1] : v[8];
    x.i[2] = b == 0 ? v[6] : b == 1 ? v[8] : v[2];
    x.r[0] = b == 0 ? Fx{0, 0} : b == 1 ? v[3] : v[5];
    x.r[1] = b == 0 ? fx_neg(v[3]) : b == 1 ? Fx{0, 0} : v[7];
    x.r[2] = b == 0 ? fx_neg(v[5]) : b == 1 ? fx_neg(v[7]) : Fx{0, 0};
    return x;
}
// S += K v
__device__ __forceinline__ void fx_add_kv(FxVS& S, const Fx k[9], const FxVP& v) {
#pragma unroll
    for (int a = 0; a < 3; ++a) fx_rdot_add(S, a, ah_row(k, a), v);
}

// the anti-Hermitian q - q^+ as 9 integers of q's unit, in the order of AHFix;
// q(e) is entry e = 3 a + b
template <class Q>
__device__ __forceinline__ void fx_antiherm(Q q, i64 d[9]) {
    d[0] = 2 * q(0).y;
    d[1] = 2 * q(4).y;
    d[2] = 2 * q(8).y;
    longlong2 u = q(1), l = q(3);
    d[3] = u.x - l.x;
    d[4] = u.y + l.y;
    u = q(2), l = q(6);
    d[5] = u.x - l.x;
    d[6] = u.y + l.y;
    u = q(5), l = q(7);
    d[7] = u.x - l.x;
    d[8] = u.y + l.y;
}

}  // namespace flue
