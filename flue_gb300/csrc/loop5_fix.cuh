// loop5_fix.cuh -- the lines, leaves and line cotangents of loop5.cuh and
// force.cu in fixed point (fix.cuh), for complex128 fields whose links are
// unitary.
//
// The 5-loop coefficients are n / 180 with n = 325, -11, 1, -32, 3 (from
// src/wloops.F90:219-224 with k5 = 1/180); a leaf is weighted by scaling one of
// its lines by n / 512 in fixed point, so that every weighted sum stays within
// +-1 and nothing is weighted afterwards.  What the sums are multiples of:
//   q   = (180/512) Q                       |q| <= 4 x 360/512 = 2.82
//   K   = (q - q^+) / 8 = (180/512) F       |K| <= 0.71   (stored)
//   Lam = (180/512)^2 (line cotangent of F)  |Lam| <= 11.9 (stored / 8)
// (norms are spectral; three planes through a direction at most).  F of a
// smooth field is small, and so would be the share of the 61 bits that K and
// everything after it uses: the cotangents take K 2^ks, ks from the largest
// |F|^2 of the time slice (of the lattice when a plane holds the time
// direction, kscale), such that |K 2^ks| <= 0.71 (Frobenius) still holds and
// the bounds above with it.  Relative gradient error at eps = 0.1 / 0.03: 7.0e-16 / 2.2e-15
// without ks (FP64: 5.1e-16).
#pragma once
#include "fix.cuh"
#include "loop5.cuh"

namespace flue {

// 512/180: Q = FXQ5 q of the 5-loop; the clover's only weight is 1
constexpr double FXQ5 = 512.0 / 180.0;

// weights n 2^20 of c_lw_w's shapes (row len - 1), as limbs of n / 512
static __constant__ int c_lw_n[3][3] = {{325 << 20, -(32 << 20), 3 << 20},
                                        {-(11 << 20), -(32 << 20), 0},
                                        {1 << 20, 3 << 20, 0}};

// line_site in fixed point; returns the state of the site's link (link_state)
template <class L>
__device__ __forceinline__ u32 line_site_fix(const L& U, const Geom& g, const Geom& gs, int t0, const PlaneArg& pa,
                                             const MatFix& lines, int64_t s, int slot) {
    const int d = sel(pa.dir, slot);
    int c[4];
    site_coords(g, s, c);
    int cd = 0, nd = 1;
    int64_t sd = 1;
#pragma unroll
    for (int k = 0; k < 4; ++k)
        if (k == d) cd = c[k], nd = g.n[k], sd = gs.st[k];
    const int64_t u = (int64_t)(t0 + c[0]) + c[1] * gs.st[1] + c[2] * gs.st[2] + c[3] * gs.st[3];
    const int64_t s1 = u + (int64_t)wrapd(cd, 1, nd) * sd;
    const int64_t s2 = u + (int64_t)wrapd(cd, 2, nd) * sd;
    const M3<double> ud = U.load(u, d);
    const M3F u0 = fx_of(ud);
    const u32 st = link_state(ud, u0);
    lines.store(s, 3 * slot, u0);
    const M3F l2 = fx_mm<false, false>(u0, fx_of(U.load(s1, d)));
    lines.store(s, 3 * slot + 1, l2);
    lines.store(s, 3 * slot + 2, fx_mm<false, false>(l2, fx_of(U.load(s2, d))));
    return st;
}

// Column b of q at one site and plane: the groups of fwd_q5 (kind 1), or the
// clover's one shape (kind 0).  Each leaf is a chain of matrices onto column b
// of its last line, which carries the leaf's weight.
template <typename I>
__device__ __forceinline__ FxVS fwd_q_fix(const Geom& g, const PlaneArg& pa, int kind, const MatFix& lines, int64_t s,
                                          const int c[4], int p, int b) {
    const int pmu = sel(pa.mu, p), pnu = sel(pa.nu, p);
    const Ctx cx = make_ctx(g, s, c, pmu, pnu, sel(pa.slot, pmu), sel(pa.slot, pnu));
    const int s0 = (int)cx.s, stm = (int)cx.stm, stn = (int)cx.stn;
    const int ng = kind == 1 ? 3 : 1;
    FxVS q = vs_zero();
    // TR and BL, grouped by the extent la along mu
#pragma unroll 1
    for (int la = 1; la <= ng; ++la) {
        const int km = cx.kmu + la - 1;
        const int mM = wrapd(cx.cm, -la, cx.nm) * stm, mP = wrapd(cx.cm, la, cx.nm) * stm;
        const int nb = kind == 1 ? (la == 1 ? 3 : 2) : 1;
        FxVS tr = vs_zero(), bl = vs_zero();
#pragma unroll 1
        for (int j = 0; j < nb; ++j) {
            const int lb = c_lw_w[la - 1][j], w = kind == 1 ? c_lw_n[la - 1][j] : 1 << 29;
            const int kn = cx.knu + lb - 1;
            const int nM = wrapd(cx.cn, -lb, cx.nn) * stn, nP = wrapd(cx.cn, lb, cx.nn) * stn;
            FxV t = fx_scaled(lines.col<true>((I)s0, kn, b), w);
            t = lines.mul<true>((I)(s0 + nP), km, t);
            lines.mac<false>(tr, (I)(s0 + mP), kn, t);
            t = fx_scaled(lines.col<false>((I)(s0 + nM), kn, b), w);
            t = lines.mul<false>((I)(s0 + mM + nM), km, t);
            lines.mac<true>(bl, (I)(s0 + mM + nM), kn, t);
        }
        lines.mac<false>(q, (I)s0, km, fx_of58(tr));
        lines.mac<true>(q, (I)(s0 + mM), km, fx_of58(bl));
    }
    // TL and BR, grouped by the extent lb along nu
#pragma unroll 1
    for (int lb = 1; lb <= ng; ++lb) {
        const int kn = cx.knu + lb - 1;
        const int nM = wrapd(cx.cn, -lb, cx.nn) * stn, nP = wrapd(cx.cn, lb, cx.nn) * stn;
        const int na = kind == 1 ? (lb == 1 ? 3 : 2) : 1;
        FxVS tl = vs_zero(), br = vs_zero();
#pragma unroll 1
        for (int j = 0; j < na; ++j) {
            const int la = c_lw_w[lb - 1][j], w = kind == 1 ? c_lw_n[lb - 1][j] : 1 << 29;
            const int km = cx.kmu + la - 1;
            const int mM = wrapd(cx.cm, -la, cx.nm) * stm, mP = wrapd(cx.cm, la, cx.nm) * stm;
            FxV t = fx_scaled(lines.col<false>((I)(s0 + mM), km, b), w);
            t = lines.mul<true>((I)(s0 + mM), kn, t);
            lines.mac<true>(tl, (I)(s0 + mM + nP), km, t);
            t = fx_scaled(lines.col<true>((I)s0, km, b), w);
            t = lines.mul<false>((I)(s0 + mP + nM), kn, t);
            lines.mac<false>(br, (I)(s0 + nM), km, t);
        }
        lines.mac<false>(q, (I)s0, kn, fx_of58(tl));
        lines.mac<true>(q, (I)(s0 + nM), kn, fx_of58(br));
    }
    return q;
}

// F = (Q - Q^+)/8 from those integers; fq = Q / q
__device__ __forceinline__ void fx_field_strength(const i64 d[9], double fq, double f[9]) {
    const double sc = fq * 0x1p-61;
#pragma unroll
    for (int e = 0; e < 9; ++e) f[e] = (double)d[e] * sc;
}
// -Re Tr F F
__device__ __forceinline__ double ah_norm2(const double f[9]) {
    double o = 0.0;
#pragma unroll
    for (int e = 3; e < 9; ++e) o = fma(f[e], f[e], o);
    return fma(2.0, o, fma(f[0], f[0], fma(f[1], f[1], f[2] * f[2])));
}

// kscale: the largest |F|^2 = -Re Tr F F seen per time slice, as the high word
// of the double (0 at the start); most sites read a value that is larger already
__device__ __forceinline__ void kscale_max(u32* kmax, double f2) {
    const u32 v = (u32)__double2hiint(f2);
    if (v > *(volatile u32*)kmax) atomicMax(kmax, v);
}
// ks >= 0 with 2^ks (180/512) |F| <= 0.71 for every |F|^2 < 2^(ex + 1)
__device__ __forceinline__ int kscale(const u32* kmax) {
    const int ex = (int)(*kmax >> 20) - 1023;
    return ex < -57 ? 29 : max(0, (1 - ex) >> 1);
}

// Column b of line_side in fixed point: C carries the weight w (n / 512 with
// the sign of the side), so t, B C, y and the two products with A do too
template <int SG, typename I>
__device__ __forceinline__ void line_side_fix(FxVS& acc, FxVS& X, int w, const MatFix& lines, const AHFix& kin, int p,
                                              int ks, I s, I Q, I off, int pf, int pB, int b) {
    constexpr bool DA = SG < 0, DC = SG > 0;
    const I R1 = Q + off, R2 = s + off;
    Fx kv[9];
    const FxV c = fx_scaled(lines.col<DC>(DC ? s : R2, pf, b), SG > 0 ? w : -w);
    const FxVP cp = fx_prep<true>(c);  // for B^+
    FxV t;
    {
        kin.load(R2, p, ks, kv);
        FxVP ck = cp;
#pragma unroll
        for (int k = 0; k < 3; ++k) ck.n[k] = fx_neg(cp.n[k]);
#pragma unroll
        for (int a = 0; a < 3; ++a) fx_rdot_limbs(t.r[a], t.i[a], ah_row(kv, a), ck);
    }
    const FxVP tp = fx_prep<true>(t);
    FxV bc;
    FxVS y = vs_zero();
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const FxR m = lines.row<true>(R2, pB, a);
        fx_rdot_limbs(bc.r[a], bc.i[a], m, cp);
        fx_rdot_add(y, a, m, tp);
    }
    kin.load(R1, p, ks, kv);
    fx_add_kv(y, kv, fx_prep<false>(bc));
    const FxVP xp = fx_prep<DA>(bc), yp = fx_prep<DA>(fx_of58(y));
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const FxR m = lines.row<DA>(DA ? R1 : Q, pf, a);
        fx_rdot_add(X, a, m, xp);
        fx_rdot_add(acc, a, m, yp);
    }
}

}  // namespace flue
