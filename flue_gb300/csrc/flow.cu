// flow.cu -- Luescher's Wilson flow (M. Luescher, JHEP 08 (2010) 071,
// appendix C) with the 3-stage Runge-Kutta integrator, in place on a device
// field.  No reference counterpart.
//
// Flow velocity: dV/dt = Z(V) V with Z = -g0^2 d S_w summed over oriented
// plaquettes, i.e. Z = 2 G where G = -1/2 TA(U N) is the su(3) gradient of
// sum_{x,mu<nu} Re Tr P (k_plaqforce in force.cu, Lie form).  One step with
// the low-storage form of the integrator:
//     Z0 = eps Z(W0);  W1 = exp(Z0/4) W0;                 B = Z0
//     Z1 = eps Z(W1);  X = 8/9 Z1 - 17/36 B; W2 = exp(X) W1; B = X
//     Z2 = eps Z(W2);  W3 = exp(3/4 Z2 - B) W2
// The update runs in the field's precision: D = exp(X) - I by the Taylor
// series summed in the basis {I, X, X^2} (expm1_ah below), scaled and squared
// for |X| > 1/2 (Moler & Van Loan, "Nineteen dubious ways to compute the
// exponential of a matrix", methods 3 and 8), then W' = W + D W.  Keeping the
// small D apart from I holds its relative precision in FP32, so the update
// adds one rounding of W per stage, as an FP64 update rounded to FP32 would.
// FP32 fields are reunitarised (FixSU3Matrix) after every stage.
#include <math.h>

#include <algorithm>

#include "flue_internal.h"

namespace flue {

size_t wflow_ws_min_bytes(const Geom& g) {
    // force (4 x 9 complex doubles per site), B (4 x 9 reals per site),
    // plaquette partials
    const size_t f = (size_t)36 * g.V * 16;
    const size_t b = (size_t)36 * g.V * 8;
    const size_t p = (size_t)plaqforce_blocks(g) * 4 * 8;
    return ((f + 255) & ~(size_t)255) + ((b + 255) & ~(size_t)255) + ((p + 255) & ~(size_t)255);
}

// the fixed-point step's scratch: a link field, X of the last stage, the gate
// (the FP64 step's buffers, used when the gate is shut, lie over the first two).
// The other link field of the stages is the caller's own: a converted link has the
// size of a complex128 one, and whole tiles of 32 sites fill it exactly; other
// lattices take a second one here (w1 > 0).  So the step needs no more memory
// than in FP64.
struct FlowFixWs {
    size_t w1, x, gate, total;
};
static FlowFixWs flow_fix_layout(const Geom& g) {
    FlowFixWs w;
    w.w1 = g.V % 32 ? MatFix::bytes(g.V, 4) : 0;
    w.x = w.w1 + MatFix::bytes(g.V, 4);
    w.gate = std::max(w.x + AHFix::bytes(g.V, 4), wflow_ws_min_bytes(g));
    w.total = w.gate + 256;
    return w;
}
size_t wflow_ws_bytes(const Geom& g, int prec) {
    return prec == PREC_C128 ? flow_fix_layout(g).total : wflow_ws_min_bytes(g);
}

template <typename T>
struct Cx {
    T re, im;
};
// Relative truncation tolerance of the series: a term whose bound
// |A|_F^k / k! is below tol |A|_F is dropped together with every later one
// (their sum is < 1.2 x the bound for |A|_F <= 1/2).
template <typename T>
__device__ __forceinline__ T exp_tol();
template <>
__device__ __forceinline__ float exp_tol<float>() {
    return 1.5e-8f;  // ~2^-26
}
template <>
__device__ __forceinline__ double exp_tol<double>() {
    return 2.8e-17;  // ~2^-55
}

// 1/k and 1/k!; at |A|_F <= 1/2 the series ends by k = 9 (FP32), 17 (FP64)
constexpr int EXP_TERMS = 24;
template <typename T>
struct ExpCoef {
    T inv[EXP_TERMS + 1], fact[EXP_TERMS + 1];
};
template <typename T>
constexpr ExpCoef<T> exp_coef() {
    ExpCoef<T> c{};
    double f = 1.0;
    c.inv[0] = c.fact[0] = T(1);
    for (int k = 1; k <= EXP_TERMS; ++k) {
        f *= k;  // exact to 22!, then rounded at 2^-53
        c.inv[k] = T(1.0 / k);
        c.fact[k] = T(1.0 / f);
    }
    return c;
}
static __constant__ ExpCoef<float> c_exp32 = exp_coef<float>();
static __constant__ ExpCoef<double> c_exp64 = exp_coef<double>();
template <typename T>
__device__ __forceinline__ const ExpCoef<T>& exp_table();
template <>
__device__ __forceinline__ const ExpCoef<float>& exp_table<float>() {
    return c_exp32;
}
template <>
__device__ __forceinline__ const ExpCoef<double>& exp_table<double>() {
    return c_exp64;
}

// exp(A) - I of an anti-Hermitian A (its upper triangle is read).
// Cayley-Hamilton, A^3 = t A^2 - m A + d I with t = tr A, m = (t^2 - tr A^2)/2,
// d = det A, gives A^k = p_k I + q_k A + r_k A^2 with (p, q, r)_{k+1} = (d r_k,
// p_k - m r_k, q_k + t r_k), so the Taylor series costs A^2 and scalar
// recurrences:
//     exp A - I = (sum_{k>=3} p_k/k!) I + (sum q_k/k!) A + (sum r_k/k!) A^2.
// A^2 is Hermitian, tr A^2 = -|A|_F^2 and m are real, t and d imaginary, which
// halves the work of the general form.  p_k, q_k, r_k are divided differences
// of x^k over the eigenvalues, bounded by k^2 |A|^(k-2), so the sum is stable at
// |A|_F <= 1/2; larger arguments are scaled by 2^-s and squared back s times
// as D <- 2 D + D D.
template <typename T>
__device__ __forceinline__ M3<T> expm1_ah(const M3<T>& x) {
    T d0 = x.i[0], d1 = x.i[4], d2 = x.i[8];
    Cx<T> b = {x.r[1], x.i[1]}, c = {x.r[2], x.i[2]}, e = {x.r[5], x.i[5]};
    auto abs2 = [](const Cx<T>& z) { return z.re * z.re + z.im * z.im; };
    T n2 = (d0 * d0 + d1 * d1 + d2 * d2) + T(2) * (abs2(b) + abs2(c) + abs2(e));
    T nrm = sqrt(n2);
    int sq = 0;
    if (nrm > T(0.5)) {
        T sc = T(1);
        while (nrm * sc > T(0.5) && sq < 60) {
            sc *= T(0.5);
            ++sq;
        }
        d0 *= sc, d1 *= sc, d2 *= sc;
        b = {b.re * sc, b.im * sc}, c = {c.re * sc, c.im * sc}, e = {e.re * sc, e.im * sc};
        nrm *= sc;
        n2 = nrm * nrm;
    }
    const T bb = abs2(b), cc = abs2(c), ee = abs2(e);
    // A^2: real diagonal, upper triangle
    const T q0 = -(d0 * d0 + bb + cc), q1 = -(d1 * d1 + bb + ee), q2 = -(d2 * d2 + cc + ee);
    const T s01 = d0 + d1, s02 = d0 + d2, s12 = d1 + d2;
    const Cx<T> S01 = {-s01 * b.im - (c.re * e.re + c.im * e.im), s01 * b.re - (c.im * e.re - c.re * e.im)};
    const Cx<T> S02 = {-s02 * c.im + (b.re * e.re - b.im * e.im), s02 * c.re + (b.re * e.im + b.im * e.re)};
    const Cx<T> S12 = {-s12 * e.im - (b.re * c.re + b.im * c.im), s12 * e.re - (b.re * c.im - b.im * c.re)};
    // t = i tau, d = i delta
    const T tau = d0 + d1 + d2, m = T(0.5) * (n2 - tau * tau);
    const Cx<T> be = {b.re * e.re - b.im * e.im, b.re * e.im + b.im * e.re};
    const T delta = d1 * cc + d2 * bb + d0 * ee - d0 * d1 * d2 - T(2) * (be.im * c.re - be.re * c.im);
    // terms k = 1, 2: A + A^2/2; state (p, q, r) of A^2
    const ExpCoef<T>& tab = exp_table<T>();
    Cx<T> w0 = {T(0), T(0)}, w1 = {T(1), T(0)}, w2 = {T(0.5), T(0)};
    Cx<T> p = {T(0), T(0)}, q = {T(0), T(0)}, r = {T(1), T(0)};
    T bnd = T(0.5) * n2;
    const T tol = exp_tol<T>() * nrm;
    for (int k = 3; k <= EXP_TERMS; ++k) {
        bnd *= nrm * tab.inv[k];
        if (!(bnd > tol)) break;
        const Cx<T> pn = {-delta * r.im, delta * r.re};
        const Cx<T> qn = {p.re - m * r.re, p.im - m * r.im};
        const Cx<T> rn = {q.re - tau * r.im, q.im + tau * r.re};
        p = pn;
        q = qn;
        r = rn;
        const T f = tab.fact[k];
        w0.re += f * p.re;
        w0.im += f * p.im;
        w1.re += f * q.re;
        w1.im += f * q.im;
        w2.re += f * r.re;
        w2.im += f * r.im;
    }
    M3<T> o;
    auto diag = [&](int k, T d, T qq) {
        o.r[k] = w0.re - w1.im * d + w2.re * qq;
        o.i[k] = w0.im + w1.re * d + w2.im * qq;
    };
    diag(0, d0, q0);
    diag(4, d1, q1);
    diag(8, d2, q2);
    // upper: w1 a + w2 S; lower: -w1 conj(a) + w2 conj(S)
    auto off = [&](int u, int l, const Cx<T>& a, const Cx<T>& S) {
        o.r[u] = (w1.re * a.re - w1.im * a.im) + (w2.re * S.re - w2.im * S.im);
        o.i[u] = (w1.re * a.im + w1.im * a.re) + (w2.re * S.im + w2.im * S.re);
        o.r[l] = (w2.re * S.re + w2.im * S.im) - (w1.re * a.re + w1.im * a.im);
        o.i[l] = (w2.im * S.re - w2.re * S.im) + (w1.re * a.im - w1.im * a.re);
    };
    off(1, 3, b, S01);
    off(2, 6, c, S02);
    off(5, 7, e, S12);
    for (int k = 0; k < sq; ++k) {
        M3<T> dd = mul(o, o);
        m_axpy(dd, T(2), o);
        o = dd;
    }
    return o;
}

template <typename T>
__device__ __forceinline__ M3<T> load_full(const void* links, int64_t V, int64_t s, int mu) {
    using C2 = typename V2<T>::type;
    if (!FLUE_INB(s >= 0 && s < V && mu >= 0 && mu < 4)) return m_zero<T>();
    const C2* q = (const C2*)links + s + V * mu;
    M3<T> m;
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            const C2 v = q[4 * V * (a + 3 * b)];
            m.r[3 * a + b] = v.x;
            m.i[3 * a + b] = v.y;
        }
    return m;
}

// Float-float accumulator of products: hi + lo holds the sum to ~2^-48
// (error-free products by fma, Knuth's two-sum; the _rn intrinsics keep the
// compiler from contracting them).
struct FF {
    float hi, lo;
};
__device__ __forceinline__ void ff_addprod(FF& s, float a, float b) {
    const float p = __fmul_rn(a, b);
    const float e = fmaf(a, b, -p);
    const float t = __fadd_rn(s.hi, p);
    const float bp = __fsub_rn(t, s.hi);
    const float err = __fadd_rn(__fsub_rn(s.hi, __fsub_rn(t, bp)), __fsub_rn(p, bp));
    s.hi = t;
    s.lo = __fadd_rn(s.lo, __fadd_rn(err, e));
}

// The same for sums that stay within +-2, in 4 instructions a product instead of
// 10: hi carries 6 + the sum, so it keeps one exponent, every step of it is a
// multiple of 2^-21 and known exactly, and what the step rounded off the product
// (below 2^-22) goes to lo.  The sum is good to about 2^-46 (2^-43 at worst), far
// below the one rounding of the result, where that is not much smaller than 1
// (reunitarise).  54 products a link: RK3 step at 32^3x64 2.94 -> 2.76 ms.
struct FB {
    float hi, lo;
    __device__ __forceinline__ float sum() const { return __fadd_rn(__fsub_rn(hi, 6.0f), lo); }
    __device__ __forceinline__ float minus1() const { return __fadd_rn(__fsub_rn(hi, 7.0f), lo); }
};
__device__ __forceinline__ void fb_addprod(FB& s, float a, float b) {
    const float t = __fmaf_rn(a, b, s.hi);
    const float q = __fsub_rn(t, s.hi);
    s.hi = t;
    s.lo = __fadd_rn(s.lo, __fmaf_rn(a, b, -q));
}

struct SumFF : FF {
    __device__ __forceinline__ SumFF() : FF{0.f, 0.f} {}
    __device__ __forceinline__ void add(float a, float b) { ff_addprod(*this, a, b); }
    __device__ __forceinline__ float sum() const { return hi + lo; }
    __device__ __forceinline__ float minus1() const { return __fadd_rn(__fsub_rn(hi, 1.0f), lo); }
};
struct SumFB : FB {
    __device__ __forceinline__ SumFB() : FB{6.f, 0.f} {}
    __device__ __forceinline__ void add(float a, float b) { fb_addprod(*this, a, b); }
};

// Row r of length^2 1 + delta -> r (1 + c), c = (1 + delta)^-1/2 - 1, with
// delta from the compensated sum so the row is rounded once; returns delta.
template <class Sum>
__device__ __forceinline__ float ff_normalise(float r[3], float i[3]) {
    Sum n;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        n.add(r[c], r[c]);
        n.add(i[c], i[c]);
    }
    const float d = n.minus1();
    const float c = fabsf(d) < 1e-3f ? d * (-0.5f + d * (0.375f - 0.3125f * d)) : rsqrtf(1.0f + d) - 1.0f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        r[k] = fmaf(c, r[k], r[k]);
        i[k] = fmaf(c, i[k], i[k]);
    }
    return d;
}

// FixSU3Matrix (row 0 normalised, row 1 orthogonalised and normalised,
// row 2 = conj(row0 x row1) normalised) in FP32.  The norms, the overlap and
// the cross products are small differences of O(1) products; summing them in
// float-float leaves one rounding per entry, as FP64 arithmetic rounded to
// FP32 would.  With plain FP32 sums the flowed B^2 of a 32^3x64 field
// drifted from the FP64 flow by 2.8e-6 (relative) after 200 steps of 0.01;
// with these sums by 9.5e-8, the same as with FixSU3Matrix in FP64.
// False when a row's length^2 was not within 1/2 of 1 (or not a number): with
// SumFB the result is then not to be used.
template <class Sum>
__device__ __forceinline__ bool fix_su3_rows_f32(float r[3][3], float i[3][3]) {
    const float n1 = r[1][0] * r[1][0] + i[1][0] * i[1][0] + r[1][1] * r[1][1] + i[1][1] * i[1][1] +
                     r[1][2] * r[1][2] + i[1][2] * i[1][2];
    const float d0 = ff_normalise<Sum>(r[0], i[0]);
    Sum dr, di;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        dr.add(r[0][c], r[1][c]);
        dr.add(i[0][c], i[1][c]);
        di.add(r[0][c], i[1][c]);
        di.add(-i[0][c], r[1][c]);
    }
    const float ovr = dr.sum(), ovi = di.sum();
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        r[1][c] -= r[0][c] * ovr - i[0][c] * ovi;
        i[1][c] -= r[0][c] * ovi + i[0][c] * ovr;
    }
    const float d1 = ff_normalise<Sum>(r[1], i[1]);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const int j = (c + 1) % 3, k = (c + 2) % 3;
        Sum re, im;
        re.add(r[0][j], r[1][k]);
        re.add(-i[0][j], i[1][k]);
        re.add(-r[0][k], r[1][j]);
        re.add(i[0][k], i[1][j]);
        im.add(r[0][j], i[1][k]);
        im.add(i[0][j], r[1][k]);
        im.add(-r[0][k], i[1][j]);
        im.add(-i[0][k], r[1][j]);
        r[2][c] = re.sum();
        i[2][c] = -im.sum();
    }
    ff_normalise<Sum>(r[2], i[2]);
    return fabsf(d0) < 0.5f && fabsf(d1) < 0.5f && fabsf(n1 - 1.0f) < 0.5f;
}

template <typename W>
__device__ __forceinline__ void reunitarise(M3<W>& w) {
    W r[3][3], im[3][3];
    auto rows = [&] {
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = 0; b < 3; ++b) {
                r[a][b] = w.r[3 * a + b];
                im[a][b] = w.i[3 * a + b];
            }
    };
    rows();
    if constexpr (sizeof(W) == 4) {
        // Off-diagonal entries that are small need sums exact to 2^-48 of
        // themselves: near a diagonal matrix (row 0 tells) the general sums, as when a
        // row is far from length 1.  At 2^-14 the bounded sums' 2^-46 is 2^-15 of the
        // rounding.
        float off = 0.f;
#pragma unroll
        for (int k = 1; k < 3; ++k) off = fmaf(w.r[k], w.r[k], fmaf(w.i[k], w.i[k], off));
        if (!(off > 0x1p-14f) || !fix_su3_rows_f32<SumFB>(r, im)) {
            rows();
            fix_su3_rows_f32<SumFF>(r, im);
        }
    } else {
        fix_su3_rows(r, im);
    }
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            w.r[3 * a + b] = r[a][b];
            w.i[3 * a + b] = im[a][b];
        }
}

// link u of direction mu at site s moved by the stage's X: f = the force G
// (Z = eps 2 G), bbuf = the kept B
template <typename T>
__device__ __forceinline__ M3<T> wflow_move(const M3<T>& f, const M3<T>& u, int64_t s, int mu,
                                            const AHPlanes<T>& bbuf, T eps, int stage, int reun) {
    const M3<T> z = m_scale(f, T(2) * eps);
    M3<T> x;
    if (stage == 0) {
        bbuf.store(s, mu, z);
        x = m_scale(z, T(0.25));
    } else if (stage == 1) {
        const M3<T> b = bbuf.load(s, mu);
        x = m_scale(z, T(8.0 / 9.0));
        m_axpy(x, T(-17.0 / 36.0), b);
        bbuf.store(s, mu, x);
    } else {
        const M3<T> b = bbuf.load(s, mu);
        x = m_scale(z, T(0.75));
        m_axpy(x, T(-1), b);
    }
    const M3<T> dm = expm1_ah(x);
    M3<T> w = mul(dm, u);
    m_axpy(w, T(1), u);
    if (reun) reunitarise(w);
    return w;
}

template <typename T>
__device__ __forceinline__ void store_full(void* links, int64_t V, int64_t s, int mu, const M3<T>& w) {
    using C2 = typename V2<T>::type;
    if (!FLUE_INB(s >= 0 && s < V && mu >= 0 && mu < 4)) return;
    C2* q = (C2*)links + s + V * mu;
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            C2 v;
            v.x = w.r[3 * a + b];
            v.y = w.i[3 * a + b];
            q[4 * V * (a + 3 * b)] = v;
        }
}

// FP64 update from the stored force (its grid is capped when gated)
__global__ void k_wflow_update(double2* links, Geom g, const double2* force, AHPlanes<double> bbuf, double eps,
                               int stage, FixGate gt) {
    if (gate_shut(gt)) return;
    for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < 4 * g.V;
         idx += (int64_t)gridDim.x * blockDim.x) {
        const int64_t s = idx % g.V;
        const int mu = (int)(idx / g.V);
        const M3<double> f = load_full<double>(force, g.V, s, mu), u = load_full<double>(links, g.V, s, mu);
        store_full(links, g.V, s, mu, wflow_move<double>(f, u, s, mu, bbuf, eps, stage, 0));
    }
}

// A stage of a complex64 field: the force of a link and its update in one
// kernel, from one field to another, so the force never goes to memory and
// every link is read once as the link to move.  The four directions of a site
// block run in adjacent blocks, where the staples' links are in L2 (a
// direction a pass over the lattice read 3.1 GB from DRAM for 0.6 GB of links).
// Bound by instruction issue (71%, three quarters of it FMA).  32^3x64, a step:
// force and update apart 4.9 ms, fused 3.42 (128 registers; 168: 3.49, 96:
// 3.48), with 32-bit offsets 3.22, with expm1_ah 3.03,
// with the site coordinates by 32-bit divisions 2.94, with the shorter
// compensated sums of FixSU3 (FB) 2.76.
template <int STAGE, class L, typename I>
__global__ void __launch_bounds__(128, 4)
    k_flow_stage32(L U, Geom g, AHPlanes<float> bbuf, float eps, float2* out) {
    const int mu = blockIdx.x & 3;
    const int64_t s64 = (int64_t)(blockIdx.x >> 2) * blockDim.x + threadIdx.x;
    if (s64 >= g.V) return;
    const I s = (I)s64;
    int c[4];
    site_coords(g, s64, c);
    I fw[4], bw[4];  // steps of +-1
#pragma unroll
    for (int d = 0; d < 4; ++d) {
        fw[d] = (I)(c[d] + 1 == g.n[d] ? -(int64_t)(g.n[d] - 1) * g.st[d] : g.st[d]);
        bw[d] = (I)(c[d] == 0 ? (int64_t)(g.n[d] - 1) * g.st[d] : -g.st[d]);
    }
    I fm = fw[0];
#pragma unroll
    for (int d = 1; d < 4; ++d)
        if (d == mu) fm = fw[d];
    const I sp = s + fm;
    M3<float> n = m_zero<float>();
#pragma unroll 1
    for (int nu = 0; nu < 4; ++nu) {
        if (nu == mu) continue;
        I fn = fw[0], bn = bw[0];
#pragma unroll
        for (int d = 1; d < 4; ++d)
            if (d == nu) fn = fw[d], bn = bw[d];
        const M3<float> up = mm<false, true>(U.load(sp, nu), U.load(s + fn, mu));
        m_add(n, mm<false, true>(up, U.load(s, nu)));
        const M3<float> dn = mm<true, true>(U.load(sp + bn, nu), U.load(s + bn, mu));
        mac<false, false>(n, dn, U.load(s + bn, nu));
    }
    const M3<float> u = U.load(s, mu);
    const M3<float> f = ta_scaled(mul(u, n), -0.5f);
    store_full<float>(out, g.V, s64, mu, wflow_move<float>(f, u, s64, mu, bbuf, eps, STAGE, 1));
}

// ---------------------------------------------------------------------------
// The step of a complex128 field in fixed point (fix.cuh): the links are
// converted once (k_flow_links), each stage computes the force of a link and
// moves it in one kernel from one fixed-point field to the other (the second lies
// over the complex128 links, FlowFixWs), and the last stage writes those.  A thread carries one column of a link
// (three warps for 32 sites), as the 5-loop kernels do.  A stage is 13 matrix
// products and exp(X) a link, bound by the integer multiply-add pipe.  RK3 step
// at 32^3x64: 92.8 ms as FP64 force and update, 22.2 with exp(X) from its even
// and odd powers on the column, 21.0 with the weights of I, X and X^2 (a third
// of the exponential's products).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(128) k_flow_links(FullLinks<double> U, Geom g, MatFix w, FixGate gt) {
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    u32 st = 0;
    if (gate_lost(gt)) return;
    if (s < g.V) {
        const int mu = (int)blockIdx.y;
        const M3<double> u = U.load(s, mu);
        const M3F f = fx_of(u);
        st = link_state(u, f);
        w.store(s, mu, f);
        if (st == 0) {
            int c[4];
            site_coords(g, s, c);
            for (int nu = mu + 1; nu < 4; ++nu)
                if (near_patch(U, g, c, mu, nu)) st = 1;
        }
    }
    gate_count(gt, st);
}

// a value of unit 2^-60 as limbs
__host__ __device__ constexpr Fx fx_const60(i64 x) {
    return {(int)((x + ((i64)1 << 30)) >> 31), (int)(x - ((x + ((i64)1 << 30)) >> 31) * ((i64)1 << 31))};
}
static Fx fx_const(double x) { return fx_const60((i64)llrint(ldexp(x, 60))); }
// 1/k!
constexpr int FLOW_TERMS = 20;
struct FlowFact {
    Fx f[FLOW_TERMS + 1];
};
constexpr FlowFact flow_fact() {
    FlowFact t{};
    i64 fact = 1;  // 20! < 2^62
    for (int k = 0; k <= FLOW_TERMS; ++k) {
        if (k) fact *= k;
        t.f[k] = fx_const60((((i64)1 << 60) + fact / 2) / fact);
    }
    return t;
}
static __constant__ FlowFact c_flow_fact = flow_fact();

// X of a stage: the off-diagonal and diagonal factor of the projected U N and
// the factor of the last stage's X
struct FlowStage {
    Fx off, diag, last;
};
// Sites a block: the three columns meet at one barrier, so many small blocks
// wait less for it than one large one.  RK3 step at 32^3x64: 128 sites 21.0 ms,
// 64 with two / three blocks an SM 18.5 / 17.7, 32 with four / five / six / seven
// 17.6 / 17.2 / 17.2 / 17.5.
constexpr int FF_BS = 32, FF_MINB = 5;

template <int STAGE, typename I>
__global__ void __launch_bounds__(3 * FF_BS, FF_MINB)
    k_flow_stage(Geom g, MatFix w, MatFix wout, AHFix xb, FlowStage sc, double2* links, FixGate gt) {
    __shared__ longlong2 sq[9][FF_BS];
    if (!gt.open()) return;
    const int mu = blockIdx.x & 3;  // the directions of a site block in adjacent blocks (L2 reuse)
    const int b = threadIdx.x / FF_BS, j = threadIdx.x % FF_BS;
    const int64_t s64 = (int64_t)(blockIdx.x >> 2) * FF_BS + j;
    const bool live = s64 < g.V;
    const I s = (I)(live ? s64 : 0);
    int c[4];
    site_coords(g, (int64_t)s, c);
    I fw[4], bw[4];  // steps of +-1
#pragma unroll
    for (int d = 0; d < 4; ++d) {
        fw[d] = (I)(c[d] + 1 == g.n[d] ? -(int64_t)(g.n[d] - 1) * g.st[d] : g.st[d]);
        bw[d] = (I)(c[d] == 0 ? (int64_t)(g.n[d] - 1) * g.st[d] : -g.st[d]);
    }
    I fm = fw[0];
#pragma unroll
    for (int d = 1; d < 4; ++d)
        if (d == mu) fm = fw[d];
    // column b of N, the sum of the six staples: |N| <= 6
    FxVS n = vs_zero();
#pragma unroll 1
    for (int k = 1; k < 4; ++k) {
        const int nu = (mu + k) & 3;
        I fn = fw[0], bn = bw[0];
#pragma unroll
        for (int d = 1; d < 4; ++d)
            if (d == nu) fn = fw[d], bn = bw[d];
        FxV v = w.mul<true>((I)(s + fn), mu, w.col<true>(s, nu, b));
        w.mac<false>(n, (I)(s + fm), nu, v);
        v = w.mul<true>((I)(s + bn), mu, w.col<false>((I)(s + bn), nu, b));
        w.mac<true>(n, (I)(s + fm + bn), nu, v);
    }
    {  // U N / 8
        FxV v;
#pragma unroll
        for (int a = 0; a < 3; ++a) v.r[a] = fx_of61(n.r[a]), v.i[a] = fx_of61(n.i[a]);
        FxVS un = vs_zero();
        w.mac<false>(un, s, mu, v);
#pragma unroll
        for (int a = 0; a < 3; ++a) sq[3 * a + b][j] = make_longlong2(un.r[a], un.i[a]);
    }
    // X_last before the barrier: the first column's warp overwrites it after
    Fx last[9];
    if (STAGE > 0) xb.load(s, mu, 0, last);
    __syncthreads();
    // X = sc . (U N - (U N)^+ without its trace) + sc.last X_last
    Fx x[9];
    {
        i64 d[9];
        fx_antiherm([&](int el) { return sq[el][j]; }, d);
        // (diagonal entries of fx_antiherm are 2 Im: 3 Im - trace from them)
        const i64 tr = (d[0] + d[1] + d[2]) >> 1;
#pragma unroll
        for (int e = 0; e < 9; ++e) {
            const i64 de = e < 3 ? d[e] + (d[e] >> 1) - tr : d[e];
            FxAcc t = {FX_HI0, FX_CR0};
            fx_mad(t, fx_of61(de), e < 3 ? sc.diag : sc.off);
            if (STAGE > 0) fx_mad(t, last[e], sc.last);
            x[e] = fx_limbs(t);
        }
        if (STAGE < 2 && live && b == 0) {
#pragma unroll
            for (int e = 0; e < 9; ++e) d[e] = ((i64)x[e].h << 32) + 2 * (i64)x[e].l;
            xb.store(s64, mu, d);
        }
    }
    // X halved until |X|_F <= 1/2
    float nrm = 0.f;
#pragma unroll
    for (int e = 0; e < 9; ++e) {
        const float t = (float)x[e].h * 0x1p-29f;
        nrm = fmaf(e < 3 ? t : 2.f * t, t, nrm);
    }
    nrm = sqrtf(nrm) * 1.0001f;
    int reps = 1;
    while (nrm > 0.5f && reps < 64) {
        nrm *= 0.5f;
        reps *= 2;
#pragma unroll
        for (int e = 0; e < 9; ++e) x[e] = fx_of61((((i64)x[e].h << 32) + 2 * (i64)x[e].l) >> 1);
    }
    // exp(X) U - U = w0 U + w1 X U + w2 X (X U), the weights from the recurrence
    // of X^k = p + q X + r X^2 with X^3 = -m X + i delta (expm1_ah; X has no trace).
    // At even k p and r are real and q imaginary, at odd k the other way round,
    // so an order takes two real products, and three into the weights.
    FxR w3;
    {
        const Fx d0 = x[0], d1 = x[1], d2 = x[2], br = x[3], bi = x[4], cr = x[5], ci = x[6], er = x[7], ei = x[8];
        auto sum2 = [](const Fx& a, const Fx& b, const Fx& c, const Fx& d) {  // a b + c d
            FxAcc t = {FX_HI0, FX_CR0};
            fx_mad(t, a, b), fx_mad(t, c, d);
            return fx_limbs(t);
        };
        const Fx bb = sum2(br, br, bi, bi), cc = sum2(cr, cr, ci, ci), ee = sum2(er, er, ei, ei);
        const Fx ber = sum2(br, er, fx_neg(bi), ei), bei = sum2(br, ei, bi, er);
        FxAcc t = {0, FX_CR0};
        fx_mad(t, d0, d0), fx_mad(t, d1, d1), fx_mad(t, d2, d2);
        // -m = -|X|^2 / 2
        const Fx nm = fx_of58(-((fx_fold(t) >> 1) + ((fx_int60(bb) + fx_int60(cc) + fx_int60(ee)) >> 2)));
        t = {FX_HI0, FX_CR0};
        fx_mad(t, fx_neg(d0), d1);
        const Fx dd = fx_limbs(t);
        FxAcc u2 = {0, FX_CR0};
        fx_mad(u2, ber, ci), fx_mad(u2, fx_neg(bei), cr);
        t = {FX_HI0 + 2 * fx_fold(u2), FX_CR0};
        fx_mad(t, d1, cc), fx_mad(t, d2, bb), fx_mad(t, d0, ee), fx_mad(t, dd, d2);
        const Fx delta = fx_limbs(t), ndelta = fx_neg(delta);
        FxAcc wr[3], wi[3];
#pragma unroll
        for (int e = 0; e < 3; ++e) {
            wr[e] = {FX_HI0 + (e ? (i64)1 << (59 - e) : 0), FX_CR0};
            wi[e] = {FX_HI0, FX_CR0};
        }
        // from X^2: p = q = 0, r = 1
        Fx p = {0, 0}, q = {0, 0}, r = {1 << 29, 0};
        float bnd = 0.5f * nrm * nrm;
        auto next = [&](int k, const Fx& dl, FxAcc& a0, FxAcc& a1, FxAcc& a2) {
            FxAcc tp = {FX_HI0, FX_CR0};
            fx_mad(tp, dl, r);
            FxAcc tq = {FX_HI0 + ((i64)p.h << 29), FX_CR0 + ((i64)p.l << 29)};
            fx_mad(tq, nm, r);
            r = q;
            p = fx_limbs(tp);
            q = fx_limbs(tq);
            const Fx f = c_flow_fact.f[k];
            fx_mad(a0, p, f), fx_mad(a1, q, f), fx_mad(a2, r, f);
        };
#pragma unroll 1
        for (int k = 3; k < FLOW_TERMS; k += 2) {
            bnd *= nrm / (float)k;  // |X|^k / k!
            if (!(bnd > 0x1p-60f)) break;
            next(k, delta, wi[0], wr[1], wi[2]);
            next(k + 1, ndelta, wr[0], wi[1], wr[2]);
            bnd *= nrm / (float)(k + 1);
        }
#pragma unroll
        for (int e = 0; e < 3; ++e) w3.r[e] = fx_limbs(wr[e]), w3.i[e] = fx_limbs(wi[e]);
        fx_row_sums<false>(w3);
    }
    FxV u = w.col<false>(s, mu, b);
#pragma unroll 1
    for (int rep = 0; rep < reps; ++rep) {
        FxV v, z;
        FxVP vp = fx_prep<false>(u);
#pragma unroll
        for (int a = 0; a < 3; ++a) fx_rdot_limbs(v.r[a], v.i[a], ah_row(x, a), vp);
        vp = fx_prep<false>(v);
#pragma unroll
        for (int a = 0; a < 3; ++a) fx_rdot_limbs(z.r[a], z.i[a], ah_row(x, a), vp);
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            FxV o;
            o.r[0] = u.r[a], o.i[0] = u.i[a];
            o.r[1] = v.r[a], o.i[1] = v.i[a];
            o.r[2] = z.r[a], o.i[2] = z.i[a];
            FxAcc dr, di;
            fx_rdot(dr, di, w3, fx_prep<false>(o), 0, 0);
            u.r[a] = fx_const60(fx_int60(u.r[a]) + 4 * fx_fold(dr));
            u.i[a] = fx_const60(fx_int60(u.i[a]) + 4 * fx_fold(di));
        }
    }
    if (!live) return;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        if (STAGE < 2) {
            wout.store_el(s64, mu, 3 * a + b, u.r[a], u.i[a]);
        } else if (FLUE_INB(s64 < g.V)) {
            links[s64 + g.V * (mu + 4 * (a + 3 * b))] =
                make_double2((double)fx_int60(u.r[a]) * 0x1p-60, (double)fx_int60(u.i[a]) * 0x1p-60);
        }
    }
}

template <typename I>
static void flow_fix_stages(void* links, const Geom& g, double eps, char* ws, const FlowFixWs& w, const FixGate& gt,
                            cudaStream_t st) {
    const MatFix w0{(int4*)ws, g.V, 4}, w1{(int4*)(w.w1 ? ws + w.w1 : links), g.V, 4};
    const AHFix xb{(longlong2*)(ws + w.x), g.V, 4};
    const unsigned nb = (unsigned)((g.V + FF_BS - 1) / FF_BS) * 4;
    // Z = -eps TA(U N): the kernel holds (U N - (U N)^+)/64 off the diagonal and
    // (3 Im - trace)/64 on it.  The kept X of stage 0 is Z0/4, so stage 1 takes
    // 8/9 Z1 - 17/36 (4 X) and stage 2 takes 3/4 Z2 - X.
    const double f[3] = {0.25, 8.0 / 9.0, 0.75}, last[3] = {0.0, -17.0 / 9.0, -1.0};
    FlowStage sc[3];
    for (int k = 0; k < 3; ++k) sc[k] = {fx_const(-32.0 * eps * f[k]), fx_const(-64.0 / 3.0 * eps * f[k]), fx_const(last[k])};
    note_launch(), k_flow_stage<0, I><<<nb, 3 * FF_BS, 0, st>>>(g, w0, w1, xb, sc[0], nullptr, gt);
    note_launch(), k_flow_stage<1, I><<<nb, 3 * FF_BS, 0, st>>>(g, w1, w0, xb, sc[1], nullptr, gt);
    note_launch(), k_flow_stage<2, I><<<nb, 3 * FF_BS, 0, st>>>(g, w0, w1, xb, sc[2], (double2*)links, gt);
}

// at(field): the accessor of a field
template <class L, typename I, class At>
static void flow32_stages(At at, float2* l0, float2* l1, float2* l2, const Geom& g, const AHPlanes<float>& b, float eps,
                          cudaStream_t st) {
    const unsigned nb = (unsigned)((g.V + 127) / 128) * 4;
    note_launch(), k_flow_stage32<0, L, I><<<nb, 128, 0, st>>>(at(l0), g, b, eps, l1);
    note_launch(), k_flow_stage32<1, L, I><<<nb, 128, 0, st>>>(at(l1), g, b, eps, l2);
    note_launch(), k_flow_stage32<2, L, I><<<nb, 128, 0, st>>>(at(l2), g, b, eps, l0);
}

cudaError_t launch_wflow_step(void* links, const Geom& g, int prec, double eps, void* ws, size_t ws_bytes,
                              cudaStream_t st) {
    char* w = (char*)ws;
    const size_t f = (((size_t)36 * g.V * 16) + 255) & ~(size_t)255;
    const size_t b = (((size_t)36 * g.V * 8) + 255) & ~(size_t)255;
    void* force = w;
    // B in the field's precision (the slot is sized for FP64)
    AHPlanes<double> bb{(double*)(w + f), g.V};
    AHPlanes<float> bbf{(float*)(w + f), g.V};
    if (prec == PREC_C64) {
        // links -> first half of the force slot -> second half -> links
        float2 *l0 = (float2*)links, *l1 = (float2*)force, *l2 = l1 + (size_t)36 * g.V;
        if (FullLinks32::fits(g.V)) {
            auto at = [&](const float2* l) { return FullLinks32{(const char*)l, (uint32_t)g.V}; };
            flow32_stages<FullLinks32, u32>(at, l0, l1, l2, g, bbf, (float)eps, st);
        } else {
            auto at = [&](const float2* l) { return FullLinks<float>{l, g.V}; };
            flow32_stages<FullLinks<float>, int64_t>(at, l0, l1, l2, g, bbf, (float)eps, st);
        }
        return cudaGetLastError();
    }
    double* part = (double*)(w + f + b);
    FieldRef U{links, g, prec};
    const unsigned nb = (unsigned)((4 * g.V + 127) / 128);
    // Fixed point for complex128 fields with its workspace; its factors leave
    // their range (|32 eps| < 4) at eps = 1/8, where a step is far too long anyway.
    const FlowFixWs fw = flow_fix_layout(g);
    FixGate gt;
    if (ws_bytes >= fw.total && eps < 0.12) {
        gt.p = (u32*)(w + fw.gate);
        gt.need = (u32)g.V;  // a quarter of the links
        cudaError_t e = cudaMemsetAsync(gt.p, 0, GATE_WORDS * sizeof(u32), st);
        if (e != cudaSuccess) return e;
        const MatFix w0{(int4*)w, g.V, 4};
        note_launch(), k_flow_links<<<dim3((unsigned)((g.V + 127) / 128), 4), 128, 0, st>>>(
            FullLinks<double>{(const double2*)links, g.V}, g, w0, gt);
        if (MatFix::fits32(g.V, 4))
            flow_fix_stages<u32>(links, g, eps, w, fw, gt, st);
        else
            flow_fix_stages<int64_t>(links, g, eps, w, fw, gt, st);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    for (int stage = 0; stage < 3; ++stage) {
        cudaError_t e = gt.p ? launch_plaquette_force_gated(U, force, gt, st)
                             : launch_plaquette_force(U, part, nullptr, force, 0, st);
        if (e != cudaSuccess) return e;
        const unsigned nbg = gt.p ? std::min(nb, 8u * (unsigned)device_sms()) : nb;
        note_launch(), k_wflow_update<<<nbg, 128, 0, st>>>((double2*)links, g, (const double2*)force, bb, eps, stage, gt);
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

FLUE_OOB_READER(flow)

}  // namespace flue
