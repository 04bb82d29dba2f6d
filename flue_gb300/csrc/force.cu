// force.cu -- clover and 5-loop F_munu, the 5-loop energy / B^2 and its
// su(3) gradient, and the Wilson plaquette-action force.
//
// The 5-loop field strength (src/wloops.F90:201-432, hep-lat/0203008) at a
// site x and plane (mu,nu) is built from the 28 counter-clockwise leaves of
// the rectangles of shapes (a,b) in {(1,1),(2,2),(3,3),(1,2),(2,1),(1,3),(3,1)}
// (a links along mu, b along nu) that have x as a corner.  The reference walks
// every leaf link by link (208 link steps and 180 products per plane-site);
// here a leaf is the product of four straight "lines"
//     L^a_mu(y) = U_mu(y) U_mu(y+mu) ... U_mu(y+(a-1)mu),   a = 1,2,3,
// precomputed once per site (2 products per direction), so a leaf costs 3
// products (84 per plane-site).  Writing the rectangle anchored at y0 (its
// lower-left corner) as the sides
//     S1 = L^a_mu(y0),  S2 = L^b_nu(y0+a mu),  S3 = L^a_mu(y0+b nu)^+,  S4 = L^b_nu(y0)^+
// with corners K1..K4 at y0, y0+a mu, y0+a mu+b nu, y0+b nu, the leaf of x in
// quadrant q is the cyclic word S_q S_q+1 S_q+2 S_q+3 of the rectangle that
// has x as its corner q.  genericPath returns the transpose of every leaf
// (:56); the kernels work with untransposed leaves and transpose on output.
//
// Energy E = -1/V sum_x sum_planes Re Tr(F F) (B^2 for the three spatial
// planes (3,2),(2,4),(4,3) of magnetic, :502-506).  Reverse mode, written as
// gathers so that no atomics are needed and results are deterministic:
//   1. lines:   L^2, L^3 per direction                    (k_lines)
//   2. forward: Q, F = AH(Q)/4, E partials; F kept as the cotangent
//               dE/dQ = -F/(2V) (stored as 9 reals)        (k_fwd)
//   3. line cotangents: Lambda^a_d(y) with dE = Re Tr(dL Lambda), summed over
//      every rectangle side that is the line (y,d,a); each side collects the
//      four corner insertions K S S S + S K S S + S S K S + S S S K with a
//      Horner scheme (8 products)                          (k_linecot)
//   4. link cotangents N_d(z) from the line cotangents of the lines through
//      the link, then the su(3)-projected gradient G = -1/2 TA(U N) or the
//      Euclidean gradient N^+                              (k_linkcot)
#include <stdlib.h>

#include <algorithm>
#include <mutex>

#include "flue_internal.h"
#include "loop5.cuh"
#include "loop5_fix.cuh"

namespace flue {

// Traversal order of the site blocks of the stencil kernels.  The lattice is
// a sequence of rows (fixed y, z) of NT*NX sites.  When a row holds a whole
// number of blocks and NY, NZ are multiples of the tile, rows are visited in
// TILE x TILE (y,z) tiles, y fastest, so that the blocks in flight cover a
// compact neighbourhood and the +-3 halo they read is still in L2 (measured
// no faster on GB300: off by default).
#ifndef FLUE_TILE_YZ
#define FLUE_TILE_YZ 0
#endif
__device__ __forceinline__ int64_t site_block(int64_t b, const Geom& g, int bs) {
#if FLUE_TILE_YZ > 0
    const int T = FLUE_TILE_YZ;
    const int64_t rowlen = (int64_t)g.n[0] * g.n[1];
    if (rowlen % bs == 0 && g.n[2] % T == 0 && g.n[3] % T == 0) {
        const int64_t bpr = rowlen / bs;
        const int64_t in_row = b % bpr, row = b / bpr;
        const int64_t tile = row / (T * T), r = row % (T * T);
        const int64_t nty = g.n[2] / T;
        const int64_t y = (tile % nty) * T + r % T, z = (tile / nty) * T + r / T;
        return (y + (int64_t)g.n[2] * z) * bpr + in_row;
    }
#endif
    return b;
}

// Patch traversal of the stencil kernels: a block of `bs` threads covers tw
// consecutive time slices x a pm x pn patch of the plane (mu, nu) x po sites
// along the third spatial direction (tw * pm * pn * po = bs), so the warps of
// a block read overlapping neighbourhoods and share them in L1.  tw = 0: the
// linear order.  Valid for spatial planes with tw | NT, pm | N_mu, pn | N_nu,
// po | N_other (make_patch checks; otherwise it returns tw = 0).
struct PatchArg {
    int tw, pm, pn, po;
};

__device__ __forceinline__ int64_t patch_site(const Geom& g, const PatchArg& pt, int pmu, int pnu, unsigned r, int tid) {
    int nm = 1, nn = 1;
    int64_t stm = 0, stn = 0, sto = 0;
    const int od = 6 - pmu - pnu;
#pragma unroll
    for (int d = 1; d < 4; ++d) {
        if (d == pmu) nm = g.n[d], stm = g.st[d];
        if (d == pnu) nn = g.n[d], stn = g.st[d];
        if (d == od) sto = g.st[d];
    }
    const unsigned ntc = g.n[0] / pt.tw, nbm = nm / pt.pm, nbn = nn / pt.pn;
    const int tc = (int)(r % ntc);
    r /= ntc;
    const int bi = (int)(r % nbm);
    r /= nbm;
    const int bj = (int)(r % nbn);
    const int bo = (int)(r / nbn);
    const int tl = tid % pt.tw, pos = tid / pt.tw;
    const int im = pos % pt.pm, in = (pos / pt.pm) % pt.pn, io = pos / (pt.pm * pt.pn);
    return (int64_t)tc * pt.tw + tl + (int64_t)(bi * pt.pm + im) * stm + (int64_t)(bj * pt.pn + in) * stn +
           (int64_t)(bo * pt.po + io) * sto;
}

#ifndef FLUE_PATCH_MIN_TW
#define FLUE_PATCH_MIN_TW 8
#endif
static PatchArg make_patch(const Geom& g, const PlaneArg& pa, int bs) {
    PatchArg pt{0, 1, 1, 1};
    int tw = 1;
    while (tw < 32 && g.n[0] % (2 * tw) == 0 && tw * 2 <= bs) tw *= 2;
    const int P = bs / tw;
    int pm = 1;
    while (pm < 4 && pm * pm * 4 <= P) pm *= 2;  // pm = pn <= 4
    const int po = P / (pm * pm);
    for (int q = 0; q < pa.np; ++q) {
        const int mu = pa.mu[q], nu = pa.nu[q], od = 6 - mu - nu;
        if (mu <= 0 || nu <= 0 || g.n[mu] % pm || g.n[nu] % pm || g.n[od] % po) return pt;
    }
    // warps keep runs of >= FLUE_PATCH_MIN_TW consecutive sites (measured at
    // 32^3x64 in 4-slice slabs, tiled intermediates: minimum 4 -> 10.74 ms a
    // step, 8 -> 10.50 ms)
    if (tw * pm * pm * po != bs || tw < FLUE_PATCH_MIN_TW) return pt;
    pt.tw = tw;
    pt.pm = pt.pn = pm;
    pt.po = po;
    return pt;
}

// ---------------------------------------------------------------------------
// 1. lines: L^1_d(y) = U_d(y) (expanded to 18 reals), L^2_d(y) = U_d(y) U_d(y+d),
//    L^3_d(y) = L^2_d(y) U_d(y+2d).  Sites are those of geometry g; the links
//    are read from a field of geometry gs at time offset t0 (gs = g, t0 = 0
//    for a whole lattice; a time slab of a larger field otherwise -- the lines
//    never step in time then).
// ---------------------------------------------------------------------------
template <class L>
__global__ void k_lines(L U, Geom g, Geom gs, int t0, PlaneArg pa, MatAoS<float> lines) {
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= g.V) return;
    line_site<L, float>(U, g, gs, t0, pa, lines, s, (int)blockIdx.y);
}

// complex128 fields: the lines in fixed point (fix.cuh), counting the links
// that are not unitary, or close to 1 together, in the gate.  32^3x64 B^2: 1.06 ms, HBM
// (2.7 GB written) and the conversion of the links to limbs.  Behind a warp that
// has shut the gate the others leave (clover of a cold 32^3x64 6.71 -> 6.14 ms, 5.99
// without fixed point).
__global__ void __launch_bounds__(128) k_lines_fix(FullLinks<double> U, Geom g, Geom gs, int t0, PlaneArg pa,
                                                   MatFix lines, FixGate gt) {
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int slot = (int)blockIdx.y;
    u32 st = 0;
    if (gate_lost(gt)) return;
    if (s < g.V) {
        st = line_site_fix(U, g, gs, t0, pa, lines, s, slot);
        if (st == 0) {
            int c[4];
            site_coords(g, s, c);
            c[0] += t0;
            for (int k = slot + 1; k < pa.nd; ++k)
                if (near_patch(U, gs, c, sel(pa.dir, slot), sel(pa.dir, k))) st = 1;
        }
    }
    gate_count(gt, st);
}

// The FP64 kernels behind a gate: every block leaves at once when the
// fixed-point kernels have the field (gate_shut), else the (capped) grid walks
// the blocks of the ungated grid.
__global__ void __launch_bounds__(128) k_lines_gated(FullLinks<double> U, Geom g, Geom gs, int t0, PlaneArg pa,
                                                     MatAoS<double> lines, FixGate gt) {
    if (gate_shut(gt)) return;
    for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < g.V; s += (int64_t)gridDim.x * blockDim.x)
        line_site<FullLinks<double>, double>(U, g, gs, t0, pa, lines, s, (int)blockIdx.y);
}

// ---------------------------------------------------------------------------
// 2. forward: one thread per (site, plane)
// ---------------------------------------------------------------------------
// block size and, in FP32, minimum resident blocks per SM (register budget) of
// the forward and line-cotangent kernels; overridable at build time.  The FP64
// kernels keep every register they need (they are bound by the FP64 pipe, not by
// latency).
#ifndef FLUE_FWD_BS
#define FLUE_FWD_BS 128
#endif
// patch traversal of the forward (PatchArg): 32^3x64 one pass 3.26 -> 2.95 ms;
// inside 4-slice time slabs it is not used (make_patch)
#ifndef FLUE_FWD_PATCH
#define FLUE_FWD_PATCH 1
#endif
#ifndef FLUE_FWD_MINB
#define FLUE_FWD_MINB 3
#endif
#ifndef FLUE_COT_BS
#define FLUE_COT_BS 128
#endif
#ifndef FLUE_COT_MINB
#define FLUE_COT_MINB 4
#endif
constexpr int FWD_BS = FLUE_FWD_BS;
// Sites a block of the fixed-point forward and line cotangents covers, three
// threads a site: 192 threads and up to 168 registers, two blocks an SM.  Both
// are bound by the integer multiply-add pipe (73% busy, waits on its results
// next), so registers count for more than warps.  32^3x64 in one pass, forward /
// line cotangents: 128 sites (one block: its last warps leave an SM idle) 18.9 /
// 43.8 ms, 64 18.5 / 42.3, 32 21.8 / 43.6; three blocks of 64 (112 registers)
// spill.  In time slabs on four streams B^2 19.4 -> 19.0 ms.
constexpr int FIX_BS = 64;
// The forward of a small lattice takes blocks of 32 sites, four an SM: with few
// blocks the last wave is mostly empty.  B^2 at 8^3x16 194 -> 173 us against 128
// sites, 10^3x16 254 -> 241, 12^3x24 497 -> 511 (so not there: the line lies at
// 3 x 128 sites and planes an SM); two halves of the leaves on twice the threads
// gave 182, 272, 502.
constexpr int FIX_BS_SMALL = 32;
static int fix_fwd_block(int64_t V, int planes) {
    return (V + 127) / 128 * planes < 3 * device_sms() ? FIX_BS_SMALL : FIX_BS;
}

// site j of the bs sites of block b of the forward's grid, plane p = b % np
// (planes of the same site block run in adjacent blocks: L2 reuse)
__device__ __forceinline__ int64_t fwd_site(const Geom& g, const PlaneArg& pa, const PatchArg& pt, unsigned b, int p,
                                            int j, int bs) {
    return pt.tw ? patch_site(g, pt, sel(pa.mu, p), sel(pa.nu, p), b / pa.np, j)
                 : site_block(b / pa.np, g, bs) * bs + j;
}

template <typename T, typename I>
__device__ __forceinline__ void fwd_block(unsigned b, const Geom& g, const PlaneArg& pa, int kind, const PatchArg& pt,
                                          const MatAoS<T>& lines, const AHAoS<T>& kout, const RefOut<T>& fout,
                                          double* part, double* sh) {
    const int p = b % pa.np;
    const int64_t s = fwd_site(g, pa, pt, b, p, threadIdx.x, blockDim.x);
    double e = 0.0;
    if (s < g.V) {
        int c[4];
        site_coords(g, s, c);
        const M3<T> q = fwd_q<T, I>(g, pa, kind, lines, s, c, p);
        const M3<T> f = ah_quarter(q);
        e = -(double)retr_mm<false, false>(f, f);
        if (kout.p) kout.store(s, p, f);
        if (fout.p) fout.store(s, 0, transp(f));
    }
    if (part) {
        const double r = block_sum(e, sh);
        if (threadIdx.x == 0) part[b] = r;
    }
}

template <typename I>
__global__ void __launch_bounds__(FWD_BS, FLUE_FWD_MINB)
    k_fwd(Geom g, PlaneArg pa, int kind, PatchArg pt, MatAoS<float> lines, AHAoS<float> kout, RefOut<float> fout,
          double* part) {
    __shared__ double sh[32];
    fwd_block<float, I>(blockIdx.x, g, pa, kind, pt, lines, kout, fout, part, sh);
}

template <typename I>
__global__ void __launch_bounds__(FWD_BS)
    k_fwd_gated(Geom g, PlaneArg pa, int kind, PatchArg pt, MatAoS<double> lines, AHAoS<double> kout,
                RefOut<double> fout, double* part, unsigned nblocks, unsigned nparts, FixGate gt) {
    __shared__ double sh[32];
    if (gate_shut(gt)) return;
    for (unsigned b = blockIdx.x; b < nblocks; b += gridDim.x)
        fwd_block<double, I>(b, g, pa, kind, pt, lines, kout, fout, part, sh);
    // the smaller blocks of the fixed-point forward have more partial sums: with
    // zeros for the rest the energy is that of the ungated kernel, bit for bit
    if (part)
        for (unsigned b = nblocks + blockIdx.x * blockDim.x + threadIdx.x; b < nparts; b += gridDim.x * blockDim.x)
            part[b] = 0.0;
}

// Forward in fixed point: the sites and partial sums of the FP64 blocks, three
// warps (columns) for every 32 sites.  32^3x64, three planes: FP64 pipe 81.1 ms,
// fixed point with a thread a site 20.7 ms (240 registers, 8 warps an SM), with
// a thread a column 18.5 ms.
template <int BS, typename I>
__global__ void __launch_bounds__(3 * BS, 128 / BS)
    k_fwd_fix(Geom g, PlaneArg pa, int kind, PatchArg pt, MatFix lines, AHFix kout, RefOut<double> fout, double* part,
              u32* kmax, bool kslice, FixGate gt) {
    __shared__ longlong2 sq[9][BS];
    __shared__ double sh[32];
    if (!gt.open()) return;
    const int p = blockIdx.x % pa.np;
    const int b = threadIdx.x / BS, j = threadIdx.x % BS;
    const int64_t s = fwd_site(g, pa, pt, blockIdx.x, p, j, BS);
    double e = 0.0;
    int c[4];
    if (s < g.V) {
        site_coords(g, s, c);
        const FxVS q = fwd_q_fix<I>(g, pa, kind, lines, s, c, p, b);
#pragma unroll
        for (int a = 0; a < 3; ++a) sq[3 * a + b][j] = make_longlong2(q.r[a], q.i[a]);
    }
    __syncthreads();
    if (threadIdx.x < BS && s < g.V) {
        i64 d[9];
        fx_antiherm([&](int el) { return sq[el][j]; }, d);
        double f[9];
        fx_field_strength(d, kind == 1 ? FXQ5 : 1.0, f);
        e = ah_norm2(f);
        if (kout.p) {
            kout.store(s, p, d);
            kscale_max(kmax + (kslice ? c[0] : 0), e);
        }
        if (fout.p) fout.store(s, 0, transp(ah_expand(f)));
    }
    if (part) {
        const double r = block_sum(e, sh);
        if (threadIdx.x == 0) part[blockIdx.x] = r;
    }
}

// ---------------------------------------------------------------------------
// 2b. forward with the lines staged in shared memory per timeslice tile
//     (FP32 5-loop energies over spatial planes; fwd_tile_ok).  A block
//     of 128 threads covers FT_TT = 2 time slices x an 8 x 8 patch of the
//     plane (mu, nu) at one value of the third spatial coordinate.  For each
//     shape (a, b) the mu-lines of length a over the patch widened by a
//     below in mu and by b on both sides in nu, and the nu-lines of length b
//     over the patch widened by a on both sides in mu and by b below in nu,
//     are copied into shared memory with cp.async (16 bytes per copy, the
//     next shape's lines in flight while the current shape is computed,
//     double buffered); the four leaves of each site then read their twelve
//     lines from shared memory with 32-bit addresses.
// ---------------------------------------------------------------------------
constexpr int FT_TT = 2, FT_TM = 8, FT_TN = 8, FT_BS = FT_TT * FT_TM * FT_TN;
// matrices of the largest shape's staging area, (3,3): 2 x 11 x 14 x 2
constexpr int FT_MAXPOS = 2 * (FT_TM + 3) * (FT_TN + 6) * FT_TT;
constexpr size_t FT_SMEM = 2 * (size_t)FT_MAXPOS * 5 * sizeof(float4);

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

__device__ __forceinline__ M3<float> lds_mat(const float4* q) {
    M3<float> m;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float4 v = q[j];
        m.r[2 * j] = v.x;
        m.i[2 * j] = v.y;
        m.r[2 * j + 1] = v.z;
        m.i[2 * j + 1] = v.w;
    }
    const float4 v = q[4];
    m.r[8] = v.x;
    m.i[8] = v.y;
    return m;
}

struct TileGeom {
    int nm, nn, stm, stn, sto;  // extents and site strides along mu, nu; stride of the third direction
};

__global__ void __launch_bounds__(FT_BS, 2)
    k_fwd_tile(Geom g, PlaneArg pa, MatAoS<float> lines, AHAoS<float> kout, double* part) {
    extern __shared__ float4 ft_sm[];
    __shared__ double sh[32];
    const int p = blockIdx.x % pa.np;
    const int mu = sel(pa.mu, p), nu = sel(pa.nu, p), od = 6 - mu - nu;
    TileGeom tg{1, 1, 0, 0, 0};
#pragma unroll
    for (int d = 1; d < 4; ++d) {
        if (d == mu) tg.nm = g.n[d], tg.stm = (int)g.st[d];
        if (d == nu) tg.nn = g.n[d], tg.stn = (int)g.st[d];
        if (d == od) tg.sto = (int)g.st[d];
    }
    int r = blockIdx.x / pa.np;
    const int ntb = g.n[0] / FT_TT, nmb = tg.nm / FT_TM, nnb = tg.nn / FT_TN;
    const int tb = r % ntb;
    r /= ntb;
    const int mb = r % nmb;
    r /= nmb;
    const int nb = r % nnb;
    const int oc = r / nnb;
    const int t0 = tb * FT_TT, m0 = mb * FT_TM, n0 = nb * FT_TN, obase = oc * tg.sto;
    const int tid = threadIdx.x;
    const int tl = tid % FT_TT, ml = (tid / FT_TT) % FT_TM, nl = tid / (FT_TT * FT_TM);
    const int kmu = 3 * sel(pa.slot, mu), knu = 3 * sel(pa.slot, nu);

    // issue the copies of shape k's lines into buf (one commit group)
    auto stage = [&](int k, float4* buf) {
        const int a = c_shapes5[k].a, b = c_shapes5[k].b;
        const int Wm = FT_TN + 2 * b, Rm = (FT_TM + a) * Wm * FT_TT;
        const int Wn = FT_TN + b, Rn = (FT_TM + 2 * a) * Wn * FT_TT;
        // exact quotient by W for the row numbers met here (< 256; W <= 14)
        const unsigned invm = (65536u + Wm - 1) / Wm, invn = (65536u + Wn - 1) / Wn;
        for (int pos = tid; pos < Rm + Rn; pos += FT_BS) {
            const bool isn = pos >= Rm;
            const int q = isn ? pos - Rm : pos;
            const int W = isn ? Wn : Wm;
            const int tt = q % FT_TT, rr = q / FT_TT;
            const int im = (int)(((unsigned)rr * (isn ? invn : invm)) >> 16);
            const int jn = rr - im * W;
            int cm = m0 + im - a;
            cm += cm < 0 ? tg.nm : 0;
            cm -= cm >= tg.nm ? tg.nm : 0;
            int cn = n0 + jn - b;
            cn += cn < 0 ? tg.nn : 0;
            cn -= cn >= tg.nn ? tg.nn : 0;
            const uint32_t site = (uint32_t)(t0 + tt + cm * tg.stm + cn * tg.stn + obase);
            const int plane = isn ? knu + b - 1 : kmu + a - 1;
            const float4* src = lines.unit0_32(site, plane);
            float4* dst = buf + pos * 5;
#pragma unroll
            for (int u = 0; u < 4; ++u) cp_async16(dst + u, src + 32 * u);
            cp_async8(dst + 4, lines.unit4_32(site, plane));
        }
        cp_async_commit();
    };

    M3<float> q = m_zero<float>();
    stage(0, ft_sm);
#pragma unroll 1
    for (int k = 0; k < 7; ++k) {
        const float4* cur = ft_sm + (k & 1) * FT_MAXPOS * 5;
        if (k + 1 < 7) {
            stage(k + 1, ft_sm + ((k + 1) & 1) * FT_MAXPOS * 5);
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        __syncthreads();
        const int a = c_shapes5[k].a, b = c_shapes5[k].b;
        const int Wm = FT_TN + 2 * b, Rm = (FT_TM + a) * Wm * FT_TT, Wn = FT_TN + b;
        // L(i, j): the line at offset (i mu + j nu) from the thread's site
        auto Lm = [&](int i, int j) { return lds_mat(cur + (((ml + i + a) * Wm + nl + j + b) * FT_TT + tl) * 5); };
        auto Ln = [&](int i, int j) {
            return lds_mat(cur + (Rm + ((ml + i + a) * Wn + nl + j + b) * FT_TT + tl) * 5);
        };
        M3<float> w;
        {
            const M3<float> m00 = Lm(0, 0);
            const M3<float> n00 = Ln(0, 0);
            M3<float> t = mm<false, false>(m00, Ln(a, 0));
            t = mm<false, true>(t, Lm(0, b));
            w = mm<false, true>(t, n00);  // TR
            const M3<float> ma0 = Lm(-a, 0);
            t = mm<false, true>(n00, Lm(-a, b));
            t = mm<false, true>(t, Ln(-a, 0));
            mac<false, false>(w, t, ma0);  // TL
            const M3<float> n0b = Ln(0, -b);
            t = mm<true, true>(ma0, Ln(-a, -b));
            t = mm<false, false>(t, Lm(-a, -b));
            mac<false, false>(w, t, n0b);  // BL
            t = mm<true, false>(n0b, Lm(0, -b));
            t = mm<false, false>(t, Ln(a, -b));
            mac<false, true>(w, t, m00);  // BR
        }
        m_axpy(q, (float)c_shapes5[k].c, w);
        __syncthreads();  // every thread is done with `cur` before it is refilled
    }
    const M3<float> f = ah_quarter(q);
    const double e = -(double)retr_mm<false, false>(f, f);
    const int64_t s = (int64_t)t0 + tl + (int64_t)(m0 + ml) * tg.stm + (int64_t)(n0 + nl) * tg.stn + obase;
    if (kout.p) kout.store(s, p, f);
    if (part) {
        const double rsum = block_sum(e, sh);
        if (threadIdx.x == 0) part[blockIdx.x] = rsum;
    }
}

// The tile kernel is used when the environment sets FLUE_FWD_TILE=1 (read at
// every launch; the L1/L2 kernel is the default, see the measurements beside
// k_fwd) for FP32 5-loop energies over spatial planes whose time extent is
// even and whose plane extents are multiples of the patch.
static bool fwd_tile_ok(const Geom& g, const PlaneArg& pa, int kind, bool fout, bool fits) {
    const char* env = getenv("FLUE_FWD_TILE");
    if (!env || atoi(env) != 1) return false;
    if (kind != 1 || fout || !fits || g.n[0] % FT_TT) return false;
    for (int q = 0; q < pa.np; ++q) {
        const int mu = pa.mu[q], nu = pa.nu[q];
        if (mu == 0 || nu == 0 || g.n[mu] % FT_TM || g.n[nu] % FT_TN) return false;
    }
    return true;
}

// ---------------------------------------------------------------------------
// 3. line cotangents: one thread per (site, slot, length)
// ---------------------------------------------------------------------------
constexpr int COT_BS = FLUE_COT_BS;



// Cotangent of the line l = L^len_e(P), P the thread's site, Q = P + len e.
// In a plane (e, f) the line is a side of the rectangles of shapes with a
// side len along e and w along f that lie on either side of it (SG = +1:
// towards +f, -1: towards -f).  Every such side, whatever its role (S1, S2,
// S3 = L^+, S4 = L^+), contributes the same form: going on from Q around the
// rectangle, A = the f-line Q -> R1 = Q + SG w f, B = the e-line R1 -> R2 =
// P + SG w f (against e, so daggered), C = the f-line R2 -> P, and
//     dLambda = SG o coef [K(Q) A B C + A K(R1) B C + A B K(R2) C + A B C K(P)]
// with o = +1 when e is the plane's first direction mu, -1 when it is nu
// (the clockwise walks are the daggers of the counter-clockwise leaf words:
// K^+ = -K).  K(Q) and K(P) are the same for every rectangle of the plane,
// so their two terms are summed over the plane's rectangles first:
//     Lambda_plane = K(Q) X + X K(P) + sum_sides SG o coef A Y,
//     X = sum_sides SG o coef A B C,   Y = K(R1) (B C) + B (K(R2) C),
// 4 full products and 2 with an anti-Hermitian K per side, and 2 of the
// latter per plane.  A is the stored line at Q (SG = +1) or the dagger of
// the one at R1 (-1); C the dagger of the one at P (+1) or the one at R2
// (-1); B the dagger of the e-line at R2.  SG is a template argument, so
// every dagger is folded into the products at compile time and only plain
// lines are stored.
template <int SG, typename T, typename I>
__device__ __forceinline__ void line_side(M3<T>& acc, M3<T>& X, T coef, const MatAoS<T>& lines, const AHAoS<T>& kin,
                                          int p, I s, I Q, I off, int pf, int pB) {
    constexpr bool DA = SG < 0, DC = SG > 0;
    const I R1 = Q + off, R2 = s + off;
    T kv[9];
    const M3<T> C = ldm(lines, DC ? s : R2, pf);
    M3<T> t = m_zero<T>();
    ldk(kin, R2, p, kv);
    mac_kx<DC>(t, kv, C);
    const M3<T> B = ldm(lines, R2, pB);
    M3<T> y = mm<true, false>(B, t);
    const M3<T> bc = mm<true, DC>(B, C);
    ldk(kin, R1, p, kv);
    mac_kx(y, kv, bc);
    const M3<T> A = ldm(lines, DA ? R1 : Q, pf);
    const M3<T> abc = mm<DA, false>(A, bc);
    const M3<T> ay = mm<DA, false>(A, y);
    const T sc = SG > 0 ? coef : -coef;
    m_axpy(X, sc, abc);
    m_axpy(acc, sc, ay);
}

template <typename T, typename I>
__device__ __forceinline__ void linecot_block(unsigned b, const Geom& g, const PlaneArg& pa, const MatAoS<T>& lines,
                                              const AHAoS<T>& kin, const MatAoS<T>& lam) {
    // the 3 * nd (direction, length) tasks of one site block run in adjacent
    // blocks, so the neighbourhood they all read stays in L2
    const int ntask = 3 * pa.nd;
    const int task = b % ntask;
    const int64_t s64 = site_block(b / ntask, g, blockDim.x) * blockDim.x + threadIdx.x;
    if (s64 >= g.V) return;
    const I s = (I)s64;
    const int slot = task / 3;
    const int len = task % 3 + 1;
    const int e = sel(pa.dir, slot);
    int c[4];
    site_coords(g, s64, c);
    int ce = 0, ne = 1;
    int64_t ste = 1;
#pragma unroll
    for (int k = 0; k < 4; ++k)
        if (k == e) ce = c[k], ne = g.n[k], ste = g.st[k];
    const I Q = s + (I)((int64_t)wrapd(ce, len, ne) * ste);
    const int pB = 3 * slot + len - 1;
    const int nw = len == 1 ? 3 : 2;
    M3<T> acc = m_zero<T>();
    for (int p = 0; p < pa.np; ++p) {
        const int pmu = sel(pa.mu, p), pnu = sel(pa.nu, p);
        if (pmu != e && pnu != e) continue;
        const int f = pmu == e ? pnu : pmu;
        const T o = pmu == e ? T(1) : T(-1);
        int cf = 0, nf = 1;
        int64_t stf = 1;
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (k == f) cf = c[k], nf = g.n[k], stf = g.st[k];
        const int kf = 3 * sel(pa.slot, f);
        M3<T> X = m_zero<T>();
#pragma unroll 1
        for (int j = 0; j < nw; ++j) {
            const int w = c_lw_w[len - 1][j];
            const T coef = lw_coef<T>(len, j) * o;
            const int pf = kf + w - 1;
            line_side<+1>(acc, X, coef, lines, kin, p, s, Q, (I)((int64_t)wrapd(cf, w, nf) * stf), pf, pB);
            line_side<-1>(acc, X, coef, lines, kin, p, s, Q, (I)((int64_t)wrapd(cf, -w, nf) * stf), pf, pB);
        }
        T kv[9];
        ldk(kin, Q, p, kv);
        mac_kx(acc, kv, X);
        ldk(kin, s, p, kv);
        mac_xk(acc, X, kv);
    }
    lam.store(s64, 3 * slot + len - 1, acc);
}

template <typename I>
__global__ void __launch_bounds__(COT_BS, FLUE_COT_MINB)
    k_linecot(Geom g, PlaneArg pa, MatAoS<float> lines, AHAoS<float> kin, MatAoS<float> lam) {
    linecot_block<float, I>(blockIdx.x, g, pa, lines, kin, lam);
}

template <typename I>
__global__ void __launch_bounds__(COT_BS) k_linecot_gated(Geom g, PlaneArg pa, MatAoS<double> lines, AHAoS<double> kin,
                                                          MatAoS<double> lam, unsigned nblocks, FixGate gt) {
    if (gate_shut(gt)) return;
    for (unsigned b = blockIdx.x; b < nblocks; b += gridDim.x) linecot_block<double, I>(b, g, pa, lines, kin, lam);
}

// line cotangents in fixed point: Lambda (180/512)^2 2^ks / 8, three warps
// (columns) for every 32 sites.  X K(P) mixes the columns of X, which the three
// warps exchange once a plane, through two buffers in turn (one barrier a plane:
// 42.3 -> 41.3 ms; barriers of the three warps alone 41.5).  32^3x64: FP64 pipe 202 ms; a thread a site
// 51.8 ms (its 255 registers spill), a thread a column 41.3 ms.
template <typename I>
__global__ void __launch_bounds__(3 * FIX_BS, 128 / FIX_BS)
    k_linecot_fix(Geom g, PlaneArg pa, MatFix lines, AHFix kin, MatFix lam, const u32* kmax, bool kslice, FixGate gt) {
    __shared__ int4 sx2[2][9][FIX_BS];
    if (!gt.open()) return;
    const int ntask = 3 * pa.nd;
    const int task = blockIdx.x % ntask;
    const int b = threadIdx.x / FIX_BS, jt = threadIdx.x % FIX_BS;
    const int64_t s64 = site_block(blockIdx.x / ntask, g, FIX_BS) * FIX_BS + jt;
    const bool live = s64 < g.V;
    const I s = (I)(live ? s64 : 0);
    const int slot = task / 3;
    const int len = task % 3 + 1;
    const int e = sel(pa.dir, slot);
    int c[4];
    site_coords(g, (int64_t)s, c);
    int ce = 0, ne = 1;
    int64_t ste = 1;
#pragma unroll
    for (int k = 0; k < 4; ++k)
        if (k == e) ce = c[k], ne = g.n[k], ste = g.st[k];
    const I Q = s + (I)((int64_t)wrapd(ce, len, ne) * ste);
    const int pB = 3 * slot + len - 1;
    const int nw = len == 1 ? 3 : 2;
    const int ks = kscale(kmax + (kslice ? c[0] : 0));
    FxVS acc = vs_zero();
    int par = 0;
#pragma unroll 1
    for (int p = 0; p < pa.np; ++p) {
        const int pmu = sel(pa.mu, p), pnu = sel(pa.nu, p);
        if (pmu != e && pnu != e) continue;
        const int f = pmu == e ? pnu : pmu;
        int cf = 0, nf = 1;
        int64_t stf = 1;
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (k == f) cf = c[k], nf = g.n[k], stf = g.st[k];
        const int kf = 3 * sel(pa.slot, f);
        FxVS X = vs_zero();
#pragma unroll 1
        for (int j = 0; j < nw; ++j) {
            const int w = c_lw_w[len - 1][j];
            const int cw = pmu == e ? c_lw_n[len - 1][j] : -c_lw_n[len - 1][j];
            const int pf = kf + w - 1;
            line_side_fix<+1>(acc, X, cw, lines, kin, p, ks, s, Q, (I)((int64_t)wrapd(cf, w, nf) * stf), pf, pB, b);
            line_side_fix<-1>(acc, X, cw, lines, kin, p, ks, s, Q, (I)((int64_t)wrapd(cf, -w, nf) * stf), pf, pB, b);
        }
        const FxV x = fx_of58(X);
        int4(*sx)[FIX_BS] = sx2[par];
        par ^= 1;
#pragma unroll
        for (int a = 0; a < 3; ++a) sx[3 * a + b][jt] = make_int4(x.r[a].h, x.r[a].l, x.i[a].h, x.i[a].l);
        Fx kv[9];
        kin.load(Q, p, ks, kv);
        fx_add_kv(acc, kv, fx_prep<false>(x));
        kin.load(s, p, ks, kv);
        const FxVP kc = fx_prep<false>(ah_col(kv, b));
        __syncthreads();
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            FxR m;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const int4 v = sx[3 * a + k][jt];
                m.r[k] = {v.x, v.y};
                m.i[k] = {v.z, v.w};
            }
            fx_row_sums<false>(m);
            fx_rdot_add(acc, a, m, kc);
        }
    }
    if (live) {
#pragma unroll
        for (int a = 0; a < 3; ++a)
            lam.store_el(s64, 3 * slot + len - 1, 3 * a + b, fx_of61(acc.r[a]), fx_of61(acc.i[a]));
    }
}

// ---------------------------------------------------------------------------
// 4. link cotangents and gradient output: one thread per (site, direction),
//    grid-strided so that a capped grid can write the gradient to host memory
//    beside other kernels
// ---------------------------------------------------------------------------
template <typename T>
__global__ void k_linkcot(Geom g, PlaneArg pa, MatAoS<T> lines, MatAoS<T> lam, T scale, int form, RefOut<T> out,
                          bool skip_zero, FixGate gt) {
    if constexpr (sizeof(T) == 8)
        if (gate_shut(gt)) return;
    const int d = blockIdx.y;
    const int slot = sel(pa.slot, d);
    if (slot < 0 && skip_zero) return;
    for (int64_t z = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; z < g.V; z += (int64_t)gridDim.x * blockDim.x) {
        if (slot < 0) {
            out.store(z, d, m_zero<T>());
            continue;
        }
        int c[4];
        site_coords(g, z, c);
        int cd = 0, nd = 1;
        int64_t sd = 1;
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (k == d) cd = c[k], nd = g.n[k], sd = g.st[k];
        const int64_t zp = z + (int64_t)wrapd(cd, 1, nd) * sd, zm = z + (int64_t)wrapd(cd, -1, nd) * sd,
                      zmm = z + (int64_t)wrapd(cd, -2, nd) * sd;
        const int l1 = 3 * slot, l2 = 3 * slot + 1;
        const M3<T> up = lines.load(zp, l1);
        const M3<T> um = lines.load(zm, l1);
        M3<T> n = lam.load(z, 3 * slot);
        mac<false, false>(n, up, lam.load(z, 3 * slot + 1));
        mac<false, false>(n, lam.load(zm, 3 * slot + 1), um);
        mac<false, false>(n, lines.load(zp, l2), lam.load(z, 3 * slot + 2));
        {
            const M3<T> t = mul(up, lam.load(zm, 3 * slot + 2));
            mac<false, false>(n, t, um);
        }
        mac<false, false>(n, lam.load(zmm, 3 * slot + 2), lines.load(zmm, l2));
        if (form == 0) {
            const M3<T> un = mul(lines.load(z, l1), n);
            out.store(z, d, ta_scaled(un, T(-0.5) * scale));
        } else {
            out.store(z, d, m_scale(dag(n), scale));
        }
    }
}

// link cotangents in fixed point: N (180/512)^2 2^ks / 8 from the stored
// Lambda; the Lie form's U N takes N shifted up to |entry| < 1/2
__global__ void __launch_bounds__(128) k_linkcot_fix(Geom g, PlaneArg pa, MatFix lines, MatFix lam, double scale,
                                                     int form, RefOut<double> out, bool skip_zero,
                                                     const u32* kmax, bool kslice, FixGate gt) {
    if (!gt.open()) return;
    const int d = blockIdx.y;
    const int slot = sel(pa.slot, d);
    if (slot < 0 && skip_zero) return;
    for (int64_t z = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; z < g.V; z += (int64_t)gridDim.x * blockDim.x) {
        if (slot < 0) {
            out.store(z, d, m_zero<double>());
            continue;
        }
        int c[4];
        site_coords(g, z, c);
        int cd = 0, nd = 1;
        int64_t sd = 1;
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (k == d) cd = c[k], nd = g.n[k], sd = g.st[k];
        const int64_t zp = z + (int64_t)wrapd(cd, 1, nd) * sd, zm = z + (int64_t)wrapd(cd, -1, nd) * sd,
                      zmm = z + (int64_t)wrapd(cd, -2, nd) * sd;
        const int l1 = 3 * slot, l2 = 3 * slot + 1;
        M3S n = s_zero();
        {
            const M3F up = lines.load(zp, l1);
            fx_mac<false, false>(n, up, lam.load(z, 3 * slot + 1));
            const M3F um = lines.load(zm, l1);
            fx_mac<false, false>(n, fx_mm<false, false>(up, lam.load(zm, 3 * slot + 2)), um);
            fx_mac<false, false>(n, lam.load(zm, 3 * slot + 1), um);
        }
        fx_mac<false, false>(n, lines.load(zp, l2), lam.load(z, 3 * slot + 2));
        fx_mac<false, false>(n, lam.load(zmm, 3 * slot + 2), lines.load(zmm, l2));
        {
            const M3F l = lam.load(z, 3 * slot);
#pragma unroll
            for (int k = 0; k < 9; ++k) {
                // h 2^-29 + l 2^-60 in units of 2^-58
                n.r[k] += ((i64)l.r[k].h << 29) + (l.r[k].l >> 2);
                n.i[k] += ((i64)l.i[k].h << 29) + (l.i[k].l >> 2);
            }
        }
        // unit 2^-58 and the factors the fixed-point sums leave out
        const double sc = ldexp(scale * (8.0 * FXQ5 * FXQ5) * 0x1p-58, -kscale(kmax + (kslice ? c[0] : 0)));
        M3<double> o;
        if (form == 0) {
            u32 big = 0;
#pragma unroll
            for (int k = 0; k < 9; ++k)
                big |= (u32)(n.r[k] >> 32) ^ (u32)(n.r[k] >> 63), big |= (u32)(n.i[k] >> 32) ^ (u32)(n.i[k] >> 63);
            const int up = max(0, __clz((int)big) - 4);
#pragma unroll
            for (int k = 0; k < 9; ++k) n.r[k] <<= up, n.i[k] <<= up;
            M3S un = s_zero();
            fx_mac<false, false>(un, lines.load(z, l1), fx_of61(n));
            // -1/2 TA: (M - M^+)/2 and a third of the trace off the diagonal
            const double s1 = sc * -0.25 * ldexp(8.0, -up), s3 = sc * (-0.5 / 3.0) * ldexp(8.0, -up);
            const i64 tr = un.i[0] + un.i[4] + un.i[8];
#pragma unroll
            for (int x = 0; x < 3; ++x) {
                o.r[4 * x] = 0.0;
                o.i[4 * x] = (double)(3 * un.i[4 * x] - tr) * s3;
#pragma unroll
                for (int y = x + 1; y < 3; ++y) {
                    const double cr = (double)(un.r[3 * x + y] - un.r[3 * y + x]) * s1;
                    const double ci = (double)(un.i[3 * x + y] + un.i[3 * y + x]) * s1;
                    o.r[3 * x + y] = cr;
                    o.i[3 * x + y] = ci;
                    o.r[3 * y + x] = -cr;
                    o.i[3 * y + x] = ci;
                }
            }
        } else {
#pragma unroll
            for (int x = 0; x < 3; ++x)
#pragma unroll
                for (int y = 0; y < 3; ++y) {
                    o.r[3 * x + y] = (double)n.r[3 * y + x] * sc;
                    o.i[3 * x + y] = (double)n.i[3 * y + x] * -sc;
                }
        }
        out.store(z, d, o);
    }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
static PlaneArg make_planes(const PlaneSet& ps) {
    PlaneArg pa;
    pa.np = ps.np;
    for (int k = 0; k < 4; ++k) pa.slot[k] = -1, pa.dir[k] = -1;
    pa.nd = 0;
    for (int p = 0; p < ps.np; ++p) {
        pa.mu[p] = ps.mu[p];
        pa.nu[p] = ps.nu[p];
        for (int d : {ps.mu[p], ps.nu[p]})
            if (pa.slot[d] < 0) {
                pa.slot[d] = pa.nd;
                pa.dir[pa.nd] = d;
                pa.nd++;
            }
    }
    return pa;
}

static inline size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

struct EnergyWs {
    size_t lines, kbuf, lam, part, gate, gate_bytes, total;  // gate: its counts, then kscale's slices
    bool fix;
};

// The scratch of one evaluation.  fix: complex128 fields with room for the
// fixed-point intermediates (whole tiles of 32 sites) and the gate; they share
// their place with the FP64 ones, since a field takes one of the two.
static EnergyWs energy_layout(const Geom& g, int prec, const PlaneArg& pa, bool with_force, bool fix) {
    const bool d = prec == PREC_C128;  // FP64 intermediates
    fix = fix && d;
    auto mat = [&](int64_t nk) {
        if (fix) return std::max(MatAoS<double>::bytes(g.V, nk), MatFix::bytes(g.V, nk));
        return d ? MatAoS<double>::bytes(g.V, nk) : MatAoS<float>::bytes(g.V, nk);
    };
    auto ah = [&](int64_t nk) {
        if (fix) return std::max(AHAoS<double>::bytes(g.V, nk), AHFix::bytes(g.V, nk));
        return d ? AHAoS<double>::bytes(g.V, nk) : AHAoS<float>::bytes(g.V, nk);
    };
    EnergyWs w;
    w.fix = fix;
    const int fbs = fix ? FIX_BS_SMALL : FWD_BS;  // (any SM count's choice of fix_fwd_block fits)
    const int nbx = (int)((g.V + fbs - 1) / fbs);
    w.lines = 0;
    // K and the line cotangents only with a gradient
    w.kbuf = align256(w.lines + mat(3 * pa.nd));
    w.lam = align256(w.kbuf + (with_force ? ah(pa.np) : 0));
    w.part = align256(w.lam + (with_force ? mat(3 * pa.nd) : 0));
    w.gate = align256(w.part + (size_t)pa.np * nbx * sizeof(double));
    w.gate_bytes = fix ? (GATE_WORDS + (size_t)g.n[0]) * sizeof(u32) : 0;
    w.total = align256(w.gate + w.gate_bytes);
    return w;
}

// the layout that fits ws_bytes: with the fixed-point intermediates, else
// without (a workspace sized for the FP64 ones alone stays enough)
static EnergyWs energy_layout_for(const Geom& g, int prec, const PlaneArg& pa, bool with_force, size_t ws_bytes) {
    const EnergyWs w = energy_layout(g, prec, pa, with_force, true);
    return ws_bytes >= w.total ? w : energy_layout(g, prec, pa, with_force, false);
}

size_t energy_ws_bytes(const Geom& g, int prec, const PlaneSet& ps, bool with_force) {
    return energy_layout(g, prec, make_planes(ps), with_force, true).total;
}
size_t energy_ws_min_bytes(const Geom& g, int prec, const PlaneSet& ps, bool with_force) {
    return energy_layout(g, prec, make_planes(ps), with_force, false).total;
}

// Optional per-stage timing of the energy pipeline (CUDA events recorded on
// the caller's stream between the stage launches): stage 0 lines, 1 forward
// (+ sum), 2 line cotangents, 3 link cotangents.
static bool g_stage_on = false;
static cudaEvent_t g_stage_ev[5] = {};
static int g_stage_n = 0;

cudaError_t stage_timing_enable(int on) {
    if (on && !g_stage_ev[0]) {
        for (auto& e : g_stage_ev) {
            cudaError_t r = cudaEventCreate(&e);
            if (r != cudaSuccess) return r;
        }
    }
    g_stage_on = on != 0;
    g_stage_n = 0;
    return cudaSuccess;
}

cudaError_t stage_times(double* ms, int maxn, int* n) {
    *n = 0;
    if (!g_stage_on || g_stage_n < 2) return cudaSuccess;
    cudaError_t r = cudaEventSynchronize(g_stage_ev[g_stage_n - 1]);
    if (r != cudaSuccess) return r;
    for (int k = 0; k + 1 < g_stage_n && k < maxn; ++k) {
        float t = 0.f;
        r = cudaEventElapsedTime(&t, g_stage_ev[k], g_stage_ev[k + 1]);
        if (r != cudaSuccess) return r;
        ms[k] = t;
        *n = k + 1;
    }
    return cudaSuccess;
}

static inline void stage_mark(int k, cudaStream_t st) {
    if (g_stage_on) {
        cudaEventRecord(g_stage_ev[k], st);
        g_stage_n = k + 1;
    }
}

// The gate of one evaluation's workspace (p = NULL without the fixed-point
// path): open when a quarter of its links is away from 1 and all are unitary.
static FixGate energy_gate(const Geom& g, const PlaneArg& pa, char* ws, const EnergyWs& w) {
    FixGate gt;
    if (w.fix) {
        gt.p = (u32*)(ws + w.gate);
        gt.need = (u32)(((uint64_t)g.V * pa.nd + 3) / 4);
    }
    return gt;
}
// Grid of a gated FP64 kernel of n blocks: all of them when it always runs,
// else at most 8 a SM, so that the blocks that leave at once cost little.
static unsigned gated_grid(const EnergyWs& w, unsigned n) {
    return w.fix ? std::min(n, 8u * (unsigned)device_sms()) : n;
}

// Part 1 of the pipeline: lines, forward (+ energy sum normalised by vnorm),
// line cotangents when `with_force`.
template <class L, typename T>
static cudaError_t energy_fwd_part(const L& U, const Geom& g, const Geom& gs, int t0, const PlaneArg& pa, int kind,
                                   double* out_E, bool with_force, double vnorm, char* ws, const EnergyWs& w,
                                   RefOut<T> fout, cudaStream_t st) {
    MatAoS<T> lines{reinterpret_cast<decltype(MatAoS<T>::p)>(ws + w.lines), g.V, 3 * pa.nd};
    AHAoS<T> kb{with_force ? reinterpret_cast<decltype(AHAoS<T>::p)>(ws + w.kbuf) : nullptr, g.V, pa.np};
    MatAoS<T> lam{reinterpret_cast<decltype(MatAoS<T>::p)>(ws + w.lam), g.V, 3 * pa.nd};
    double* part = out_E ? (double*)(ws + w.part) : nullptr;
    const unsigned nbl = (unsigned)((g.V + 127) / 128);
    const int fbs = w.fix ? fix_fwd_block(g.V, pa.np) : FWD_BS;  // sites a block of the forward covers
    const unsigned nbx = (unsigned)((g.V + fbs - 1) / fbs);
    const unsigned nbc = (unsigned)((g.V + COT_BS - 1) / COT_BS);
    const PatchArg pt = FLUE_FWD_PATCH ? make_patch(g, pa, fbs) : PatchArg{};
    const bool fits = MatAoS<T>::fits32(g.V, 3 * pa.nd), cfits = fits && AHAoS<T>::fits32(g.V, pa.np);
    const bool ksl = pa.slot[0] < 0;  // no plane steps in time: one scale of K per time slice
    cudaError_t e = cudaSuccess;
    stage_mark(0, st);
    if constexpr (sizeof(T) == 8) {
        const FixGate gt = energy_gate(g, pa, ws, w);
        const MatFix flines{(int4*)(ws + w.lines), g.V, 3 * pa.nd};
        const AHFix fkb{with_force ? (longlong2*)(ws + w.kbuf) : nullptr, g.V, pa.np};
        const bool ffits = MatFix::fits32(g.V, 3 * pa.nd);
        if (w.fix) {
            if ((e = cudaMemsetAsync(gt.p, 0, w.gate_bytes, st)) != cudaSuccess) return e;
            note_launch(), k_lines_fix<<<dim3(nbl, pa.nd), 128, 0, st>>>(U, g, gs, t0, pa, flines, gt);
        }
        note_launch(), k_lines_gated<<<dim3(gated_grid(w, nbl), pa.nd), 128, 0, st>>>(U, g, gs, t0, pa, lines, gt);
        stage_mark(1, st);
        if (w.fix) {
            auto fwd = [&](auto kernel) {
                note_launch(), kernel<<<nbx * pa.np, 3 * fbs, 0, st>>>(g, pa, kind, pt, flines, fkb, fout, part,
                                                                       gt.p + GATE_WORDS, ksl, gt);
            };
            if (fbs == FIX_BS_SMALL)
                fwd(k_fwd_fix<FIX_BS_SMALL, u32>);  // (a small lattice fits 32-bit offsets)
            else if (ffits)
                fwd(k_fwd_fix<FIX_BS, u32>);
            else
                fwd(k_fwd_fix<FIX_BS, int64_t>);
        }
        const unsigned nf = (unsigned)((g.V + FWD_BS - 1) / FWD_BS) * pa.np, gf = gated_grid(w, nf);
        const PatchArg pt64 = FLUE_FWD_PATCH ? make_patch(g, pa, FWD_BS) : PatchArg{};
        auto fwd64 = [&](auto kernel) {
            note_launch(), kernel<<<gf, FWD_BS, 0, st>>>(g, pa, kind, pt64, lines, kb, fout, part, nf, nbx * pa.np, gt);
        };
        if (fits)
            fwd64(k_fwd_gated<u32>);
        else
            fwd64(k_fwd_gated<int64_t>);
    } else {
        note_launch(), k_lines<L><<<dim3(nbl, pa.nd), 128, 0, st>>>(U, g, gs, t0, pa, lines);
        stage_mark(1, st);
        bool tiled = false;
        if (fwd_tile_ok(g, pa, kind, fout.p != nullptr, fits)) {
            static_assert(FT_BS == FWD_BS, "the tile forward writes one partial per FWD_BS sites");
            // (the attribute is per function and per device; setting it again is harmless)
            cudaError_t ae = cudaFuncSetAttribute(k_fwd_tile, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FT_SMEM);
            if (ae != cudaSuccess) return ae;
            note_launch(), k_fwd_tile<<<nbx * pa.np, FT_BS, FT_SMEM, st>>>(g, pa, lines, kb, part);
            tiled = true;
        }
        if (!tiled) {
            if (fits)
                note_launch(), k_fwd<uint32_t><<<nbx * pa.np, FWD_BS, 0, st>>>(g, pa, kind, pt, lines, kb, fout, part);
            else
                note_launch(), k_fwd<int64_t><<<nbx * pa.np, FWD_BS, 0, st>>>(g, pa, kind, pt, lines, kb, fout, part);
        }
    }
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if (out_E) {
        e = launch_finish_sums(part, (int)(nbx * pa.np), 1, out_E, st, 1.0 / vnorm);
        if (e != cudaSuccess) return e;
    }
    stage_mark(2, st);
    if (!with_force) return cudaSuccess;
    if constexpr (sizeof(T) == 8) {
        const FixGate gt = energy_gate(g, pa, ws, w);
        const MatFix flines{(int4*)(ws + w.lines), g.V, 3 * pa.nd}, flam{(int4*)(ws + w.lam), g.V, 3 * pa.nd};
        const AHFix fkb{(longlong2*)(ws + w.kbuf), g.V, pa.np};
        const unsigned nl = nbc * 3 * pa.nd, gl = gated_grid(w, nl);
        if (w.fix) {
            const unsigned nlf = (unsigned)((g.V + FIX_BS - 1) / FIX_BS) * 3 * pa.nd;
            auto cot = [&](auto kernel) {
                note_launch(), kernel<<<nlf, 3 * FIX_BS, 0, st>>>(g, pa, flines, fkb, flam, gt.p + GATE_WORDS, ksl, gt);
            };
            if (MatFix::fits32(g.V, 3 * pa.nd) && AHFix::fits32(g.V, pa.np))
                cot(k_linecot_fix<u32>);
            else
                cot(k_linecot_fix<int64_t>);
        }
        if (cfits)
            note_launch(), k_linecot_gated<u32><<<gl, COT_BS, 0, st>>>(g, pa, lines, kb, lam, nl, gt);
        else
            note_launch(), k_linecot_gated<int64_t><<<gl, COT_BS, 0, st>>>(g, pa, lines, kb, lam, nl, gt);
    } else {
        if (cfits)
            note_launch(), k_linecot<uint32_t><<<nbc * 3 * pa.nd, COT_BS, 0, st>>>(g, pa, lines, kb, lam);
        else
            note_launch(), k_linecot<int64_t><<<nbc * 3 * pa.nd, COT_BS, 0, st>>>(g, pa, lines, kb, lam);
    }
    stage_mark(3, st);
    return cudaGetLastError();
}

// Part 2: link cotangents, gradient of E/vnorm written through `fo`.
template <typename T>
static cudaError_t energy_out_part(const Geom& g, const PlaneArg& pa, double vnorm, int form, char* ws,
                                   const EnergyWs& w, RefOut<T> fo, unsigned max_blocks, cudaStream_t st,
                                   bool skip_zero = false) {
    MatAoS<T> lines{reinterpret_cast<decltype(MatAoS<T>::p)>(ws + w.lines), g.V, 3 * pa.nd};
    MatAoS<T> lam{reinterpret_cast<decltype(MatAoS<T>::p)>(ws + w.lam), g.V, 3 * pa.nd};
    const T scale = (T)(-1.0 / (2.0 * vnorm));
    unsigned nb = (unsigned)((g.V + 127) / 128);
    if (max_blocks && nb > max_blocks) nb = max_blocks;
    FixGate gt;
    unsigned nbg = nb;
    if constexpr (sizeof(T) == 8) {
        gt = energy_gate(g, pa, ws, w);
        if (w.fix) {
            const MatFix flines{(int4*)(ws + w.lines), g.V, 3 * pa.nd}, flam{(int4*)(ws + w.lam), g.V, 3 * pa.nd};
            note_launch(), k_linkcot_fix<<<dim3(nb, 4), 128, 0, st>>>(g, pa, flines, flam, scale, form, fo, skip_zero,
                                                                   gt.p + GATE_WORDS, pa.slot[0] < 0, gt);
            nbg = gated_grid(w, nb);
        }
    }
    note_launch(), k_linkcot<T><<<dim3(nbg, 4), 128, 0, st>>>(g, pa, lines, lam, scale, form, fo, skip_zero, gt);
    stage_mark(4, st);
    return cudaGetLastError();
}

template <class L, typename T>
static cudaError_t energy_impl(const L& U, const Geom& g, const PlaneArg& pa, int kind, double* out_E, void* force,
                               int form, char* ws, const EnergyWs& w, RefOut<T> fout, cudaStream_t st) {
    using C2 = typename V2<T>::type;
    cudaError_t e =
        energy_fwd_part<L, T>(U, g, g, 0, pa, kind, out_E, force != nullptr, (double)g.V, ws, w, fout, st);
    if (e != cudaSuccess || !force) return e;
    RefOut<T> fo{(C2*)force, g.V, 4};
    return energy_out_part<T>(g, pa, (double)g.V, form, ws, w, fo, 0, st);
}

cudaError_t launch_energy(const FieldRef& U, const PlaneSet& ps, double* out_E, void* force, int force_form, void* ws,
                          size_t ws_bytes, cudaStream_t st) {
    const PlaneArg pa = make_planes(ps);
    const EnergyWs w = energy_layout_for(U.g, U.prec, pa, force != nullptr, ws_bytes);
    if (ws_bytes < w.total) return cudaErrorInvalidValue;
    FLUE_DISPATCH_LINKS(U, {
        RefOut<T> none{nullptr, U.g.V, 1};
        return energy_impl<decltype(L), T>(L, U.g, pa, 1, out_E, force, force_form, (char*)ws, w, none, st);
    });
    return cudaSuccess;
}

static bool has_time_plane(const PlaneSet& ps) {
    for (int p = 0; p < ps.np; ++p)
        if (ps.mu[p] == 0 || ps.nu[p] == 0) return true;
    return false;
}

cudaError_t launch_energy_slab_fwd(const FieldRef& U, int t0, int nts, const PlaneSet& ps, int64_t vfull,
                                   double* out_E, bool with_force, void* ws, size_t ws_bytes, cudaStream_t st) {
    if (has_time_plane(ps) || t0 < 0 || nts < 1 || t0 + nts > U.g.n[0]) return cudaErrorInvalidValue;
    const Geom g = make_geom(nts, U.g.n[1], U.g.n[2], U.g.n[3]);
    if (vfull < g.V) return cudaErrorInvalidValue;
    const PlaneArg pa = make_planes(ps);
    const EnergyWs w = energy_layout_for(g, U.prec, pa, with_force, ws_bytes);
    if (ws_bytes < w.total) return cudaErrorInvalidValue;
    FLUE_DISPATCH_LINKS(U, {
        RefOut<T> none{nullptr, g.V, 1};
        return energy_fwd_part<decltype(L), T>(L, g, U.g, t0, pa, 1, out_E, with_force, (double)vfull, (char*)ws, w,
                                               none, st);
    });
    return cudaSuccess;
}

cudaError_t launch_energy_slab_out(const FieldRef& U, const PlaneSet& ps, int64_t vfull, int ntf, int t0, void* force,
                                   int force_form, void* ws, size_t ws_bytes, unsigned max_blocks, cudaStream_t st,
                                   int out_dtype, bool skip_zero) {
    if (has_time_plane(ps) || vfull < U.g.V || t0 < 0 || t0 + U.g.n[0] > ntf) return cudaErrorInvalidValue;
    const PlaneArg pa = make_planes(ps);
    const EnergyWs w = energy_layout_for(U.g, U.prec, pa, true, ws_bytes);
    if (ws_bytes < w.total) return cudaErrorInvalidValue;
    // the gradient array: time extent ntf, the slab's spatial extents (the
    // whole lattice's gradient, or a chunk of ntf time slices of it); vfull
    // only normalises
    const int64_t vout = (int64_t)ntf * (U.g.V / U.g.n[0]);
    if (U.prec == PREC_C128) {
        if (out_dtype != PREC_C128) return cudaErrorInvalidValue;
        RefOut<double> fo{(double2*)force, vout, 4, U.g.n[0], ntf, t0};
        return energy_out_part<double>(U.g, pa, (double)vfull, force_form, (char*)ws, w, fo, max_blocks, st,
                                       skip_zero);
    }
    RefOut<float> fo{(float2*)force, vout, 4, U.g.n[0], ntf, t0};
    if (out_dtype == PREC_C128) fo.p = nullptr, fo.pd = (double2*)force;
    return energy_out_part<float>(U.g, pa, (double)vfull, force_form, (char*)ws, w, fo, max_blocks, st, skip_zero);
}

// ---------------------------------------------------------------------------
// Energy (and gradient) of a device field over time slabs on several streams.
// Plane sets without the time direction (B^2) leave time slices independent,
// so the field is processed as nslab slabs of consecutive time slices, slab
// k on stream k % nstream (the caller's stream and nstream - 1 library
// streams, forked from and joined back to the caller's stream by events).
// The memory-bound stages (lines, link cotangents) of one slab then overlap
// the compute-bound ones of another, and each slab's intermediates are 1/nslab
// of the lattice's.  Per-slab energies are added in slab order by one
// finisher; the gradient is written in place through the slab mapping, so
// both are bitwise independent of the stream schedule.
// ---------------------------------------------------------------------------
namespace {
constexpr int kMaxSlabStreams = 4;
struct SlabStreams {
    std::mutex m;
    cudaStream_t s[kMaxSlabStreams - 1] = {};
    cudaEvent_t fork = nullptr, join[kMaxSlabStreams - 1] = {};
};
std::mutex g_slab_mtx;
SlabStreams* g_slab[64] = {};

cudaError_t slab_streams(SlabStreams** out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lk(g_slab_mtx);
    if (!g_slab[dev]) {
        SlabStreams* ss = new SlabStreams();
        for (int i = 0; i < kMaxSlabStreams - 1 && e == cudaSuccess; ++i) {
            e = cudaStreamCreateWithFlags(&ss->s[i], cudaStreamNonBlocking);
            if (e == cudaSuccess) e = cudaEventCreateWithFlags(&ss->join[i], cudaEventDisableTiming);
        }
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&ss->fork, cudaEventDisableTiming);
        if (e != cudaSuccess) return e;  // (a failed setup keeps its handles; it is retried on the next call)
        g_slab[dev] = ss;
    }
    *out = g_slab[dev];
    return cudaSuccess;
}

struct SlabWs {
    size_t slot, spart, total;
};
SlabWs slab_ws_layout(const Geom& g, int prec, const PlaneArg& pa, bool with_force, int nslab, int nstream, bool fix) {
    const int nts = (g.n[0] + nslab - 1) / nslab;
    const Geom gs = make_geom(nts, g.n[1], g.n[2], g.n[3]);
    SlabWs w;
    w.slot = energy_layout(gs, prec, pa, with_force, fix).total;
    w.spart = (size_t)nstream * w.slot;
    w.total = align256(w.spart + (size_t)nslab * sizeof(double));
    return w;
}
}  // namespace

bool stage_timing_on() { return g_stage_on; }

size_t energy_slabs_ws_min_bytes(const Geom& g, int prec, const PlaneSet& ps, bool with_force, int nslab, int nstream) {
    return slab_ws_layout(g, prec, make_planes(ps), with_force, nslab, nstream, false).total;
}
size_t energy_slabs_ws_bytes(const Geom& g, int prec, const PlaneSet& ps, bool with_force, int nslab, int nstream) {
    return slab_ws_layout(g, prec, make_planes(ps), with_force, nslab, nstream, true).total;
}

cudaError_t launch_energy_slabs(const FieldRef& U, const PlaneSet& ps, double* out_E, void* force, int form, void* ws,
                                size_t ws_bytes, int nslab, int nstream, cudaStream_t st) {
    if (has_time_plane(ps) || nslab < 1 || nslab > U.g.n[0] || nstream < 1 || nstream > kMaxSlabStreams)
        return cudaErrorInvalidValue;
    const PlaneArg pa = make_planes(ps);
    const bool with_force = force != nullptr;
    SlabWs w = slab_ws_layout(U.g, U.prec, pa, with_force, nslab, nstream, true);
    if (ws_bytes < w.total) w = slab_ws_layout(U.g, U.prec, pa, with_force, nslab, nstream, false);
    if (ws_bytes < w.total) return cudaErrorInvalidValue;
    const int nts = (U.g.n[0] + nslab - 1) / nslab;
    nslab = (U.g.n[0] + nts - 1) / nts;
    if (nstream > nslab) nstream = nslab;
    SlabStreams* ss = nullptr;
    cudaError_t e = slab_streams(&ss);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lk(ss->m);
    double* spart = out_E ? (double*)((char*)ws + w.spart) : nullptr;
    if ((e = cudaEventRecord(ss->fork, st)) != cudaSuccess) return e;
    for (int i = 1; i < nstream; ++i)
        if ((e = cudaStreamWaitEvent(ss->s[i - 1], ss->fork, 0)) != cudaSuccess) return e;
    for (int k = 0; k < nslab && e == cudaSuccess; ++k) {
        const int i = k % nstream, t0 = k * nts, n = U.g.n[0] - t0 < nts ? U.g.n[0] - t0 : nts;
        cudaStream_t sk = i == 0 ? st : ss->s[i - 1];
        char* slot = (char*)ws + (size_t)i * w.slot;
        e = launch_energy_slab_fwd(U, t0, n, ps, U.g.V, spart ? spart + k : nullptr, with_force, slot, w.slot, sk);
        if (e == cudaSuccess && with_force) {
            const FieldRef Us{U.links, make_geom(n, U.g.n[1], U.g.n[2], U.g.n[3]), U.prec};
            e = launch_energy_slab_out(Us, ps, U.g.V, U.g.n[0], t0, force, form, slot, w.slot, 0, sk,
                                       U.prec == PREC_C128 ? PREC_C128 : PREC_C64);
        }
    }
    // join every library stream back into the caller's stream, also on error
    for (int i = 1; i < nstream; ++i) {
        cudaError_t r = cudaEventRecord(ss->join[i - 1], ss->s[i - 1]);
        if (r == cudaSuccess) r = cudaStreamWaitEvent(st, ss->join[i - 1], 0);
        if (e == cudaSuccess) e = r;
    }
    if (e == cudaSuccess && out_E) e = launch_finish_sums(spart, nslab, 1, out_E, st, 1.0);
    return e;
}

// Clover of an FP32 field straight from the links: its only lines are links, so
// the line buffers were a copy of them, written and read back.  12 products from
// eight links a site, the links' second and third reads from L2: latency and L2
// bound.  24^3x48 c64 117 us through the line buffers, 60 us so, at 4 blocks of
// 128 an SM (128 registers; with 3 the latency is less hidden, with 5 it spills).
constexpr int CLOVER_MINB = 4;
template <class L, typename I>
__global__ void __launch_bounds__(FWD_BS, CLOVER_MINB) k_clover(L U, Geom g, int mu, int nu, RefOut<float> fout) {
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= g.V) return;
    int c[4];
    site_coords(g, s, c);
    int mM = 0, mP = 0, nM = 0, nP = 0;
#pragma unroll
    for (int d = 0; d < 4; ++d) {
        const int up = wrapd(c[d], 1, g.n[d]) * (int)g.st[d], dn = wrapd(c[d], -1, g.n[d]) * (int)g.st[d];
        if (d == mu) mP = up, mM = dn;
        if (d == nu) nP = up, nM = dn;
    }
    const M3<float> q = four_leaves<float>([&](int site) { return U.load((I)site, mu); },
                                           [&](int site) { return U.load((I)site, nu); }, (int)s, mM, mP, nM, nP);
    fout.store(s, 0, transp(ah_quarter(q)));
}

// F_munu of one plane: kind 0 = clover (cloverLoopMuNuCoord), 1 = 5-loop
// (Loop5MuNuCoord).  Output (NT,NX,NY,NZ,3,3) in the field's compute dtype.
cudaError_t launch_fmunu(const FieldRef& U, int kind, int mu, int nu, void* out, void* ws, size_t ws_bytes,
                         cudaStream_t st) {
    PlaneSet ps;
    ps.np = 1;
    ps.mu[0] = mu;
    ps.nu[0] = nu;
    const PlaneArg pa = make_planes(ps);
    const EnergyWs w = energy_layout_for(U.g, U.prec, pa, false, ws_bytes);
    if (ws_bytes < w.total) return cudaErrorInvalidValue;
    if (kind == 0 && U.prec != PREC_C128) {
        const RefOut<float> fo{(float2*)out, U.g.V, 1};
        const unsigned nb = (unsigned)((U.g.V + FWD_BS - 1) / FWD_BS);
        stage_mark(0, st);
        stage_mark(1, st);  // (no lines)
        if (U.prec == PREC_R12)
            note_launch(), k_clover<R12Links, int64_t><<<nb, FWD_BS, 0, st>>>(R12Links{(const float4*)U.links, U.g.V}, U.g, mu, nu, fo);
        else if (FullLinks32::fits(U.g.V))
            note_launch(), k_clover<FullLinks32, u32><<<nb, FWD_BS, 0, st>>>(FullLinks32{(const char*)U.links, (u32)U.g.V}, U.g, mu, nu, fo);
        else
            note_launch(), k_clover<FullLinks<float>, int64_t><<<nb, FWD_BS, 0, st>>>(FullLinks<float>{(const float2*)U.links, U.g.V}, U.g, mu, nu, fo);
        stage_mark(2, st);
        return cudaGetLastError();
    }
    FLUE_DISPATCH_LINKS(U, {
        using C2 = typename V2<T>::type;
        RefOut<T> fo{(C2*)out, U.g.V, 1};
        return energy_impl<decltype(L), T>(L, U.g, pa, kind, nullptr, nullptr, 0, (char*)ws, w, fo, st);
    });
    return cudaSuccess;
}

// ---------------------------------------------------------------------------
// Wilson plaquette action S = sum_{x,mu<nu} Re Tr P_munu(x) and its gradient:
// N_mu(x) = sum_{nu != mu} [U_nu(x+mu) U_mu(x+nu)^+ U_nu(x)^+
//                           + U_nu(x+mu-nu)^+ U_mu(x-nu)^+ U_nu(x-nu)]
// ---------------------------------------------------------------------------
constexpr int PF_BS = 128;
int plaqforce_blocks(const Geom& g) { return (int)((g.V + PF_BS - 1) / PF_BS); }

// Staple sum and gradient of direction MU at site s; MU and the staple
// directions are compile-time, so every coordinate and stride is a register.
template <int MU, class L, typename T>
__device__ __forceinline__ double plaqforce_dir(const L& U, const Geom& g, int64_t s, const int c[4], int form,
                                                const RefOut<T>& out) {
    const int64_t sp = s + (int64_t)wrapd(c[MU], 1, g.n[MU]) * g.st[MU];
    const M3<T> u = U.load(s, MU);
    M3<T> n = m_zero<T>();
    double acc = 0.0;
#pragma unroll
    for (int nu = 0; nu < 4; ++nu) {
        if (nu == MU) continue;
        const int64_t dn1 = (int64_t)wrapd(c[nu], 1, g.n[nu]) * g.st[nu];
        const int64_t dm1 = (int64_t)wrapd(c[nu], -1, g.n[nu]) * g.st[nu];
        const M3<T> up = mm<false, true>(U.load(sp, nu), U.load(s + dn1, MU));
        const M3<T> upper = mm<false, true>(up, U.load(s, nu));
        if (nu > MU) acc += (double)retr_mm<false, false>(u, upper);
        m_add(n, upper);
        const M3<T> dn = mm<true, true>(U.load(sp + dm1, nu), U.load(s + dm1, MU));
        mac<false, false>(n, dn, U.load(s + dm1, nu));
    }
    if (out.p) {
        if (form == 0)
            out.store(s, MU, ta_scaled(mul(u, n), T(-0.5)));
        else
            out.store(s, MU, dag(n));
    }
    return acc;
}

// Minimum resident blocks per SM (register cap) of k_plaqforce, measured on
// GB300 at 32^3x64: c64 2.03 ms per call with runtime directions (80-byte
// local frame), 1.64 with compile-time ones, 1.48 capped at 3 blocks; r12
// 1.27 -> 1.15 capped at 4; FP64 keeps its registers (21.1 ms either way).
template <class L, typename T>
struct PfMinBlocks {
    static constexpr int v = sizeof(T) == 4 ? 3 : 1;
};
template <>
struct PfMinBlocks<R12Links, float> {
    static constexpr int v = 4;
};

// block b of nb (the grid's x) of direction d
template <class L, typename T>
__device__ __forceinline__ void plaqforce_block(unsigned b, unsigned nb, int d, const L& U, const Geom& g, int form,
                                                const RefOut<T>& out, double* part, double* sh) {
    const int64_t s = (int64_t)b * blockDim.x + threadIdx.x;
    double acc = 0.0;
    if (s < g.V) {
        int c[4];
        site_coords(g, s, c);
        switch (d) {
            case 0: acc = plaqforce_dir<0>(U, g, s, c, form, out); break;
            case 1: acc = plaqforce_dir<1>(U, g, s, c, form, out); break;
            case 2: acc = plaqforce_dir<2>(U, g, s, c, form, out); break;
            default: acc = plaqforce_dir<3>(U, g, s, c, form, out); break;
        }
    }
    if (part) {
        const double r = block_sum(acc, sh);
        if (threadIdx.x == 0) part[(int64_t)d * nb + b] = r;
    }
}

template <class L, typename T>
__global__ void __launch_bounds__(PF_BS, PfMinBlocks<L, T>::v)
    k_plaqforce(L U, Geom g, int form, RefOut<T> out, double* part) {
    __shared__ double sh[32];
    plaqforce_block<L, T>(blockIdx.x, gridDim.x, blockIdx.y, U, g, form, out, part, sh);
}

// the FP64 force behind a gate, its grid capped (the Wilson flow's fields that
// do not take fixed point)
__global__ void __launch_bounds__(PF_BS)
    k_plaqforce_gated(FullLinks<double> U, Geom g, RefOut<double> out, unsigned nb, FixGate gt) {
    __shared__ double sh[32];
    if (gate_shut(gt)) return;
    for (unsigned b = blockIdx.x; b < nb; b += gridDim.x)
        plaqforce_block<FullLinks<double>, double>(b, nb, blockIdx.y, U, g, 0, out, nullptr, sh);
}

cudaError_t launch_plaquette_force_gated(const FieldRef& U, void* force, const FixGate& gt, cudaStream_t st) {
    const unsigned nb = (unsigned)plaqforce_blocks(U.g), cap = 8u * (unsigned)device_sms();
    const FullLinks<double> L{(const double2*)U.links, U.g.V};
    const RefOut<double> fo{(double2*)force, U.g.V, 4};
    note_launch(), k_plaqforce_gated<<<dim3(std::min(nb, cap), 4), PF_BS, 0, st>>>(L, U.g, fo, nb, gt);
    return cudaGetLastError();
}

cudaError_t launch_plaquette_force(const FieldRef& U, double* part, double* out_S, void* force, int force_form,
                                   cudaStream_t st) {
    const int nb = plaqforce_blocks(U.g);
    FLUE_DISPATCH_LINKS(U, {
        using C2 = typename V2<T>::type;
        RefOut<T> fo{(C2*)force, U.g.V, 4};
        note_launch(), k_plaqforce<decltype(L), T><<<dim3(nb, 4), PF_BS, 0, st>>>(L, U.g, force_form, fo, out_S ? part : nullptr);
    });
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess || !out_S) return e;
    return launch_finish_sums(part, 4 * nb, 1, out_S, st);
}

FLUE_OOB_READER(force)

}  // namespace flue
