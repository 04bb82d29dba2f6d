// observables.cu -- layout conversion, SU(3) batch products, and the scalar
// observables of src/wloops.F90: plaquette (:915-1017, same observable as
// genPlaquette :59-127), polyakov (:1019-1069), wmunu / wmunutau
// (:567-791), genericPath (:20-57) and the Landau-gauge mean link used by
// uzerobar.  Every scalar is accumulated per thread in FP64 (the FP32 path
// computes link products in FP32 and converts each per-site trace), reduced
// per block with warp shuffles, and finished by a one-block kernel that adds
// the block partials in index order, so results are bitwise reproducible for
// a given lattice size.
#include <algorithm>
#include <atomic>

#include "flue_internal.h"

namespace flue {

static inline int grid_for(int64_t n, int bs, int cap) {
    int64_t b = (n + bs - 1) / bs;
    if (b > cap) b = cap;
    if (b < 1) b = 1;
    return (int)b;
}

int device_sms() {
    static std::atomic<int> cache[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
        cudaGetLastError();
        return 152;
    }
    int n = cache[dev].load(std::memory_order_relaxed);
    if (n > 0) return n;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1) {
        cudaGetLastError();
        return 152;
    }
    cache[dev].store(n, std::memory_order_relaxed);
    return n;
}

// Grid-strided reductions run 4 blocks per SM of the current device, at most
// kMaxRedBlocks; their partial-sum workspaces are sized for kMaxRedBlocks.
static int red_cap() {
    const int c = 4 * device_sms();
    return c > kMaxRedBlocks ? kMaxRedBlocks : c;
}

// ---------------------------------------------------------------------------
// reduction finisher
// ---------------------------------------------------------------------------
__device__ __forceinline__ void finish_sum(const double* p, int nparts, double scale, double* out, double* sh) {
    double acc = 0.0;
    int i = threadIdx.x;
    const int st = blockDim.x;
    for (; i + 7 * st < nparts; i += 8 * st) {  // eight loads in flight, added in order
        double v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = __ldcg(p + i + k * st);
#pragma unroll
        for (int k = 0; k < 8; ++k) acc += v[k];
    }
    for (; i < nparts; i += st) acc += p[i];
    double r = block_sum(acc, sh);
    if (threadIdx.x == 0) *out = scale == 1.0 ? r : r * scale;
}

__global__ void k_finish_sums(const double* __restrict__ part, int nparts, double scale, double* __restrict__ out) {
    __shared__ double sh[32];
    finish_sum(part + (int64_t)blockIdx.x * nparts, nparts, scale, out + blockIdx.x, sh);
}

cudaError_t launch_finish_sums(const double* partial, int nparts, int nout, double* out, cudaStream_t st, double scale) {
    note_launch(), k_finish_sums<<<nout, 256, 0, st>>>(partial, nparts, scale, out);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// pack: arbitrary-strided (t,x,y,z,mu,a,b) complex128/complex64 -> device
// layout, optionally reunitarised.  One thread per (site, mu), grid-strided
// so that a capped grid can stream a field in beside other kernels.
// ---------------------------------------------------------------------------
struct Strides7 {
    int64_t s[7];
};

template <typename SRC>
__device__ __forceinline__ void pack_one(const SRC* __restrict__ src, const Strides7& sd, const Geom& g,
                                         void* __restrict__ dst, int dst_prec, int reun, int64_t idx) {
    const int64_t s = idx % g.V;
    const int mu = (int)(idx / g.V);
    int c[4];
    site_coords(g, s, c);
    const int64_t base = c[0] * sd.s[0] + c[1] * sd.s[1] + c[2] * sd.s[2] + c[3] * sd.s[3] + mu * sd.s[4];
    double r[3][3], im[3][3];
    // reconstruct-12 keeps the first two rows: without reunitarisation the
    // third row is not read at all (in the reference's layout its elements
    // are planes of their own, a third of the field's bytes -- a host field
    // read over NVLink-C2C moves 2/3 of its size)
    const int na = (dst_prec == PREC_R12 && !reun) ? 2 : 3;
    for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 3; ++b) {
            r[a][b] = im[a][b] = 0.0;
            if (a < na) {
                const SRC v = src[base + a * sd.s[5] + b * sd.s[6]];
                r[a][b] = (double)v.x;
                im[a][b] = (double)v.y;
            }
        }
    if (reun) fix_su3_rows(r, im);
    if (dst_prec == PREC_C128) {
        double2* o = (double2*)dst + s + g.V * mu;
        for (int a = 0; a < 3; ++a)
            for (int b = 0; b < 3; ++b) o[4 * g.V * (a + 3 * b)] = make_double2(r[a][b], im[a][b]);
    } else if (dst_prec == PREC_C64) {
        float2* o = (float2*)dst + s + g.V * mu;
        for (int a = 0; a < 3; ++a)
            for (int b = 0; b < 3; ++b) o[4 * g.V * (a + 3 * b)] = make_float2((float)r[a][b], (float)im[a][b]);
    } else {
        float4* o = (float4*)dst + s + g.V * (3 * mu);
        o[0] = make_float4((float)r[0][0], (float)im[0][0], (float)r[0][1], (float)im[0][1]);
        o[g.V] = make_float4((float)r[0][2], (float)im[0][2], (float)r[1][0], (float)im[1][0]);
        o[2 * g.V] = make_float4((float)r[1][1], (float)im[1][1], (float)r[1][2], (float)im[1][2]);
    }
}

template <typename SRC>
__global__ void k_pack(const SRC* __restrict__ src, Strides7 sd, Geom g, void* __restrict__ dst, int dst_prec, int reun,
                       int mu0) {
    for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < (4 - mu0) * g.V;
         idx += (int64_t)gridDim.x * blockDim.x)
        pack_one(src, sd, g, dst, dst_prec, reun, idx + mu0 * g.V);
}

cudaError_t launch_pack(const void* src, int src_dtype, const int64_t strides[7], const Geom& g, void* dst, int dst_prec,
                        int reunitarise, cudaStream_t st, unsigned max_blocks, int mu0) {
    Strides7 sd;
    for (int k = 0; k < 7; ++k) sd.s[k] = strides[k];
    if (mu0 < 0 || mu0 > 3) return cudaErrorInvalidValue;
    const int64_t n = (4 - mu0) * g.V;
    const int bs = 256;
    unsigned nb = (unsigned)((n + bs - 1) / bs);
    if (max_blocks && nb > max_blocks) nb = max_blocks;
    if (src_dtype == PREC_C128)
        note_launch(), k_pack<double2><<<nb, bs, 0, st>>>((const double2*)src, sd, g, dst, dst_prec, reunitarise, mu0);
    else
        note_launch(), k_pack<float2><<<nb, bs, 0, st>>>((const float2*)src, sd, g, dst, dst_prec, reunitarise, mu0);
    return cudaGetLastError();
}

// in-place FixSU3Matrix of a device field (any precision)
__global__ void k_fix_field(void* links, Geom g, int prec) {
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= 4 * g.V) return;
    const int64_t s = idx % g.V;
    const int mu = (int)(idx / g.V);
    double r[3][3], im[3][3];
    if (prec == PREC_C128) {
        double2* o = (double2*)links + s + g.V * mu;
        for (int a = 0; a < 3; ++a)
            for (int b = 0; b < 3; ++b) {
                const double2 v = o[4 * g.V * (a + 3 * b)];
                r[a][b] = v.x;
                im[a][b] = v.y;
            }
        fix_su3_rows(r, im);
        for (int a = 0; a < 3; ++a)
            for (int b = 0; b < 3; ++b) o[4 * g.V * (a + 3 * b)] = make_double2(r[a][b], im[a][b]);
    } else if (prec == PREC_C64) {
        float2* o = (float2*)links + s + g.V * mu;
        for (int a = 0; a < 3; ++a)
            for (int b = 0; b < 3; ++b) {
                const float2 v = o[4 * g.V * (a + 3 * b)];
                r[a][b] = v.x;
                im[a][b] = v.y;
            }
        fix_su3_rows(r, im);
        for (int a = 0; a < 3; ++a)
            for (int b = 0; b < 3; ++b) o[4 * g.V * (a + 3 * b)] = make_float2((float)r[a][b], (float)im[a][b]);
    } else {
        float4* o = (float4*)links + s + g.V * (3 * mu);
        const float4 q0 = o[0], q1 = o[g.V], q2 = o[2 * g.V];
        r[0][0] = q0.x; im[0][0] = q0.y; r[0][1] = q0.z; im[0][1] = q0.w;
        r[0][2] = q1.x; im[0][2] = q1.y; r[1][0] = q1.z; im[1][0] = q1.w;
        r[1][1] = q2.x; im[1][1] = q2.y; r[1][2] = q2.z; im[1][2] = q2.w;
        fix_su3_rows(r, im);
        o[0] = make_float4((float)r[0][0], (float)im[0][0], (float)r[0][1], (float)im[0][1]);
        o[g.V] = make_float4((float)r[0][2], (float)im[0][2], (float)r[1][0], (float)im[1][0]);
        o[2 * g.V] = make_float4((float)r[1][1], (float)im[1][1], (float)r[1][2], (float)im[1][2]);
    }
}

cudaError_t launch_fix_field(void* links, const Geom& g, int prec, cudaStream_t st) {
    const int64_t n = 4 * g.V;
    note_launch(), k_fix_field<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(links, g, prec);
    return cudaGetLastError();
}

// unpack: device layout -> reference layout (complex128 or complex64)
template <class L, typename T, typename D2>
__global__ void k_unpack(L U, Geom g, D2* __restrict__ dst) {
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= 4 * g.V) return;
    const int64_t s = idx % g.V;
    const int mu = (int)(idx / g.V);
    const M3<T> m = U.load(s, mu);
    D2* o = dst + s + g.V * mu;
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            D2 v;
            v.x = m.r[3 * a + b];
            v.y = m.i[3 * a + b];
            o[4 * g.V * (a + 3 * b)] = v;
        }
}

cudaError_t launch_unpack(const FieldRef& U, void* dst, int dst_dtype, cudaStream_t st) {
    const int64_t n = 4 * U.g.V;
    const unsigned nb = (unsigned)((n + 255) / 256);
    FLUE_DISPATCH_LINKS(U, {
        if (dst_dtype == PREC_C128)
            note_launch(), k_unpack<decltype(L), T, double2><<<nb, 256, 0, st>>>(L, U.g, (double2*)dst);
        else
            note_launch(), k_unpack<decltype(L), T, float2><<<nb, 256, 0, st>>>(L, U.g, (float2*)dst);
    });
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// batched MultiplyMatMat (src/SU3MatrixOps.f90:19-37) / MultiplyMatdagMatdag
// (:39-58; its code forms conj(sum_k L(k,i) R(j,k)) = (L^+ R^+)(i,j), although
// its comment reads (L R)^+): n matrices of 9 complex, Fortran order (a + 3b).
// ---------------------------------------------------------------------------
template <typename T>
__global__ void k_matmul_batch(const typename V2<T>::type* __restrict__ l, const typename V2<T>::type* __restrict__ r,
                               typename V2<T>::type* __restrict__ o, int64_t n, int dagger) {
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    M3<T> A, B;
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            const auto x = l[9 * j + a + 3 * b];
            const auto y = r[9 * j + a + 3 * b];
            A.r[3 * a + b] = x.x;
            A.i[3 * a + b] = x.y;
            B.r[3 * a + b] = y.x;
            B.i[3 * a + b] = y.y;
        }
    // MultiplyMatdagMatdag computes L^+ R^+ (src/SU3MatrixOps.f90:47-57)
    const M3<T> C = dagger ? mm<true, true>(A, B) : mul(A, B);
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            typename V2<T>::type v;
            v.x = C.r[3 * a + b];
            v.y = C.i[3 * a + b];
            o[9 * j + a + 3 * b] = v;
        }
}

cudaError_t launch_matmul_batch(const void* l, const void* r, void* o, int64_t n, int dtype, int dagger, cudaStream_t st) {
    const unsigned nb = (unsigned)((n + 127) / 128);
    if (dtype == PREC_C128)
        note_launch(), k_matmul_batch<double><<<nb, 128, 0, st>>>((const double2*)l, (const double2*)r, (double2*)o, n, dagger);
    else
        note_launch(), k_matmul_batch<float><<<nb, 128, 0, st>>>((const float2*)l, (const float2*)r, (float2*)o, n, dagger);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// plaquette over planes mu in [mu0,mu1], nu in (mu,nu1] (0-based):
// Re Tr[(U_mu(x) U_nu(x+mu)) (U_mu(x+nu) U_nu(x))^+]  (src/wloops.F90:960-1005)
// ---------------------------------------------------------------------------
constexpr int RED_BS = 256;

int plaquette_blocks(const Geom& g) { return grid_for(g.V, RED_BS, red_cap()); }
int plaquette_slots(const Geom& g) { return grid_for(g.V, RED_BS, kMaxRedBlocks); }

// FP32: at most 128 registers (two 256-thread blocks per SM): measured on
// GB300 at 32^3x64, all planes, c64 0.53 -> 0.36 ms per call against the
// unbounded unrolled kernel's 0.45 ms; then with 32-bit offsets (FullLinks32)
// and site coordinates 48^3x96 1.60 -> 1.26 ms (HBM floor 0.83 ms; bound by
// the latency of its L2 reads).  FP64 keeps its registers (bound by the FP64
// pipe, it spills under the cap)
#ifndef FLUE_PLAQ_MINB
#define FLUE_PLAQ_MINB 2
#endif
template <class L, typename T>
__device__ __forceinline__ void plaquette_block(const L& U, const Geom& g, int mu0, int mu1, int nu1,
                                                double* __restrict__ part, double* sh) {
    double acc = 0.0;
    for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < g.V; s += (int64_t)gridDim.x * blockDim.x) {
        int c[4];
        site_coords(g, s, c);
        int64_t sp[4];  // s + mu for every direction (compile-time indices only)
#pragma unroll
        for (int d = 0; d < 4; ++d) sp[d] = s + (c[d] + 1 == g.n[d] ? -(int64_t)(g.n[d] - 1) * g.st[d] : g.st[d]);
        // the six planes unrolled; the requested range selects them at run time
#pragma unroll
        for (int mu = 0; mu < 3; ++mu) {
            if (mu < mu0 || mu > mu1) continue;
            const M3<T> umu = U.load(s, mu);
#pragma unroll
            for (int nu = mu + 1; nu < 4; ++nu) {
                if (nu > nu1) continue;
                // MultiplyMatdagMatdag(Umu_xnu, Unu_x) = Umu_xnu^+ Unu_x^+ = (Unu_x Umu_xnu)^+
                const M3<T> a = mul(umu, U.load(sp[mu], nu));
                const M3<T> b = mul(U.load(s, nu), U.load(sp[nu], mu));
                acc += (double)retr_mm<false, true>(a, b);
            }
        }
    }
    const double r = block_sum(acc, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = r;
}

template <class L, typename T>
__global__ void __launch_bounds__(RED_BS, sizeof(T) == 4 ? FLUE_PLAQ_MINB : 1)
    k_plaquette(L U, Geom g, int mu0, int mu1, int nu1, double* __restrict__ part) {
    __shared__ double sh[32];
    plaquette_block<L, T>(U, g, mu0, mu1, nu1, part, sh);
}

// After the fixed-point kernel below: sums its nfix block partials when the gate
// is open; else computes them in FP64, in the grid of the ungated kernel, and the
// last block to finish sums them.
__global__ void __launch_bounds__(RED_BS) k_plaquette_finish(FullLinks<double> U, Geom g, int mu0, int mu1, int nu1,
                                                             double* part, int nfix, FixGate gt, double* out) {
    __shared__ double sh[32];
    const bool open = gt.open();
    if (open) {
        if (blockIdx.x) return;
    } else {
        plaquette_block<FullLinks<double>, double>(U, g, mu0, mu1, nu1, part, sh);
        if (!gate_last_block(gt, gridDim.x)) return;
    }
    finish_sum(part, open ? nfix : (int)gridDim.x, 1.0, out, sh);
}

// Plaquettes of a complex128 field in fixed point (all planes at 32^3x64 4.7 ->
// 1.6 ms, half integer multiply-adds, half the conversion of 16 links a site),
// a thread a site: the site's
// own links are converted once into shared memory (each of them is in up to
// three planes), the neighbours' as they are read.  They are counted in the
// gate on the way: the partial sums stand when the gate turns out open, else
// k_plaquette_finish replaces them.  Real traces are of order 1 however close the
// links are to 1, so the gate only asks that they are unitary; the first warp that
// meets one that is not ends the work of all (32^3x64, no link unitary: 6.52 ms
// when every block went on, 5.03 so, 5.02 without fixed point).
constexpr int PLF_BS = 128;
constexpr int PLF_SMEM = 36 * PLF_BS * (int)sizeof(int4);  // 73,728: three blocks an SM
static int plaqfix_blocks(const Geom& g) { return grid_for(g.V, PLF_BS, std::min(3 * device_sms(), kMaxRedBlocks)); }

__device__ __forceinline__ M3F smem_link(const int4* p, int mu) {
    M3F m;
#pragma unroll
    for (int e = 0; e < 9; ++e) {
        const int4 v = p[(9 * mu + e) * PLF_BS];
        m.r[e] = {v.x, v.y};
        m.i[e] = {v.z, v.w};
    }
    return m;
}

__global__ void __launch_bounds__(PLF_BS, 3)
    k_plaquette_fix(FullLinks<double> U, Geom g, int mu0, int mu1, int nu1, double* __restrict__ part, FixGate gt) {
    extern __shared__ int4 own_sm[];
    __shared__ double sh[32];
    int4* own = own_sm + threadIdx.x;
    double acc = 0.0;
    int turn = 0;
    for (int64_t s0 = (int64_t)blockIdx.x * PLF_BS; s0 < g.V; s0 += (int64_t)gridDim.x * PLF_BS) {
        const int64_t s = s0 + threadIdx.x;
        const bool live = s < g.V;
        int c[4];
        site_coords(g, live ? s : 0, c);
        // (every eighth time: 1% of the call when looked at each time)
        u32 lost = 0;
        if ((turn++ & 7) == 0) lost = *(volatile const u32*)gt.p;
#pragma unroll 1
        for (int mu = mu0; mu <= nu1; ++mu) {
            u32 st = 0;
            if (live) {
                const M3<double> u = U.load(s, mu);
                const M3F f = fx_of(u);
                st = link_state(u, f);
#pragma unroll
                for (int e = 0; e < 9; ++e)
                    own[(9 * mu + e) * PLF_BS] = make_int4(f.r[e].h, f.r[e].l, f.i[e].h, f.i[e].l);
            }
            lost |= gate_count(gt, st).x;
        }
        if (__any_sync(0xffffffffu, lost != 0)) break;
        if (!live) continue;
        int64_t fw[4];
#pragma unroll
        for (int d = 0; d < 4; ++d) fw[d] = c[d] + 1 == g.n[d] ? -(int64_t)(g.n[d] - 1) * g.st[d] : g.st[d];
        i64 t = 0;
#pragma unroll 1
        for (int mu = mu0; mu <= mu1; ++mu) {
            const int64_t sm = s + (mu == 0 ? fw[0] : mu == 1 ? fw[1] : mu == 2 ? fw[2] : fw[3]);
#pragma unroll 1
            for (int nu = mu + 1; nu <= nu1; ++nu) {
                const int64_t sn = s + (nu == 1 ? fw[1] : nu == 2 ? fw[2] : fw[3]);
                const M3F a = fx_mm<false, false>(smem_link(own, mu), fx_of(U.load(sm, nu)));
                const M3F b = fx_mm<false, false>(smem_link(own, nu), fx_of(U.load(sn, mu)));
                t += fx_retr<false, true>(a, b);  // six planes: below 2^63
            }
        }
        acc += (double)t * 0x1p-58;
    }
    const double r = block_sum(acc, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = r;
}

size_t plaquette_ws_bytes(const Geom& g, int prec) {
    const size_t red = ((size_t)plaquette_slots(g) * 8 + 255) & ~(size_t)255;
    return prec == PREC_C128 ? std::max(red, (size_t)kMaxRedBlocks * 8) + 256 : red;
}
size_t plaquette_ws_min_bytes(const Geom& g) { return ((size_t)plaquette_slots(g) * 8 + 255) & ~(size_t)255; }

// the gate at the end of a reduction's workspace; need: links away from 1
static FixGate red_gate(void* ws, size_t bytes, uint64_t need, cudaStream_t st, cudaError_t* e) {
    FixGate gt;
    gt.p = (u32*)((char*)ws + bytes - 256);
    gt.need = (u32)need;
    *e = cudaMemsetAsync(gt.p, 0, GATE_WORDS * sizeof(u32), st);
    return gt;
}

cudaError_t launch_plaquette(const FieldRef& U, int mu0, int mu1, int nu1, double* part, size_t ws_bytes, double* out,
                             cudaStream_t st) {
    const size_t fws = plaquette_ws_bytes(U.g, U.prec);
    if (U.prec == PREC_C128 && ws_bytes >= fws && mu0 <= mu1 && mu0 < nu1) {
        const FullLinks<double> L{(const double2*)U.links, U.g.V};
        cudaError_t e;
        const FixGate gt = red_gate(part, fws, 0, st, &e);
        if (e != cudaSuccess) return e;
        const int nb = plaqfix_blocks(U.g);
        // (the attribute is per function and per device; setting it again is harmless)
        e = cudaFuncSetAttribute(k_plaquette_fix, cudaFuncAttributeMaxDynamicSharedMemorySize, PLF_SMEM);
        if (e != cudaSuccess) return e;
        note_launch(), k_plaquette_fix<<<nb, PLF_BS, PLF_SMEM, st>>>(L, U.g, mu0, mu1, nu1, part, gt);
        note_launch(), k_plaquette_finish<<<plaquette_blocks(U.g), RED_BS, 0, st>>>(L, U.g, mu0, mu1, nu1, part, nb, gt,
                                                                                   out);
        return cudaGetLastError();
    }
    const int nb = plaquette_blocks(U.g);
    if (U.prec == PREC_C64 && FullLinks32::fits(U.g.V)) {
        const FullLinks32 L{(const char*)U.links, (uint32_t)U.g.V};
        note_launch(), k_plaquette<FullLinks32, float><<<nb, RED_BS, 0, st>>>(L, U.g, mu0, mu1, nu1, part);
    } else {
        FLUE_DISPATCH_LINKS(U, note_launch(), k_plaquette<decltype(L), T><<<nb, RED_BS, 0, st>>>(L, U.g, mu0, mu1, nu1, part));
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    return launch_finish_sums(part, nb, 1, out, st);
}

// ---------------------------------------------------------------------------
// Polyakov loop: ordered product of U_t over t = 1..NT at every spatial site
// (src/wloops.F90:1043-1066); out2 = [sum Re Tr, sum Im Tr].
// ---------------------------------------------------------------------------
// FP32: one warp per spatial site: lane l multiplies the links of its time
// range [l k, (l+1) k), k = ceil(NT/32) (the lanes read consecutive links,
// so the loads coalesce), then five shuffle levels multiply neighbouring
// partial products in order, P[0,2w) = P[0,w) P[w,2w); lanes past NT hold
// the identity.  Same ordered product, associated as a tree.  FP64: one
// thread per spatial site walks its column (the tree issues ~3x the FP64
// products per site and the FP64 pipe is the bound: 32^3x64 0.53 ms serial
// against 1.11 ms as a tree; FP32 0.17 -> 0.13 ms per call as a tree).
static int polyakov_blocks_serial(const Geom& g) { return grid_for(g.V / g.n[0], RED_BS, red_cap()); }
int polyakov_blocks(const Geom& g) { return grid_for(g.V / g.n[0], RED_BS / 32, red_cap()); }
int polyakov_slots(const Geom& g) { return grid_for(g.V / g.n[0], RED_BS / 32, kMaxRedBlocks); }  // the larger grid

template <typename T>
__device__ __forceinline__ M3<T> shfl_down_m3(const M3<T>& m, int off) {
    M3<T> o;
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        o.r[k] = __shfl_down_sync(0xffffffffu, m.r[k], off);
        o.i[k] = __shfl_down_sync(0xffffffffu, m.i[k], off);
    }
    return o;
}

template <class L, typename T>
__device__ __forceinline__ void polyakov_block(const L& U, const Geom& g, double* __restrict__ part, double* sh) {
    double accr = 0.0, acci = 0.0;
    const int nt = g.n[0];
    const int64_t V3 = g.V / nt;
    const int lane = threadIdx.x & 31;
    const int k = (nt + 31) / 32;
    const int t0 = lane * k, t1 = min(nt, t0 + k);
    if (sizeof(T) == 8) {
        for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < V3; r += (int64_t)gridDim.x * blockDim.x) {
            const int64_t s0 = r * nt;
            M3<T> p = U.load(s0, 0);
            for (int t = 1; t < nt; ++t) p = mul(p, U.load(s0 + t, 0));
            accr += (double)retr(p);
            acci += (double)(p.i[0] + p.i[4] + p.i[8]);
        }
    } else {
        const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
        for (int64_t r = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); r < V3; r += warps) {
            const int64_t s0 = r * nt;
            M3<T> p = m_ident<T>();
            if (t0 < nt) {
                p = U.load(s0 + t0, 0);
                for (int t = t0 + 1; t < t1; ++t) p = mul(p, U.load(s0 + t, 0));
            }
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const M3<T> q = shfl_down_m3(p, off);
                if ((lane & (2 * off - 1)) == 0) p = mul(p, q);
            }
            if (lane == 0) {
                accr += (double)retr(p);
                acci += (double)(p.i[0] + p.i[4] + p.i[8]);
            }
        }
    }
    double a = block_sum(accr, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = a;
    a = block_sum(acci, sh);
    if (threadIdx.x == 0) part[gridDim.x + blockIdx.x] = a;
}

template <class L, typename T>
__global__ void __launch_bounds__(RED_BS) k_polyakov(L U, Geom g, double* __restrict__ part) {
    __shared__ double sh[32];
    polyakov_block<L, T>(U, g, part, sh);
}

// as k_plaquette_finish
__global__ void __launch_bounds__(RED_BS) k_polyakov_finish(FullLinks<double> U, Geom g, double* part, int nfix,
                                                            FixGate gt, double* out2) {
    __shared__ double sh[32];
    const bool open = gt.open();
    if (open) {
        if (blockIdx.x) return;
    } else {
        polyakov_block<FullLinks<double>, double>(U, g, part, sh);
        if (!gate_last_block(gt, gridDim.x)) return;
    }
    const int n = open ? nfix : (int)gridDim.x;
    finish_sum(part, n, 1.0, out2, sh);
    finish_sum(part + n, n, 1.0, out2 + 1, sh);
}

// Polyakov loops of a complex128 field in fixed point: nl lanes a column (a
// power of two with at least eight links a lane, as far as NT has them), each
// the ordered product of its run of links, then log2(nl) shuffle levels: few
// enough for the levels' idle lanes (a lane a link made 6 of 7 products idle
// work), enough columns in flight for the chip.  32^3x64 0.53 -> 0.24 ms a call.
// The links are counted in the gate; k_polyakov_finish replaces the sums when it
// turns out shut.  The imaginary part of the trace of a cold column is small, so a
// quarter of the links has to be away from 1, and the first warp that finds none
// among 32 ends the work of all, as does a link that is not unitary: a cold
// 32^3x64 took 1.13 ms when every block went on, 0.56 so, 0.54 without fixed point.
constexpr int POLF_BS = 128;
static int polyfix_lanes(int nt) {
    int nl = 1;
    while (nl < 32 && nt >= 16 * nl) nl *= 2;
    return nl;
}
static int polyfix_blocks(const Geom& g) {
    return grid_for(g.V / g.n[0], POLF_BS / polyfix_lanes(g.n[0]), kMaxRedBlocks);
}

__global__ void __launch_bounds__(POLF_BS) k_polyakov_fix(FullLinks<double> U, Geom g, int nl,
                                                          double* __restrict__ part, FixGate gt) {
    __shared__ double sh[32];
    const int nt = g.n[0], lane = threadIdx.x % nl, k = (nt + nl - 1) / nl;
    const int t0 = min(nt, lane * k), t1 = min(nt, t0 + k);
    const int64_t V3 = g.V / nt;
    const int per = POLF_BS / nl;
    double accr = 0.0, acci = 0.0;
    for (int64_t r0 = (int64_t)blockIdx.x * per; r0 < V3; r0 += (int64_t)gridDim.x * per) {
        const int64_t r = r0 + threadIdx.x / nl;
        const bool live = r < V3;
        M3F p;
#pragma unroll
        for (int e = 0; e < 9; ++e) p.r[e] = {e % 4 == 0 ? 1 << 29 : 0, 0}, p.i[e] = {0, 0};
        u32 lost = *(volatile const u32*)gt.p;
        const bool whole = __all_sync(0xffffffffu, live && t0 < nt);
#pragma unroll 1
        for (int j = 0; j < k; ++j) {  // the same count for every lane: gate_count is warp-wide
            const int t = t0 + j;
            u32 st = 0;
            if (live && t < t1) {
                const M3<double> u = U.load(r * nt + t, 0);
                const M3F f = fx_of(u);
                st = link_state(u, f);
                p = j ? fx_mm<false, false>(p, f) : f;
            }
            const uint2 n = gate_count(gt, st);
            if (j == 0 && whole && !n.y) {  // 32 links, none away from 1
                lost = 1;
                if ((threadIdx.x & 31) == 0) atomicAdd(gt.p, 1u);
            }
            lost |= n.x;
            if (__any_sync(0xffffffffu, lost != 0)) break;
        }
        if (__any_sync(0xffffffffu, lost != 0)) break;
#pragma unroll 1
        for (int off = 1; off < nl; off <<= 1) {
            const M3F q = fx_shfl_down(p, off);
            if ((lane & (2 * off - 1)) == 0) p = fx_mm<false, false>(p, q);
        }
        if (live && lane == 0) {
            accr += (double)(fx_int60(p.r[0]) + fx_int60(p.r[4]) + fx_int60(p.r[8])) * 0x1p-60;
            acci += (double)(fx_int60(p.i[0]) + fx_int60(p.i[4]) + fx_int60(p.i[8])) * 0x1p-60;
        }
    }
    double a = block_sum(accr, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = a;
    a = block_sum(acci, sh);
    if (threadIdx.x == 0) part[gridDim.x + blockIdx.x] = a;
}

size_t polyakov_ws_min_bytes(const Geom& g) { return ((size_t)polyakov_slots(g) * 16 + 255) & ~(size_t)255; }
size_t polyakov_ws_bytes(const Geom& g, int prec) {
    const size_t red = polyakov_ws_min_bytes(g);
    return prec == PREC_C128 ? std::max(red, (size_t)kMaxRedBlocks * 16) + 256 : red;
}

cudaError_t launch_polyakov(const FieldRef& U, double* part, size_t ws_bytes, double* out2, cudaStream_t st) {
    const size_t fws = polyakov_ws_bytes(U.g, U.prec);
    // (products of up to 4096 links keep their norms within the fixed-point bounds)
    if (U.prec == PREC_C128 && ws_bytes >= fws && U.g.n[0] <= 4096) {
        const FullLinks<double> L{(const double2*)U.links, U.g.V};
        cudaError_t e;
        const FixGate gt = red_gate(part, fws, ((uint64_t)U.g.V + 3) / 4, st, &e);
        if (e != cudaSuccess) return e;
        const int nbf = polyfix_blocks(U.g);
        note_launch(), k_polyakov_fix<<<nbf, POLF_BS, 0, st>>>(L, U.g, polyfix_lanes(U.g.n[0]), part, gt);
        note_launch(), k_polyakov_finish<<<polyakov_blocks_serial(U.g), RED_BS, 0, st>>>(L, U.g, part, nbf, gt, out2);
        return cudaGetLastError();
    }
    const int nb = U.prec == PREC_C128 ? polyakov_blocks_serial(U.g) : polyakov_blocks(U.g);
    FLUE_DISPATCH_LINKS(U, note_launch(), k_polyakov<decltype(L), T><<<nb, RED_BS, 0, st>>>(L, U.g, part));
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    return launch_finish_sums(part, nb, 2, out2, st);
}

// ---------------------------------------------------------------------------
// nMu x nNu Wilson loop at every site (tau < 0) or on the slice t = tau
// (src/wloops.F90:599-675 and :711-789).
// ---------------------------------------------------------------------------
int wloop_blocks(const Geom& g) { return grid_for(g.V, RED_BS, red_cap()); }
int wloop_slots(const Geom& g) { return grid_for(g.V, RED_BS, kMaxRedBlocks); }

// coordinate, extent and stride of direction d (runtime) without
// runtime-indexed arrays (they would go to local memory)
__device__ __forceinline__ void dir_of(const Geom& g, const int c[4], int d, int& cd, int& nd, int64_t& sd) {
#pragma unroll
    for (int k = 0; k < 4; ++k)
        if (k == d) cd = c[k], nd = g.n[k], sd = g.st[k];
}

// product U_d(x) U_d(x+d) ... of n links starting at site s, whose
// coordinate along d is cd (extent nd, stride sd)
template <class L, typename T>
__device__ __forceinline__ M3<T> line_walk(const L& U, int64_t s, int d, int cd, int nd, int64_t sd, int n) {
    M3<T> p = U.load(s, d);
    for (int k = 1; k < n; ++k) {
        s += (cd + 1 == nd) ? -(int64_t)(nd - 1) * sd : sd;
        cd = (cd + 1 == nd) ? 0 : cd + 1;
        p = mul(p, U.load(s, d));
    }
    return p;
}

template <class L, typename T>
__global__ void __launch_bounds__(RED_BS)
    k_wloop(L U, Geom g, int tau, int mu, int nu, int nmu, int nnu, double* __restrict__ part) {
    __shared__ double sh[32];
    double acc = 0.0;
    const int64_t nsites = tau < 0 ? g.V : g.V / g.n[0];
    for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < nsites; j += (int64_t)gridDim.x * blockDim.x) {
        const int64_t s = tau < 0 ? j : (int64_t)tau + j * g.n[0];
        int c[4];
        site_coords(g, s, c);
        int cm = 0, nm = 1, cn = 0, nn = 1;
        int64_t sm = 1, sn = 1;
        dir_of(g, c, mu, cm, nm, sm);
        dir_of(g, c, nu, cn, nn, sn);
        const int cm2 = (int)(((int64_t)cm + nmu) % nm), cn2 = (int)(((int64_t)cn + nnu) % nn);
        const int64_t smu = s + (int64_t)(cm2 - cm) * sm, snu = s + (int64_t)(cn2 - cn) * sn;
        const M3<T> a = line_walk<L, T>(U, s, mu, cm, nm, sm, nmu);
        const M3<T> b = line_walk<L, T>(U, smu, nu, cn, nn, sn, nnu);   // x + nMu mu: same nu coordinate
        const M3<T> cc = line_walk<L, T>(U, snu, mu, cm, nm, sm, nmu);  // x + nNu nu: same mu coordinate
        const M3<T> d = line_walk<L, T>(U, s, nu, cn, nn, sn, nnu);
        // Re Tr[(A B) (C^+ D^+)] with C^+ D^+ = (D C)^+  (MultiplyMatdagMatdag, :669)
        const M3<T> ab = mul(a, b);
        const M3<T> dc = mul(d, cc);
        acc += (double)retr_mm<false, true>(ab, dc);
    }
    const double r = block_sum(acc, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = r;
}

cudaError_t launch_wloop(const FieldRef& U, int tau, int mu, int nu, int nmu, int nnu, double* part, double* out,
                         cudaStream_t st) {
    const int nb = wloop_blocks(U.g);
    FLUE_DISPATCH_LINKS(U, note_launch(), k_wloop<decltype(L), T><<<nb, RED_BS, 0, st>>>(L, U.g, tau, mu, nu, nmu, nnu, part));
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const double norm = tau < 0 ? (double)U.g.V : (double)(U.g.V / U.g.n[0]);
    return launch_finish_sums(part, nb, 1, out, st, 1.0 / norm);
}

// ---------------------------------------------------------------------------
// W_munu table: wmunu(mu, nu, R, T) for every R <= rmax, T <= tmax at once
// (the reference evaluates src/wloops.F90:679-791 once per (R, T), walking
// every line anew).  k_wt_lines stores per site the mu-lines L_R = U_mu(x)
// ... U_mu(x+(R-1)mu) and the nu-lines L_T, built incrementally; k_wt_loops
// forms each loop from four stored lines, Re Tr[(A B)(D C)^+] with A = L_R(x),
// B = L_T(x+R mu), C = L_R(x+T nu), D = L_T(x) -- the formula of k_wloop --
// with the rmax * tmax tasks of one site block in adjacent blocks (the
// neighbour lines they read stay in L2).
// ---------------------------------------------------------------------------
constexpr int WT_BS = 128;

template <class L, typename T>
__device__ __forceinline__ void wt_lines_site(int64_t s, const L& U, const Geom& g, int mu, int nu, int rmax, int tmax,
                                              const MatAoS<T>& lines) {
    int c[4];
    site_coords(g, s, c);
    for (int pass = 0; pass < 2; ++pass) {
        const int d = pass ? nu : mu, n = pass ? tmax : rmax, k0 = pass ? rmax : 0;
        int cd = 0, nd = 1;
        int64_t sd = 1;
        dir_of(g, c, d, cd, nd, sd);
        int64_t sw = s;
        M3<T> p = U.load(sw, d);
        lines.store(s, k0, p);
        for (int k = 1; k < n; ++k) {
            sw += (cd + 1 == nd) ? -(int64_t)(nd - 1) * sd : sd;
            cd = (cd + 1 == nd) ? 0 : cd + 1;
            p = mul(p, U.load(sw, d));
            lines.store(s, k0 + k, p);
        }
    }
}

template <class L, typename T>
__global__ void k_wt_lines(L U, Geom g, int mu, int nu, int rmax, int tmax, MatAoS<T> lines) {
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s < g.V) wt_lines_site<L, T>(s, U, g, mu, nu, rmax, tmax, lines);
}

// block blk of nsb site blocks (of the block's size) x rmax tmax tasks
template <typename T>
__device__ __forceinline__ void wt_loop_block(unsigned blk, int nsb, const Geom& g, int mu, int nu, int rmax, int tmax,
                                              const MatAoS<T>& lines, double* __restrict__ part, double* sh) {
    const int nrt = rmax * tmax;
    const int rt = blk % nrt;
    const int sb = blk / nrt;
    const int R = rt / tmax + 1, Tl = rt % tmax + 1;
    const int64_t s = (int64_t)sb * blockDim.x + threadIdx.x;
    double acc = 0.0;
    if (s < g.V) {
        int c[4];
        site_coords(g, s, c);
        int cm = 0, nm = 1, cn = 0, nn = 1;
        int64_t sm = 1, sn = 1;
        dir_of(g, c, mu, cm, nm, sm);
        dir_of(g, c, nu, cn, nn, sn);
        const int64_t sR = s + (int64_t)((cm + R) % nm - cm) * sm;
        const int64_t sT = s + (int64_t)((cn + Tl) % nn - cn) * sn;
        const M3<T> ab = mul(lines.load(s, R - 1), lines.load(sR, rmax + Tl - 1));
        const M3<T> dc = mul(lines.load(s, rmax + Tl - 1), lines.load(sT, R - 1));
        acc = (double)retr_mm<false, true>(ab, dc);
    }
    const double r = block_sum(acc, sh);
    if (threadIdx.x == 0) part[(int64_t)rt * nsb + sb] = r;
}

template <typename T>
__global__ void __launch_bounds__(WT_BS) k_wt_loops(Geom g, int mu, int nu, int rmax, int tmax, MatAoS<T> lines,
                                                    double* __restrict__ part) {
    __shared__ double sh[32];
    wt_loop_block<T>(blockIdx.x, gridDim.x / (rmax * tmax), g, mu, nu, rmax, tmax, lines, part, sh);
}

// the FP64 kernels of a complex128 field whose gate is shut, their grids capped
__global__ void __launch_bounds__(WT_BS) k_wt_lines_gated(FullLinks<double> U, Geom g, int mu, int nu, int rmax,
                                                          int tmax, MatAoS<double> lines, FixGate gt) {
    if (gate_shut(gt)) return;
    for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < g.V; s += (int64_t)gridDim.x * blockDim.x)
        wt_lines_site<FullLinks<double>, double>(s, U, g, mu, nu, rmax, tmax, lines);
}
__global__ void __launch_bounds__(WT_BS) k_wt_loops_gated(Geom g, int mu, int nu, int rmax, int tmax, int nsb,
                                                          MatAoS<double> lines, double* __restrict__ part, FixGate gt) {
    __shared__ double sh[32];
    if (gate_shut(gt)) return;
    for (unsigned b = blockIdx.x; b < (unsigned)(nsb * rmax * tmax); b += gridDim.x)
        wt_loop_block<double>(b, nsb, g, mu, nu, rmax, tmax, lines, part, sh);
}

// The lines in fixed point, a thread a (site, direction); real traces, so the gate
// only asks for unitary links (k_plaquette_fix)
__global__ void __launch_bounds__(WT_BS) k_wt_lines_fix(FullLinks<double> U, Geom g, int mu, int nu, int rmax, int tmax,
                                                        MatFix lines, FixGate gt) {
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int d = blockIdx.y ? nu : mu, n = blockIdx.y ? tmax : rmax, k0 = blockIdx.y ? rmax : 0;
    u32 st = 0;
    if (gate_lost(gt)) return;
    if (s < g.V) {
        int c[4];
        site_coords(g, s, c);
        int cd = 0, nd = 1;
        int64_t sd = 1;
        dir_of(g, c, d, cd, nd, sd);
        int64_t sw = s;
        const M3<double> u = U.load(sw, d);
        M3F p = fx_of(u);
        st = link_state(u, p);
        lines.store(s, k0, p);
#pragma unroll 1
        for (int k = 1; k < n; ++k) {
            sw += (cd + 1 == nd) ? -(int64_t)(nd - 1) * sd : sd;
            cd = (cd + 1 == nd) ? 0 : cd + 1;
            p = fx_mm<false, false>(p, fx_of(U.load(sw, d)));
            lines.store(s, k0 + k, p);
        }
    }
    gate_count(gt, st);
}

// The loops in fixed point, three warps (columns) for 32 sites.  A block has
// one R and the tmax loops of its sites: column b of A B and of D C and their
// part of the trace, two matrix-vector products a thread and loop.  32^3x64, 8 x
// 8 table: FP64 58.8 ms; fixed point 22.6 ms with a barrier a loop, and with one
// barrier 16.7 ms (128 sites a block, 12 warps an SM), 13.7 (64 sites, 18 warps,
// 112 registers, spills), 13.4 (32 sites, 15 warps, 128 registers, 80-96 bytes of
// stack); 13.2 with the site coordinates by 32-bit divisions, 12.3 with the sums
// of a warp kept as integers (no conversion on the FP64 pipe).
constexpr int WTF_BS = 32, WTF_WARPS = 3 * WTF_BS / 32, WT_MAXT = 64;

template <typename I>
__global__ void __launch_bounds__(3 * WTF_BS, 5)
    k_wt_loops_fix(Geom g, int mu, int nu, int rmax, int tmax, MatFix lines, i64* __restrict__ part, FixGate gt) {
    __shared__ i64 sh[WT_MAXT][WTF_WARPS];  // one barrier for all the loops
    if (!gt.open()) return;
    const int R = blockIdx.x % rmax + 1, sb = blockIdx.x / rmax, nsb = gridDim.x / rmax;
    const int b = threadIdx.x / WTF_BS, w = threadIdx.x >> 5;
    const int64_t s64 = (int64_t)sb * WTF_BS + threadIdx.x % WTF_BS;
    const bool live = s64 < g.V;
    const I s = (I)(live ? s64 : 0);
    int c[4];
    site_coords(g, (int64_t)s, c);
    int cm = 0, nm = 1, cn = 0, nn = 1;
    int64_t sm = 1, sn = 1;
    dir_of(g, c, mu, cm, nm, sm);
    dir_of(g, c, nu, cn, nn, sn);
    const I sR = (I)((int64_t)s + ((cm + R) % nm - cm) * sm);
    int ct = cn;
#pragma unroll 1
    for (int T = 1; T <= tmax; ++T) {
        ct = ct + 1 == nn ? 0 : ct + 1;
        const I sT = (I)((int64_t)s + (ct - cn) * sn);
        const FxV ab = lines.mul<false>(s, R - 1, lines.col<false>(sR, rmax + T - 1, b));
        const FxV dc = lines.mul<false>(s, rmax + T - 1, lines.col<false>(sT, R - 1, b));
        const i64 r = warp_sum_fix54(live ? fx_rezdot(ab, dc) : 0);
        if ((threadIdx.x & 31) == 0) sh[T - 1][w] = r;
    }
    __syncthreads();
    if (threadIdx.x < tmax) {
        i64 sum = 0;
#pragma unroll
        for (int k = 0; k < WTF_WARPS; ++k) sum += sh[threadIdx.x][k];  // at most 3 x 2^59
        part[(int64_t)((R - 1) * tmax + threadIdx.x) * nsb + sb] = sum;
    }
}

// Means of the loops from the block sums, a block a loop: integers of unit 2^-54,
// added exactly (as FP64 sums the four times as many blocks of the fixed-point
// kernel cost a tenth of an ulp at 32^3x64), or where the gate is shut the FP64
// sums of n64 blocks as k_finish_sums takes them.
__global__ void __launch_bounds__(256) k_wt_finish(const double* __restrict__ part, int nfix, int n64, double scale,
                                                   FixGate gt, double* __restrict__ out) {
    __shared__ double sh[32];
    __shared__ i64 shl[8], shh[8];
    if (!gt.open()) {
        finish_sum(part + (int64_t)blockIdx.x * n64, n64, scale, out + blockIdx.x, sh);
        return;
    }
    const i64* p = reinterpret_cast<const i64*>(part) + (int64_t)blockIdx.x * nfix;
    i64 lo = 0, hi = 0;
#pragma unroll 8
    for (int i = threadIdx.x; i < nfix; i += 256) {
        const i64 v = __ldcg(p + i);
        lo += (u32)v;
        hi += v >> 32;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lo += __shfl_down_sync(0xffffffffu, lo, o);
        hi += __shfl_down_sync(0xffffffffu, hi, o);
    }
    if ((threadIdx.x & 31) == 0) shl[threadIdx.x >> 5] = lo, shh[threadIdx.x >> 5] = hi;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < 8; ++k) lo += shl[k], hi += shh[k];
        hi += lo >> 32;
        out[blockIdx.x] = fma((double)hi, 0x1p-22, (double)(u32)lo * 0x1p-54) * scale;
    }
}

// the stored mu- and nu-lines of every length, rounded to 256 bytes
static size_t wt_lines_bytes(const Geom& g, int prec, int rmax, int tmax, bool fix) {
    size_t b = prec == PREC_C128 ? MatAoS<double>::bytes(g.V, rmax + tmax) : MatAoS<float>::bytes(g.V, rmax + tmax);
    if (fix) b = std::max(b, MatFix::bytes(g.V, rmax + tmax));
    return (b + 255) & ~(size_t)255;
}

static size_t wt_ws_bytes(const Geom& g, int prec, int rmax, int tmax, bool fix) {
    const int bs = fix ? WTF_BS : WT_BS;
    const size_t nsb = (size_t)((g.V + bs - 1) / bs);
    const size_t lines = wt_lines_bytes(g, prec, rmax, tmax, fix);
    return lines + (((size_t)rmax * tmax * nsb * sizeof(double) + 255) & ~(size_t)255) + (fix ? 256 : 0);
}
size_t wmunu_table_ws_bytes(const Geom& g, int prec, int rmax, int tmax) {
    return wt_ws_bytes(g, prec, rmax, tmax, prec == PREC_C128);
}
size_t wmunu_table_ws_min_bytes(const Geom& g, int prec, int rmax, int tmax) {
    return wt_ws_bytes(g, prec, rmax, tmax, false);
}

cudaError_t launch_wmunu_table(const FieldRef& U, int mu, int nu, int rmax, int tmax, double* out, void* ws,
                               size_t ws_bytes, cudaStream_t st) {
    const Geom& g = U.g;
    const size_t fws = wmunu_table_ws_bytes(g, U.prec, rmax, tmax);
    const bool fix = U.prec == PREC_C128 && ws_bytes >= fws;
    const size_t lines_b = wt_lines_bytes(g, U.prec, rmax, tmax, fix);
    double* part = (double*)((char*)ws + lines_b);
    const unsigned nsb = (unsigned)((g.V + WT_BS - 1) / WT_BS);
    const unsigned nrt = (unsigned)(rmax * tmax);
    if (fix) {
        const FullLinks<double> L{(const double2*)U.links, g.V};
        cudaError_t e;
        const FixGate gt = red_gate(ws, fws, 0, st, &e);
        if (e != cudaSuccess) return e;
        const MatFix fl{(int4*)ws, g.V, rmax + tmax};
        const MatAoS<double> dl{(double2*)ws, g.V, rmax + tmax};
        const unsigned cap = 8u * (unsigned)device_sms(), nsf = (unsigned)((g.V + WTF_BS - 1) / WTF_BS);
        note_launch(), k_wt_lines_fix<<<dim3(nsb, 2), WT_BS, 0, st>>>(L, g, mu, nu, rmax, tmax, fl, gt);
        i64* ipart = reinterpret_cast<i64*>(part);
        if (MatFix::fits32(g.V, rmax + tmax))
            note_launch(), k_wt_loops_fix<u32><<<nsf * rmax, 3 * WTF_BS, 0, st>>>(g, mu, nu, rmax, tmax, fl, ipart, gt);
        else
            note_launch(), k_wt_loops_fix<int64_t><<<nsf * rmax, 3 * WTF_BS, 0, st>>>(g, mu, nu, rmax, tmax, fl, ipart, gt);
        note_launch(), k_wt_lines_gated<<<std::min(nsb, cap), WT_BS, 0, st>>>(L, g, mu, nu, rmax, tmax, dl, gt);
        note_launch(), k_wt_loops_gated<<<std::min(nsb * nrt, cap), WT_BS, 0, st>>>(g, mu, nu, rmax, tmax, (int)nsb, dl,
                                                                                   part, gt);
        note_launch(), k_wt_finish<<<nrt, 256, 0, st>>>(part, (int)nsf, (int)nsb, 1.0 / (double)g.V, gt, out);
        return cudaGetLastError();
    }
    FLUE_DISPATCH_LINKS(U, {
        MatAoS<T> ln{reinterpret_cast<decltype(MatAoS<T>::p)>(ws), g.V, rmax + tmax};
        note_launch(), k_wt_lines<decltype(L), T><<<nsb, WT_BS, 0, st>>>(L, g, mu, nu, rmax, tmax, ln);
        note_launch(), k_wt_loops<T><<<nsb * nrt, WT_BS, 0, st>>>(g, mu, nu, rmax, tmax, ln, part);
    });
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    return launch_finish_sums(part, (int)nsb, (int)nrt, out, st, 1.0 / (double)g.V);
}

// ---------------------------------------------------------------------------
// genericPath (src/wloops.F90:20-57) at every site or one site.  Output is the
// TRANSPOSE of the ordered product, in the layout (NT,NX,NY,NZ,3,3) (or one
// 3x3 Fortran-ordered matrix), complex128 for FP64 fields, complex64 else.
// ---------------------------------------------------------------------------
constexpr int MAX_PATH = 256;
struct PathArg {
    int n;
    int step[MAX_PATH];  // +-(mu+1)
};

template <class L, typename T>
__global__ void k_genericpath(L U, Geom g, PathArg path, int64_t s_single, typename V2<T>::type* __restrict__ out) {
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool single = s_single >= 0;
    if (single ? j > 0 : j >= g.V) return;
    const int64_t s0 = single ? s_single : j;
    int c[4];
    site_coords(g, s0, c);
    int64_t s = s0;
    M3<T> p = m_ident<T>();
    // one periodic step of +-1 along direction mu (runtime); the branch over
    // the four directions keeps coordinates and strides in registers
    auto move = [&](int mu, int dir) {
#pragma unroll
        for (int d = 0; d < 4; ++d)
            if (d == mu) {
                const int n = g.n[d];
                int cd = c[d] + dir;
                int64_t ds = dir * g.st[d];
                if (cd < 0) cd += n, ds += (int64_t)n * g.st[d];
                if (cd >= n) cd -= n, ds -= (int64_t)n * g.st[d];
                c[d] = cd;
                s += ds;
            }
    };
    for (int k = 0; k < path.n; ++k) {
        const int st = path.step[k];
        if (st < 0) {
            const int mu = -st - 1;
            move(mu, -1);
            p = mm<false, true>(p, U.load(s, mu));
        } else {
            const int mu = st - 1;
            p = mul(p, U.load(s, mu));
            move(mu, 1);
        }
    }
    RefOut<T> o{out, single ? 1 : g.V, 1};
    o.store(single ? 0 : s0, 0, transp(p));
}

cudaError_t launch_genericpath(const FieldRef& U, const int* path_host, int npath, const int* coord_host, void* out,
                               cudaStream_t st) {
    PathArg pa;
    pa.n = npath;
    for (int k = 0; k < npath; ++k) pa.step[k] = path_host[k];
    int64_t ss = -1;
    if (coord_host) {
        ss = (int64_t)(coord_host[0] - 1) + U.g.st[1] * (coord_host[1] - 1) + U.g.st[2] * (coord_host[2] - 1) +
             U.g.st[3] * (coord_host[3] - 1);
    }
    const unsigned nb = coord_host ? 1u : (unsigned)((U.g.V + 127) / 128);
    FLUE_DISPATCH_LINKS(U, note_launch(), k_genericpath<decltype(L), T><<<nb, 128, 0, st>>>(L, U.g, pa, ss, (typename V2<T>::type*)out));
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Landau-gauge mean link: per direction sum over sites of
// Re Tr(G(x) U_mu(x) G(x+mu)^+), G in (NT,NX,NY,NZ,3,3) layout.
// ---------------------------------------------------------------------------
int meanlink_blocks(const Geom& g) { return grid_for(g.V, RED_BS, red_cap()); }
int meanlink_slots(const Geom& g) { return grid_for(g.V, RED_BS, kMaxRedBlocks); }

template <typename T, typename G2>
__device__ __forceinline__ M3<T> load_g(const G2* __restrict__ G, int64_t V, int64_t s) {
    M3<T> m;
    if (!FLUE_INB(s >= 0 && s < V)) return m_zero<T>();
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            const G2 v = G[s + V * (a + 3 * b)];
            m.r[3 * a + b] = (T)v.x;
            m.i[3 * a + b] = (T)v.y;
        }
    return m;
}

template <class L, typename T, typename G2>
__global__ void __launch_bounds__(RED_BS) k_meanlink(L U, Geom g, const G2* __restrict__ G, double* __restrict__ part) {
    __shared__ double sh[32];
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < g.V; s += (int64_t)gridDim.x * blockDim.x) {
        int c[4];
        site_coords(g, s, c);
        const M3<T> gx = load_g<T>(G, g.V, s);
#pragma unroll
        for (int mu = 0; mu < 4; ++mu) {
            const M3<T> gp = load_g<T>(G, g.V, s + disp(g, mu, c[mu], 1));
            const M3<T> gu = mul(gx, U.load(s, mu));
            acc[mu] += (double)retr_mm<false, true>(gu, gp);
        }
    }
#pragma unroll
    for (int mu = 0; mu < 4; ++mu) {
        const double r = block_sum(acc[mu], sh);
        if (threadIdx.x == 0) part[mu * gridDim.x + blockIdx.x] = r;
    }
}

cudaError_t launch_meanlink(const FieldRef& U, const void* G, int g_dtype, double* part, double* out4, cudaStream_t st) {
    const int nb = meanlink_blocks(U.g);
    FLUE_DISPATCH_LINKS(U, {
        if (g_dtype == PREC_C128)
            note_launch(), k_meanlink<decltype(L), T, double2><<<nb, RED_BS, 0, st>>>(L, U.g, (const double2*)G, part);
        else
            note_launch(), k_meanlink<decltype(L), T, float2><<<nb, RED_BS, 0, st>>>(L, U.g, (const float2*)G, part);
    });
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    return launch_finish_sums(part, nb, 4, out4, st);
}

FLUE_OOB_READER(observables)

}  // namespace flue
