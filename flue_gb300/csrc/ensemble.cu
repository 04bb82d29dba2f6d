// ensemble.cu -- plaquette / Polyakov / B^2 of an ensemble of gauge fields of
// uneven volume in ONE persistent launch, replayed from a CUDA graph.
//
// The launch is a dataflow scheduler: a cooperative persistent grid (every
// block resident at once) takes tasks from a global counter in list order.
//   LINES(j, c): the straight lines L^1..3 of the spatial directions for
//                chunk c of time slab j (one block of sites), written into
//                ring slot j % kSlots of the workspace;
//   FWD(j, c):   the 5-loop F of the planes (3,2), (2,4), (4,3) at the sites
//                of chunk c of slab j, built from those lines (84 products
//                per plane-site), and the partial sum of -Re Tr(F F);
//   COLS(f, c):  spatial and temporal plaquettes and the Polyakov loops of a
//                run of time columns of field f.
// FWD(j, .) waits until every LINES(j, .) has finished, and LINES(j, .)
// waits until every FWD(j - kSlots, .) has released the slot.  complex128
// fields are shared out between two launches, fixed point and FP64, one after
// the other: each skips the tasks of the other's fields, and its LINES(j, .)
// wait for the last slab of the slot that it did not skip (ring_prev; a skipped
// slab says nothing of the one before it).  The list
// places LINES(j) before FWD(j - 1), so every task waits only on tasks with
// lower indices: those were taken by resident blocks and finish, so the
// schedule always progresses.  Every wait is bounded; a wait that runs out
// sets an error flag (the call then reports FLUE_ERR_TIMEOUT), and the
// other waits give up as soon as they see it.  Each task writes its own FP64
// partials; a finisher sums each field's partials in list order, so results
// do not depend on which block took which task.
//
// Per site: spatial and temporal plaquettes (src/wloops.F90:915-1017), the
// 5-loop B^2 integrand -Re Tr(F F) of the planes (3,2),(2,4),(4,3)
// (src/wloops.F90:479-544), and per column the Polyakov loop
// (src/wloops.F90:1019-1069).
//
// Output per field (6 doubles): [sum Re Tr P spatial, sum Re Tr P temporal,
// sum Re Tr Polyakov, sum Im Tr Polyakov, B^2 (already divided by V), V].
#include <stdlib.h>

#include <algorithm>
#include <mutex>
#include <vector>

#include "../../include/flue_gb300.h"
#include "flue_internal.h"
#include "loop5.cuh"
#include "loop5_fix.cuh"

namespace flue {

constexpr int NOBS = 6;

struct EnsField {
    const void* links;
    Geom g;
};

enum EnsTaskType : int { TASK_LINES = 0, TASK_FWD = 1, TASK_COLS = 2 };

struct EnsTask {
    int type;
    int a;  // LINES / FWD: slab; COLS: field
    int b;  // LINES / FWD: chunk (block-sized run of the slab's sites); COLS: first column
    int n;  // COLS: number of columns
};

// A time slab: the time slices [t0, t0 + nts) of one field, as a lattice of
// its own (time extent nts); B^2 never steps in time, so slabs are
// independent.
struct EnsSlab {
    int field, t0, nts, nchunk;
};

// ring slots of slab lines
constexpr int kSlots = 4;
// sites per slab aimed at (whole time slices): 2^17, as the device B^2, or
// FLUE_ENS_SLAB_SITES (read when an ensemble is created; small values make
// many slabs, which the tests use to exercise the ring)
static int64_t slab_sites() {
    const char* env = getenv("FLUE_ENS_SLAB_SITES");
    const long long v = env ? atoll(env) : 0;
    if (v <= 0) return (int64_t)1 << 17;
    return v > ((long long)1 << 22) ? (int64_t)1 << 22 : (int64_t)v;
}

struct EnsFlowArgs {
    const EnsField* fields;
    const EnsSlab* slabs;
    const EnsTask* tasks;
    int ntasks, nslabs;
    int* ctr;      // [0] task counter, [1] error flag, [2, 2 + nslabs) lines done, then fwd done
    double* part;  // NOBS per task
    char* ring;    // kSlots slots of slot_bytes
    size_t slot_bytes;
    PlaneArg pa;   // the B^2 planes
    int nfields;
    u32* gates;    // complex128: two words a field (FixGate); NULL otherwise
};

// complex128: whether field f takes the fixed-point kernel, and whether any
// field does not (block-wide)
__device__ __forceinline__ bool ens_open(const EnsFlowArgs& a, int f) {
    return FixGate{a.gates + 2 * f, (u32)a.fields[f].g.V}.open();
}
__device__ __forceinline__ bool ens_any(const EnsFlowArgs& a, bool open) {
    bool any = false;
    for (int f = threadIdx.x; f < a.nfields; f += blockDim.x) any = any || ens_open(a, f) == open;
    return __syncthreads_or(any);
}

// The slab whose FWD tasks have to be done before this launch writes the lines
// of slab j: the last one of j's ring slot among the fields it takes, those whose
// gate is `open` (-1: none).  Called by a whole warp; a turn looks at 32 slabs.
// (Inlined, the fixed-point kernel came out 1% slower.)
__device__ __noinline__ int ring_prev(const EnsFlowArgs& a, int j, bool open, bool mixed) {
    if (!mixed) return j < kSlots ? -1 : j - kSlots;
    for (int i0 = j - kSlots; i0 >= 0; i0 -= 32 * kSlots) {
        const int i = i0 - kSlots * (int)(threadIdx.x & 31);
        const u32 own = __ballot_sync(0xffffffffu, i >= 0 && ens_open(a, a.slabs[max(i, 0)].field) == open);
        if (own) return i0 - kSlots * (__ffs((int)own) - 1);
    }
    return -1;
}

// Counts every field's links in its gate (all four directions: a quarter of
// them has to be away from 1).  B^2 only knows the spatial links and the Polyakov
// loop the others, so either may be small while the rest of the field is rough: a
// near_patch of spatial links, or 32 time links in a row that are close to 1 but not
// all equal to it (temporal gauge), shut the gate.  Fields too long for the Polyakov
// product's bounds count as not unitary.
__global__ void __launch_bounds__(128) k_ens_gates(EnsFlowArgs a) {
    for (int f = blockIdx.y; f < a.nfields; f += gridDim.y) {
        const EnsField fl = a.fields[f];
        const FullLinks<double> U{(const double2*)fl.links, fl.g.V};
        const FixGate gt{a.gates + 2 * f, 0};
        if (fl.g.n[0] > 4096 && blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(gt.p, 1u);
        const int64_t n = 4 * fl.g.V;
        for (int64_t i0 = (int64_t)blockIdx.x * blockDim.x; i0 < n; i0 += (int64_t)gridDim.x * blockDim.x) {
            const int64_t i = i0 + threadIdx.x;
            u32 st = 0;
            if (gate_lost(gt)) break;
            const int mu = (i >= fl.g.V) + (i >= 2 * fl.g.V) + (i >= 3 * fl.g.V);
            M3<double> u = m_zero<double>();
            if (i < n) {
                const int64_t s = i - (int64_t)mu * fl.g.V;
                u = U.load(s, mu);
                st = link_state(u, fx_of(u));
                if (st == 0 && mu > 0) {
                    int c[4];
                    site_coords(fl.g, s, c);
                    for (int nu = mu + 1; nu < 4; ++nu)
                        if (near_patch(U, fl.g, c, mu, nu)) st = 1;
                }
            }
            if (__all_sync(0xffffffffu, st == 0 && mu == 0) && !__all_sync(0xffffffffu, is_one(u))) st = 1;
            gate_count(gt, st);
        }
    }
}

// Thread 0: wait until *p >= target, at most ~1.7 s; false (and the error
// flag set) when the wait runs out or another wait already failed.
__device__ __forceinline__ bool flow_wait(const int* p, int target, int* err) {
    for (int it = 0; it < (1 << 24); ++it) {
        int v;
        asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
        if (v >= target) {
            __threadfence();
            return true;
        }
        if ((it & 255) == 255 && *(volatile int*)err) return false;
        __nanosleep(100);
    }
    atomicExch(err, 1);
    return false;
}

// link accessor of a field's pointer in the precision L reads
template <class L>
struct LinksFrom;
template <>
struct LinksFrom<FullLinks<double>> {
    __device__ static FullLinks<double> make(const void* p, int64_t V) { return {(const double2*)p, V}; }
};
template <>
struct LinksFrom<FullLinks<float>> {
    __device__ static FullLinks<float> make(const void* p, int64_t V) { return {(const float2*)p, V}; }
};
template <>
struct LinksFrom<R12Links> {
    __device__ static R12Links make(const void* p, int64_t V) { return {(const float4*)p, V}; }
};

template <class L, typename T>
__device__ __forceinline__ void plaq_site(const L& U, const Geom& g, int64_t s, const int c[4], double& sp, double& tp) {
#pragma unroll
    for (int mu = 0; mu < 4; ++mu) {
        const int64_t smu = s + disp(g, mu, c[mu], 1);
        const M3<T> umu = U.load(s, mu);
#pragma unroll
        for (int nu = mu + 1; nu < 4; ++nu) {
            const int64_t snu = s + disp(g, nu, c[nu], 1);
            const M3<T> a = mul(umu, U.load(smu, nu));
            const M3<T> b = mul(U.load(s, nu), U.load(snu, mu));
            const double v = (double)retr_mm<false, true>(a, b);
            if (mu == 0)
                tp += v;
            else
                sp += v;
        }
    }
}

// FP32: registers capped for 12 resident warps per SM (the forward kernel's
// budget); FP64 keeps what it needs (bound by the FP64 pipe)
template <typename T, int BS>
struct FlowMinBlocks {
    static constexpr int value = 1;
};
template <>
struct FlowMinBlocks<float, 128> {
    static constexpr int value = 3;
};
template <class L, typename T, int BS>
__global__ void __launch_bounds__(BS, (FlowMinBlocks<T, BS>::value)) k_ens_flow(EnsFlowArgs a) {
    __shared__ double sh[32];
    __shared__ int cur, ok;
    int* const err = a.ctr + 1;
    int* const lines_done = a.ctr + 2;
    int* const fwd_done = a.ctr + 2 + a.nslabs;
    // complex128: only the fields that the fixed-point kernel left out
    if (a.gates && !ens_any(a, false)) return;
    const bool mixed = a.gates && ens_any(a, true);
    // every task is taken once: at most ntasks + 1 turns per block
    for (int guard = 0; guard <= a.ntasks; ++guard) {
        if (threadIdx.x == 0) cur = atomicAdd(a.ctr, 1);
        __syncthreads();
        const int t = cur;
        if (t >= a.ntasks) break;
        const EnsTask tk = a.tasks[t];
        const bool mine = !a.gates || !ens_open(a, tk.type == TASK_COLS ? tk.a : a.slabs[tk.a].field);
        if (!mine) {
            // the scheduler's counts still move on
            if (threadIdx.x == 0 && tk.type != TASK_COLS)
                atomicAdd((tk.type == TASK_LINES ? lines_done : fwd_done) + tk.a, 1);
        } else if (tk.type == TASK_COLS) {
            const EnsField f = a.fields[tk.a];
            const L U = LinksFrom<L>::make(f.links, f.g.V);
            const int nt = f.g.n[0];
            double sp = 0.0, tp = 0.0, pr = 0.0, pi = 0.0;
            const int nsites = tk.n * nt;
            for (int k = threadIdx.x; k < nsites; k += BS) {
                const int64_t s = (int64_t)tk.b * nt + k;
                int c[4];
                site_coords(f.g, s, c);
                plaq_site<L, T>(U, f.g, s, c, sp, tp);
            }
            for (int col = threadIdx.x; col < tk.n; col += BS) {
                const int64_t s0 = (int64_t)(tk.b + col) * nt;
                M3<T> pl = U.load(s0, 0);
                for (int tt = 1; tt < nt; ++tt) pl = mul(pl, U.load(s0 + tt, 0));
                pr += (double)retr(pl);
                pi += (double)(pl.i[0] + pl.i[4] + pl.i[8]);
            }
            const double v[4] = {sp, tp, pr, pi};
#pragma unroll
            for (int o = 0; o < 4; ++o) {
                const double r = block_sum(v[o], sh);
                if (threadIdx.x == 0) a.part[(int64_t)t * NOBS + o] = r;
            }
        } else {
            const int j = tk.a;
            const EnsSlab sl = a.slabs[j];
            const EnsField f = a.fields[sl.field];
            const Geom g = make_geom(sl.nts, f.g.n[1], f.g.n[2], f.g.n[3]);
            using VP = decltype(MatAoS<T>::p);
            const MatAoS<T> lines{reinterpret_cast<VP>(a.ring + (size_t)(j % kSlots) * a.slot_bytes), g.V,
                                  3 * a.pa.nd};
            const int64_t s = (int64_t)tk.b * BS + threadIdx.x;
            if (tk.type == TASK_LINES) {
                // the slot is free once every FWD task of its last slab is done
                if (threadIdx.x < 32) {
                    const int i = ring_prev(a, j, false, mixed);
                    if (threadIdx.x == 0) ok = i < 0 || flow_wait(fwd_done + i, a.slabs[i].nchunk, err);
                }
                __syncthreads();
                if (ok && s < g.V) {
                    const L U = LinksFrom<L>::make(f.links, f.g.V);
#pragma unroll 1
                    for (int slot = 0; slot < a.pa.nd; ++slot) line_site<L, T>(U, g, f.g, sl.t0, a.pa, lines, s, slot);
                }
                __syncthreads();
                if (threadIdx.x == 0) {
                    __threadfence();
                    atomicAdd(lines_done + j, 1);
                }
            } else {
                if (threadIdx.x == 0) ok = flow_wait(lines_done + j, sl.nchunk, err);
                __syncthreads();
                double e = 0.0;
                if (ok && s < g.V) {
                    int c[4];
                    site_coords(g, s, c);
#pragma unroll 1
                    for (int p = 0; p < a.pa.np; ++p) {
                        const M3<T> fm = ah_quarter(fwd_q<T, uint32_t>(g, a.pa, 1, lines, s, c, p));
                        e -= (double)retr_mm<false, false>(fm, fm);
                    }
                }
                const double r = block_sum(e, sh);
                if (threadIdx.x == 0) {
                    a.part[(int64_t)t * NOBS + 4] = r;
                    __threadfence();
                    atomicAdd(fwd_done + j, 1);
                }
            }
        }
        __syncthreads();
    }
}

// The same scheduler for complex128 fields in fixed point: 384 threads, three
// (columns) for each of 128 sites.  CH: sites a chunk.
constexpr int EF_BS = 128;
template <int CH>
__global__ void __launch_bounds__(3 * EF_BS) k_ens_flow_fix(EnsFlowArgs a) {
    __shared__ longlong2 sq2[2][9][EF_BS];  // in turn: one barrier a plane
    __shared__ double sh[32];
    __shared__ int cur, ok;
    int* const err = a.ctr + 1;
    int* const lines_done = a.ctr + 2;
    int* const fwd_done = a.ctr + 2 + a.nslabs;
    const int b = threadIdx.x / EF_BS, jt = threadIdx.x % EF_BS;
    if (!ens_any(a, true)) return;
    const bool mixed = ens_any(a, false);
    for (int guard = 0; guard <= a.ntasks; ++guard) {
        if (threadIdx.x == 0) cur = atomicAdd(a.ctr, 1);
        __syncthreads();
        const int t = cur;
        if (t >= a.ntasks) break;
        const EnsTask tk = a.tasks[t];
        const int fi = tk.type == TASK_COLS ? tk.a : a.slabs[tk.a].field;
        const EnsField f = a.fields[fi];
        const FullLinks<double> U{(const double2*)f.links, f.g.V};
        const bool mine = ens_open(a, fi);
        if (!mine) {
            if (threadIdx.x == 0 && tk.type != TASK_COLS)
                atomicAdd((tk.type == TASK_LINES ? lines_done : fwd_done) + tk.a, 1);
        } else if (tk.type == TASK_COLS) {
            const int nt = f.g.n[0];
            double v[4] = {0.0, 0.0, 0.0, 0.0};
            for (int k = threadIdx.x; k < tk.n * nt; k += 3 * EF_BS) {
                const int64_t s = (int64_t)tk.b * nt + k;
                int c[4];
                site_coords(f.g, s, c);
                i64 tp = 0, sp = 0;
#pragma unroll 1
                for (int mu = 0; mu < 3; ++mu) {
                    const int64_t smu = s + (mu == 0 ? disp(f.g, 0, c[0], 1) : mu == 1 ? disp(f.g, 1, c[1], 1) : disp(f.g, 2, c[2], 1));
                    const M3F umu = fx_of(U.load(s, mu));
#pragma unroll 1
                    for (int nu = mu + 1; nu < 4; ++nu) {
                        const int64_t snu = s + (nu == 1 ? disp(f.g, 1, c[1], 1) : nu == 2 ? disp(f.g, 2, c[2], 1) : disp(f.g, 3, c[3], 1));
                        const M3F p = fx_mm<false, false>(umu, fx_of(U.load(smu, nu)));
                        const M3F q = fx_mm<false, false>(fx_of(U.load(s, nu)), fx_of(U.load(snu, mu)));
                        const i64 r = fx_retr<false, true>(p, q);
                        if (mu == 0)
                            tp += r;
                        else
                            sp += r;
                    }
                }
                v[0] += (double)sp * 0x1p-58;
                v[1] += (double)tp * 0x1p-58;
            }
            // eight lanes a column, each its run of links, then three levels
            // (as k_polyakov_fix); short columns one lane
            const int nl = nt >= 16 ? 8 : 1, per = 3 * EF_BS / nl, kk = (nt + nl - 1) / nl, lane = threadIdx.x % nl;
            const int t0 = min(nt, lane * kk), t1 = min(nt, t0 + kk);
#pragma unroll 1
            for (int c0 = 0; c0 < tk.n; c0 += per) {
                const int col = c0 + threadIdx.x / nl;
                M3F p;
#pragma unroll
                for (int e = 0; e < 9; ++e) p.r[e] = {e % 4 == 0 ? 1 << 29 : 0, 0}, p.i[e] = {0, 0};
                if (col < tk.n) {
                    const int64_t s0 = (int64_t)(tk.b + col) * nt;
#pragma unroll 1
                    for (int tt = t0; tt < t1; ++tt) {
                        const M3F u = fx_of(U.load(s0 + tt, 0));
                        p = tt > t0 ? fx_mm<false, false>(p, u) : u;
                    }
                }
#pragma unroll 1
                for (int off = 1; off < nl; off <<= 1) {
                    const M3F q = fx_shfl_down(p, off);
                    if ((lane & (2 * off - 1)) == 0) p = fx_mm<false, false>(p, q);
                }
                if (col < tk.n && lane == 0) {
                    v[2] += (double)(fx_int60(p.r[0]) + fx_int60(p.r[4]) + fx_int60(p.r[8])) * 0x1p-60;
                    v[3] += (double)(fx_int60(p.i[0]) + fx_int60(p.i[4]) + fx_int60(p.i[8])) * 0x1p-60;
                }
            }
#pragma unroll
            for (int o = 0; o < 4; ++o) {
                const double r = block_sum(v[o], sh);
                if (threadIdx.x == 0) a.part[(int64_t)t * NOBS + o] = r;
            }
        } else {
            const int j = tk.a;
            const EnsSlab sl = a.slabs[j];
            const Geom g = make_geom(sl.nts, f.g.n[1], f.g.n[2], f.g.n[3]);
            const MatFix lines{(int4*)(a.ring + (size_t)(j % kSlots) * a.slot_bytes), g.V,
                                  3 * a.pa.nd};
            if (tk.type == TASK_LINES) {
                if (threadIdx.x < 32) {
                    const int i = ring_prev(a, j, true, mixed);
                    if (threadIdx.x == 0) ok = i < 0 || flow_wait(fwd_done + i, a.slabs[i].nchunk, err);
                }
                __syncthreads();
#pragma unroll 1
                for (int h = 0; h < CH && ok; h += EF_BS) {  // a thread a (site, direction)
                    const int64_t s = (int64_t)tk.b * CH + h + jt;
                    if (s < g.V) line_site_fix(U, g, f.g, sl.t0, a.pa, lines, s, b);
                }
                __syncthreads();
                if (threadIdx.x == 0) {
                    __threadfence();
                    atomicAdd(lines_done + j, 1);
                }
            } else {
                if (threadIdx.x == 0) ok = flow_wait(lines_done + j, sl.nchunk, err);
                __syncthreads();
                double e = 0.0;
                int par = 0;
#pragma unroll 1
                for (int h = 0; h < CH && ok; h += EF_BS) {
                    const int64_t s = (int64_t)tk.b * CH + h + jt;
#pragma unroll 1
                    for (int p = 0; p < a.pa.np; ++p) {
                        longlong2(*sq)[EF_BS] = sq2[par];
                        par ^= 1;
                        if (s < g.V) {
                            int c[4];
                            site_coords(g, s, c);
                            const FxVS q = fwd_q_fix<u32>(g, a.pa, 1, lines, s, c, p, b);
#pragma unroll
                            for (int k = 0; k < 3; ++k) sq[3 * k + b][jt] = make_longlong2(q.r[k], q.i[k]);
                        }
                        __syncthreads();
                        if (b == p % 3 && s < g.V) {
                            i64 d[9];
                            fx_antiherm([&](int el) { return sq[el][jt]; }, d);
                            double fv[9];
                            fx_field_strength(d, FXQ5, fv);
                            e += ah_norm2(fv);
                        }
                    }
                }
                const double r = block_sum(e, sh);
                if (threadIdx.x == 0) {
                    a.part[(int64_t)t * NOBS + 4] = r;
                    __threadfence();
                    atomicAdd(fwd_done + j, 1);
                }
            }
        }
        __syncthreads();
    }
}

// out[f*NOBS + o] = sum of the field's task partials in list order (its
// tasks are ftask[ffirst[f] .. ffirst[f+1])); B^2 divided by V.  When a wait
// of the scheduler ran out (err != 0) every observable is NaN.
__global__ void k_ensemble_finish(const double* __restrict__ part, const int* __restrict__ ffirst,
                                  const int* __restrict__ ftask, const EnsField* fields, int nfields,
                                  const int* __restrict__ err, const int* __restrict__ err2,
                                  double* __restrict__ out) {
    const int f = blockIdx.x;
    if (f >= nfields) return;
    const int o = threadIdx.x;
    if (o >= NOBS) return;
    if (o == 5) {
        out[f * NOBS + 5] = (double)fields[f].g.V;
        return;
    }
    double acc = 0.0;
    for (int k = ffirst[f]; k < ffirst[f + 1]; ++k) acc += part[(int64_t)ftask[k] * NOBS + o];
    if (o == 4) acc /= (double)fields[f].g.V;
    out[f * NOBS + o] = (*err || *err2) ? __longlong_as_double(0x7ff8000000000000LL) : acc;
}

FLUE_OOB_READER(ensemble)

}  // namespace flue

// ===========================================================================
// C ABI
// ===========================================================================
using namespace flue;

struct flue_ensemble {
    int prec = 0;
    int nfields = 0;
    int ntasks = 0;
    int nslabs = 0;
    int tile = 0;
    int grid = 0, grid_fix = 0;
    int block = 128;
    int with_b2 = 1;
    bool fix = false;  // complex128 in fixed point where a field's gate allows
    EnsField* d_fields = nullptr;
    EnsSlab* d_slabs = nullptr;
    EnsTask* d_tasks = nullptr;
    int* d_ffirst = nullptr;
    int* d_ftask = nullptr;
    int* d_ctr = nullptr;  // task counter, error flag, per-slab done counters (complex128: twice, then the gates)
    double* d_part = nullptr;
    char* d_ring = nullptr;
    size_t slot_bytes = 0;
    double* d_out = nullptr;  // output the graph writes to
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    // pipeline mode (tile_cols = 0): per field the device entry points
    // (plaquettes, Polyakov loop, line-based B^2) with one library workspace
    int pipeline = 0;
    std::vector<flue_field> hfields;
    void* d_ws = nullptr;
    size_t ws_bytes = 0;
    uint64_t launches_per_eval = 2;  // kernels one replay runs
};

// V of every field (and B^2 = 0 without it) into the output of pipeline mode
__global__ void k_ensemble_volumes(const EnsField* __restrict__ fields, int nfields, int with_b2,
                                   double* __restrict__ out) {
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= nfields) return;
    out[f * NOBS + 5] = (double)fields[f].g.V;
    if (!with_b2) out[f * NOBS + 4] = 0.0;
}

static cudaError_t ens_launch_pipeline(flue_ensemble* e, double* d_out, cudaStream_t st) {
    for (int f = 0; f < e->nfields; ++f) {
        const flue_field* U = &e->hfields[f];
        double* o = d_out + (size_t)f * NOBS;
        int rc = flue_plaquette(U, 2, 4, 4, o, e->d_ws, e->ws_bytes, st);  // spatial planes
        if (!rc) rc = flue_plaquette(U, 1, 1, 4, o + 1, e->d_ws, e->ws_bytes, st);  // temporal planes
        if (!rc) rc = flue_polyakov(U, o + 2, e->d_ws, e->ws_bytes, st);
        if (!rc && e->with_b2) rc = flue_magnetic(U, o + 4, e->d_ws, e->ws_bytes, st);
        if (rc) return cudaErrorUnknown;
    }
    note_launch(), k_ensemble_volumes<<<(e->nfields + 127) / 128, 128, 0, st>>>(e->d_fields, e->nfields, e->with_b2,
                                                                                d_out);
    return cudaGetLastError();
}

template <class L, typename T, int BS>
static cudaError_t flow_launch(const EnsFlowArgs& args, int grid, cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(BS);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;  // every block resident: the waits in the kernel progress
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    note_launch();
    return cudaLaunchKernelEx(&cfg, k_ens_flow<L, T, BS>, args);
}

template <int BS>
static cudaError_t flow_dispatch(const flue_ensemble* e, const EnsFlowArgs& args, cudaStream_t st) {
    if (e->prec == PREC_C128) return flow_launch<FullLinks<double>, double, BS>(args, e->grid, st);
    if (e->prec == PREC_C64) return flow_launch<FullLinks<float>, float, BS>(args, e->grid, st);
    return flow_launch<R12Links, float, BS>(args, e->grid, st);
}

static PlaneArg b2_plane_arg() {
    // magnetic: Loop5(3,2), Loop5(2,4), Loop5(4,3) (src/wloops.F90:502-506), 0-based
    PlaneArg pa;
    pa.np = 3;
    const int mu[3] = {2, 1, 3}, nu[3] = {1, 3, 2};
    for (int k = 0; k < 4; ++k) pa.slot[k] = -1, pa.dir[k] = -1;
    pa.nd = 0;
    for (int p = 0; p < 3; ++p) {
        pa.mu[p] = mu[p];
        pa.nu[p] = nu[p];
        for (int d : {mu[p], nu[p]})
            if (pa.slot[d] < 0) pa.slot[d] = pa.nd, pa.dir[pa.nd++] = d;
    }
    for (int p = 3; p < 6; ++p) pa.mu[p] = pa.nu[p] = 0;
    return pa;
}

template <int CH>
static cudaError_t flow_fix_launch(const flue_ensemble* e, const EnsFlowArgs& args, cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)e->grid_fix);
    cfg.blockDim = dim3(3 * EF_BS);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    note_launch();
    return cudaLaunchKernelEx(&cfg, k_ens_flow_fix<CH>, args);
}

// ints of one scheduler's counters, and of all of them (see d_ctr)
static size_t ctr_ints(const flue_ensemble* e) { return 2 + 2 * (size_t)e->nslabs; }
static size_t ctr_total(const flue_ensemble* e) {
    return e->fix ? 2 * ctr_ints(e) + 2 * (size_t)e->nfields : ctr_ints(e);
}

static cudaError_t ens_launch(flue_ensemble* e, double* d_out, cudaStream_t st) {
    if (e->pipeline) return ens_launch_pipeline(e, d_out, st);
    cudaError_t r = cudaMemsetAsync(e->d_ctr, 0, sizeof(int) * ctr_total(e), st);
    if (r != cudaSuccess) return r;
    EnsFlowArgs args;
    args.fields = e->d_fields;
    args.slabs = e->d_slabs;
    args.tasks = e->d_tasks;
    args.ntasks = e->ntasks;
    args.nslabs = e->nslabs;
    args.ctr = e->d_ctr;
    args.part = e->d_part;
    args.ring = e->d_ring;
    args.slot_bytes = e->slot_bytes;
    args.pa = b2_plane_arg();
    args.nfields = e->nfields;
    args.gates = nullptr;
    const int* err2 = e->d_ctr + 1;
    if (e->fix) {
        // fields that pass the gate in fixed point, then the others in FP64 (a
        // scheduler and counters of their own; nothing to do, as a rule)
        args.gates = (u32*)(e->d_ctr + 2 * ctr_ints(e));
        const unsigned gy = (unsigned)std::min(e->nfields, 65535);
        note_launch(), k_ens_gates<<<dim3(std::max(1u, 4096u / gy), gy), 128, 0, st>>>(args);
        r = e->block == 256 ? flow_fix_launch<256>(e, args, st) : flow_fix_launch<128>(e, args, st);
        if (r != cudaSuccess) return r;
        args.ctr = e->d_ctr + ctr_ints(e);
        err2 = args.ctr + 1;
    }
    r = e->block == 256 ? flow_dispatch<256>(e, args, st) : flow_dispatch<128>(e, args, st);
    if (r != cudaSuccess) return r;
    note_launch(), k_ensemble_finish<<<e->nfields, 32, 0, st>>>(e->d_part, e->d_ffirst, e->d_ftask, e->d_fields,
                                                               e->nfields, e->d_ctr + 1, err2, d_out);
    return cudaGetLastError();
}

static void ens_free(flue_ensemble* e) {
    if (e->exec) cudaGraphExecDestroy(e->exec);
    if (e->graph) cudaGraphDestroy(e->graph);
    cudaFree(e->d_fields);
    cudaFree(e->d_slabs);
    cudaFree(e->d_tasks);
    cudaFree(e->d_ffirst);
    cudaFree(e->d_ftask);
    cudaFree(e->d_ctr);
    cudaFree(e->d_part);
    cudaFree(e->d_ring);
    cudaFree(e->d_ws);
    delete e;
}

template <class L, typename T, int BS>
static int flow_blocks_per_sm() {
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_ens_flow<L, T, BS>, BS, 0) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

static int flow_occupancy(int prec, int block) {
    if (block == 256) {
        if (prec == PREC_C128) return flow_blocks_per_sm<FullLinks<double>, double, 256>();
        if (prec == PREC_C64) return flow_blocks_per_sm<FullLinks<float>, float, 256>();
        return flow_blocks_per_sm<R12Links, float, 256>();
    }
    if (prec == PREC_C128) return flow_blocks_per_sm<FullLinks<double>, double, 128>();
    if (prec == PREC_C64) return flow_blocks_per_sm<FullLinks<float>, float, 128>();
    return flow_blocks_per_sm<R12Links, float, 128>();
}

extern "C" {

int flue_ensemble_create(flue_ensemble** out, const flue_field* fields, int nfields, int tile_cols, int block,
                         int blocks_per_sm, int with_b2) {
    if (!out || !fields || nfields < 1) return FLUE_ERR_ARG;
    const bool pipeline = tile_cols == 0;
    if (tile_cols < 0 || (!pipeline && ((block != 128 && block != 256) || blocks_per_sm < 1 || blocks_per_sm > 16)))
        return FLUE_ERR_ARG;
    const int prec = fields[0].prec;
    std::vector<EnsField> hf(nfields);
    for (int f = 0; f < nfields; ++f) {
        const flue_field& F = fields[f];
        if (!F.links) return FLUE_ERR_ARG;
        if (F.prec != prec) return FLUE_ERR_DTYPE;  // one precision per ensemble
        if (F.prec != FLUE_C128 && F.prec != FLUE_C64 && F.prec != FLUE_R12) return FLUE_ERR_DTYPE;
        if (F.nt < 1 || F.nx < 1 || F.ny < 1 || F.nz < 1 || (int64_t)F.nt * F.nx * F.ny * F.nz >= ((int64_t)1 << 31))
            return FLUE_ERR_SHAPE;
        hf[f].links = F.links;
        hf[f].g = make_geom(F.nt, F.nx, F.ny, F.nz);
    }
    // the task list (see the top of the file): per slab j its LINES tasks,
    // then the FWD tasks of slab j - 1; the COLS tasks last
    std::vector<EnsSlab> slabs;
    std::vector<EnsTask> tasks;
    std::vector<std::vector<int>> per_field(nfields);
    int64_t max_slab = 1;
    bool fix = prec == FLUE_C128;
    if (!pipeline) {
        for (int f = 0; f < nfields && with_b2; ++f) {
            const Geom& g = hf[f].g;
            const int64_t v3 = g.V / g.n[0];
            const int64_t want = slab_sites();
            int nts = (int)((want + v3 - 1) / v3);
            if (nts > g.n[0]) nts = g.n[0];
            if (nts < 1) nts = 1;
            for (int t0 = 0; t0 < g.n[0]; t0 += nts) {
                const int n = g.n[0] - t0 < nts ? g.n[0] - t0 : nts;
                const int64_t vs = (int64_t)n * v3;
                // the forward reads a slab's lines with 32-bit offsets
                if (!(prec == FLUE_C128 ? MatAoS<double>::fits32(vs, 9) : MatAoS<float>::fits32(vs, 9)))
                    return FLUE_ERR_SHAPE;
                fix = fix && MatFix::fits32(vs, 9);
                if (vs > max_slab) max_slab = vs;
                slabs.push_back({f, t0, n, (int)((vs + block - 1) / block)});
            }
        }
        const int ns = (int)slabs.size();
        for (int j = 0; j <= ns; ++j) {
            if (j < ns)
                for (int c = 0; c < slabs[j].nchunk; ++c) tasks.push_back({TASK_LINES, j, c, 0});
            if (j >= 1)
                for (int c = 0; c < slabs[j - 1].nchunk; ++c) {
                    per_field[slabs[j - 1].field].push_back((int)tasks.size());
                    tasks.push_back({TASK_FWD, j - 1, c, 0});
                }
        }
        for (int f = 0; f < nfields; ++f) {
            const int ncol = fields[f].nx * fields[f].ny * fields[f].nz;
            for (int c0 = 0; c0 < ncol; c0 += tile_cols) {
                per_field[f].push_back((int)tasks.size());
                tasks.push_back({TASK_COLS, f, c0, std::min(tile_cols, ncol - c0)});
            }
        }
    }
    std::vector<int> ffirst(nfields + 1, 0), ftask;
    for (int f = 0; f < nfields; ++f) {
        ffirst[f] = (int)ftask.size();
        ftask.insert(ftask.end(), per_field[f].begin(), per_field[f].end());
    }
    ffirst[nfields] = (int)ftask.size();
    if (ftask.empty()) ftask.push_back(0);  // (keeps the allocations non-empty)
    if (slabs.empty()) slabs.push_back({0, 0, 1, 0});
    if (tasks.empty()) tasks.push_back({TASK_COLS, 0, 0, 0});
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    flue_ensemble* e = new flue_ensemble();
    e->prec = prec;
    e->nfields = nfields;
    e->tile = tile_cols;
    e->block = block;
    e->with_b2 = with_b2 ? 1 : 0;
    e->fix = fix;
    cudaError_t r = cudaSuccess;
    if (pipeline) {
        e->pipeline = 1;
        e->hfields.assign(fields, fields + nfields);
        for (const flue_field& F : e->hfields)
            for (int op : {FLUE_OP_PLAQUETTE, FLUE_OP_POLYAKOV, FLUE_OP_MAGNETIC}) {
                if (op == FLUE_OP_MAGNETIC && !e->with_b2) continue;
                const size_t n = flue_workspace_bytes(op, F.nt, F.nx, F.ny, F.nz, F.prec);
                if (n > e->ws_bytes) e->ws_bytes = n;
            }
        if ((r = cudaMalloc(&e->d_ws, e->ws_bytes < 256 ? 256 : e->ws_bytes)) != cudaSuccess) {
            ens_free(e);
            cudaGetLastError();
            return FLUE_ERR_NOMEM;
        }
    } else {
        // every block must be resident (cooperative launch)
        const int occ = flow_occupancy(prec, block);
        if (occ < 1) {
            ens_free(e);
            return FLUE_ERR_CUDA;
        }
        e->grid = nsm * (blocks_per_sm < occ ? blocks_per_sm : occ);
        e->ntasks = (int)tasks.size();
        e->nslabs = (int)slabs.size();
        if (fix) {
            int n = 0;
            const cudaError_t ro =
                block == 256 ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_ens_flow_fix<256>, 3 * EF_BS, 0)
                             : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_ens_flow_fix<128>, 3 * EF_BS, 0);
            if (ro != cudaSuccess || n < 1) {
                ens_free(e);
                cudaGetLastError();
                return FLUE_ERR_CUDA;
            }
            e->grid_fix = nsm * n;
        }
        e->slot_bytes = prec == PREC_C128 ? std::max(MatAoS<double>::bytes(max_slab, 9), MatFix::bytes(max_slab, 9))
                                          : MatAoS<float>::bytes(max_slab, 9);
        e->slot_bytes = (e->slot_bytes + 255) & ~(size_t)255;
        if ((r = cudaMalloc(&e->d_ring, kSlots * e->slot_bytes)) != cudaSuccess) {
            ens_free(e);
            cudaGetLastError();
            return FLUE_ERR_NOMEM;
        }
    }
    if ((r = cudaMalloc(&e->d_fields, sizeof(EnsField) * nfields)) != cudaSuccess ||
        (r = cudaMalloc(&e->d_slabs, sizeof(EnsSlab) * slabs.size())) != cudaSuccess ||
        (r = cudaMalloc(&e->d_tasks, sizeof(EnsTask) * tasks.size())) != cudaSuccess ||
        (r = cudaMalloc(&e->d_ffirst, sizeof(int) * (nfields + 1))) != cudaSuccess ||
        (r = cudaMalloc(&e->d_ftask, sizeof(int) * ftask.size())) != cudaSuccess ||
        (r = cudaMalloc(&e->d_ctr, sizeof(int) * (2 * (2 + 2 * slabs.size()) + 2 * (size_t)nfields))) != cudaSuccess ||
        (r = cudaMalloc(&e->d_part, sizeof(double) * NOBS * tasks.size())) != cudaSuccess) {
        ens_free(e);
        cudaGetLastError();
        return FLUE_ERR_NOMEM;
    }
    if ((r = cudaMemcpy(e->d_fields, hf.data(), sizeof(EnsField) * nfields, cudaMemcpyHostToDevice)) != cudaSuccess ||
        (r = cudaMemcpy(e->d_slabs, slabs.data(), sizeof(EnsSlab) * slabs.size(), cudaMemcpyHostToDevice)) !=
            cudaSuccess ||
        (r = cudaMemcpy(e->d_tasks, tasks.data(), sizeof(EnsTask) * tasks.size(), cudaMemcpyHostToDevice)) !=
            cudaSuccess ||
        (r = cudaMemcpy(e->d_ffirst, ffirst.data(), sizeof(int) * (nfields + 1), cudaMemcpyHostToDevice)) !=
            cudaSuccess ||
        (r = cudaMemcpy(e->d_ftask, ftask.data(), sizeof(int) * ftask.size(), cudaMemcpyHostToDevice)) !=
            cudaSuccess ||
        (r = cudaMemset(e->d_part, 0, sizeof(double) * NOBS * tasks.size())) != cudaSuccess) {
        ens_free(e);
        return FLUE_ERR_CUDA;
    }
    *out = e;
    return FLUE_OK;
}

int flue_ensemble_items(const flue_ensemble* e) { return e ? e->ntasks : -1; }

// Direct (uncaptured) launch of the memset + persistent kernel + finisher.
int flue_ensemble_run(flue_ensemble* e, double* d_out, void* stream) {
    if (!e || !d_out) return FLUE_ERR_ARG;
    return ens_launch(e, d_out, (cudaStream_t)stream) == cudaSuccess ? FLUE_OK : FLUE_ERR_CUDA;
}

// Capture the launch sequence writing to d_out into a CUDA graph (on a
// private stream) and instantiate it; flue_ensemble_replay then launches it.
int flue_ensemble_capture(flue_ensemble* e, double* d_out) {
    if (!e || !d_out) return FLUE_ERR_ARG;
    cudaStream_t cs;
    if (cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking) != cudaSuccess) return FLUE_ERR_CUDA;
    cudaError_t r = cudaSuccess;
    if (e->pipeline) {
        // one uncaptured evaluation first: the entry points set up their
        // library streams and caches on first use, outside the capture
        r = ens_launch(e, d_out, cs);
        if (r == cudaSuccess) r = cudaStreamSynchronize(cs);
    }
    if (r == cudaSuccess) r = cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal);
    if (r == cudaSuccess) {
        // captured launches are counted by note_launch although they do not
        // run here; take them back out and count them at each replay
        const uint64_t n0 = flue_kernel_launches();
        cudaError_t rl = ens_launch(e, d_out, cs);
        const uint64_t n1 = flue_kernel_launches();
        e->launches_per_eval = n1 - n0;
        flue::note_launch(-(int)(n1 - n0));
        cudaGraph_t g = nullptr;
        r = cudaStreamEndCapture(cs, &g);
        if (rl != cudaSuccess) r = rl;
        if (r == cudaSuccess) {
            if (e->exec) cudaGraphExecDestroy(e->exec);
            if (e->graph) cudaGraphDestroy(e->graph);
            e->graph = g;
            r = cudaGraphInstantiate(&e->exec, g, 0);
            e->d_out = d_out;
        } else if (g) {
            cudaGraphDestroy(g);
        }
    }
    cudaStreamDestroy(cs);
    if (r != cudaSuccess) {
        cudaGetLastError();
        return FLUE_ERR_CUDA;
    }
    return FLUE_OK;
}

int flue_ensemble_replay(flue_ensemble* e, void* stream) {
    if (!e || !e->exec) return FLUE_ERR_ARG;
    flue::note_launch((int)e->launches_per_eval);  // the kernels the graph holds
    return cudaGraphLaunch(e->exec, (cudaStream_t)stream) == cudaSuccess ? FLUE_OK : FLUE_ERR_CUDA;
}

int flue_ensemble_destroy(flue_ensemble* e) {
    if (!e) return FLUE_ERR_ARG;
    ens_free(e);
    return FLUE_OK;
}

}  // extern "C"
