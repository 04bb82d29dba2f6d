"""Kernels whose warps or blocks meet at barriers and counters, run on the CPU
(cuda_emu.h) under several orders of warps and blocks: the result may not depend
on the order.  A wrong order is rare on a GPU, and a test there proves nothing."""
import os
import re
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "flue_gb300", "csrc")

# the inline PTX of the sources, in C++
PTX = [
    ('asm("shr.u64 %0, %0, %1;" : "+l"(m) : "r"(sh));', "m = sh < 64 ? m >> sh : 0;"),
    ('asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");',
     "v = *(volatile const int*)p;"),
]


def _source(name):
    text = open(os.path.join(CSRC, name)).read()
    for ptx, cpp in PTX:
        text = text.replace(ptx, cpp)
    assert not re.search(r"\basm\b", text), name
    return text


def _cut(text, start, end):
    """From the line `start` up to the line `end`."""
    a = text.index(start)
    return text[a:text.index(end, a)]


def _build(tmp_path, body):
    """Compiles body (C++) over the headers of csrc/; returns the program."""
    from flue_gb300 import build

    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build.nvcc()))), "include")
    for h in ("flue_common.cuh", "fix.cuh", "loop5.cuh", "loop5_fix.cuh"):
        (tmp_path / h).write_text(_source(h))
    (tmp_path / "main.cpp").write_text('#include "cuda_emu.h"\n#include "fix.cuh"\n#include "loop5.cuh"\n'
                                       '#include "loop5_fix.cuh"\nnamespace flue {\n' + body)
    exe = tmp_path / "main"
    r = subprocess.run([shutil.which("g++"), "-std=c++17", "-O1", "-ffp-contract=off", "-w", "-pthread", "-I", str(tmp_path), "-I", HERE, "-I",
                        include, str(tmp_path / "main.cpp"), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-4000:]
    return str(exe)


# random links: rows 0 and 1 orthonormalised, row 2 = conj(row0 x row1)
LINKS = r"""
struct Rng {
    uint64_t s;
    double operator()() {  // (-1, 1)
        s = s * 6364136223846793005ull + 1442695040888963407ull;
        return (double)(int64_t)s * 0x1p-63;
    }
};
static void random_link(Rng& rng, double r[3][3], double i[3][3]) {
    for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 3; ++b) r[a][b] = rng(), i[a][b] = rng();
    fix_su3_rows(r, i);
}
"""

FLOW_MAIN = LINKS + r"""
template <int STAGE>
static void stage(const std::vector<int>& order, const Geom& g, MatFix w, MatFix wo, AHFix xb, FlowStage sc, FixGate gt,
                  double2* links) {
    const unsigned nb = (unsigned)((g.V + FF_BS - 1) / FF_BS) * 4;
    emu::launch(nb, 3 * FF_BS, order, [=] { k_flow_stage<STAGE, u32>(g, w, wo, xb, sc, links, gt); });
}
static std::vector<double> step(const std::vector<int>& order, double eps) {
    const Geom g = make_geom(5, 3, 2, 2);
    std::vector<int4> a(MatFix::bytes(g.V, 4) / 16), b(a.size());
    std::vector<longlong2> x(AHFix::bytes(g.V, 4) / 16);
    MatFix w0{a.data(), g.V}, w1{b.data(), g.V};
    AHFix xb{x.data(), g.V};
    Rng rng{5};
    for (int mu = 0; mu < 4; ++mu)
        for (int64_t s = 0; s < g.V; ++s) {
            double r[3][3], i[3][3];
            random_link(rng, r, i);
            for (int k = 0; k < 9; ++k) w0.store_el(s, mu, k, fx_of(r[k / 3][k % 3]), fx_of(i[k / 3][k % 3]));
        }
    u32 gate[3] = {0, 0, 0};
    FixGate gt;
    gt.p = gate;
    const double f[3] = {0.25, 8.0 / 9.0, 0.75}, last[3] = {0.0, -17.0 / 9.0, -1.0};
    FlowStage sc[3];
    for (int k = 0; k < 3; ++k) sc[k] = {fx_const(-32.0 * eps * f[k]), fx_const(-64.0 / 3.0 * eps * f[k]), fx_const(last[k])};
    std::vector<double> out(72 * g.V);
    stage<0>(order, g, w0, w1, xb, sc[0], gt, nullptr);
    stage<1>(order, g, w1, w0, xb, sc[1], gt, nullptr);
    stage<2>(order, g, w0, w1, xb, sc[2], gt, (double2*)out.data());
    return out;
}
}  // namespace flue
int main() {
    const auto a = flue::step({0, 1, 2}, 0.05);
    const size_t n = a.size() / 18;  // links; element k of link l at 2 (l + n k)
    for (size_t l = 0; l < n; ++l)
        for (int p = 0; p < 3; ++p)
            for (int q = 0; q < 3; ++q) {  // columns p and q of the link
                double re = p == q ? -1.0 : 0.0, im = 0.0;
                for (int k = 0; k < 3; ++k) {
                    const double *u = &a[2 * (l + n * (k + 3 * p))], *v = &a[2 * (l + n * (k + 3 * q))];
                    re += u[0] * v[0] + u[1] * v[1], im += u[0] * v[1] - u[1] * v[0];
                }
                if (std::fabs(re) + std::fabs(im) > 1e-14) return printf("not unitary: %g %g\n", re, im), 1;
            }
    for (const std::vector<int>& o : {std::vector<int>{1, 2, 0}, {2, 1, 0}, {1, 0, 2}})
        if (memcmp(flue::step(o, 0.05).data(), a.data(), a.size() * 8)) return printf("depends on the order\n"), 1;
    return 0;
}
"""


def test_flow_stage_in_any_order_of_its_warps(tmp_path):
    """The three warps of a link (one a column) in four orders of a Wilson-flow
    step: the same links, bit for bit, and unitary."""
    flow = _source("flow.cu")
    body = _cut(flow, "// a value of unit 2^-60 as limbs\n", "template <typename I>\nstatic void flow_fix_stages")
    exe = _build(tmp_path, body + FLOW_MAIN)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


ENS_MAIN = LINKS + r"""
// Five fields of 18-site time slices, one slab a slice, every other one left to
// the other scheduler; `part` after one scheduler over all of them.  turns: one resident
// block each, and the waits it may take before the next one runs.
static std::vector<double> run(const std::vector<int>& turns, bool fixed, std::vector<EnsTask>& tasks) {
    const int nts[5] = {6, 5, 7, 6, 6};
    std::vector<EnsField> fields;
    std::vector<EnsSlab> slabs;
    std::vector<std::vector<double2>> links(5);
    std::vector<u32> gates;
    Rng rng{7};
    for (int f = 0; f < 5; ++f) {
        const Geom g = make_geom(nts[f], 2, 3, 3);
        links[f].resize(36 * g.V);
        for (int mu = 0; mu < 4; ++mu)
            for (int64_t s = 0; s < g.V; ++s) {
                double r[3][3], i[3][3];
                random_link(rng, r, i);
                for (int a = 0; a < 3; ++a)
                    for (int b = 0; b < 3; ++b) links[f][s + g.V * (mu + 4 * (a + 3 * b))] = {r[a][b], i[a][b]};
            }
        fields.push_back({links[f].data(), g});
        for (int t = 0; t < nts[f]; ++t) slabs.push_back({f, t, 1, 1});
        // fields 0, 2 and 4 are the scheduler's own (FP64: those that are shut)
        gates.push_back((f % 2 == 0) != fixed), gates.push_back((u32)(4 * g.V));
    }
    const int ns = (int)slabs.size();
    tasks.clear();
    for (int j = 0; j <= ns; ++j) {
        if (j < ns) tasks.push_back({TASK_LINES, j, 0, 0});
        if (j >= 1) tasks.push_back({TASK_FWD, j - 1, 0, 0});
    }
    const size_t slot = std::max(MatFix::bytes(18, 9), MatAoS<double>::bytes(18, 9));
    std::vector<int> ctr(2 + 2 * ns);
    std::vector<double> part(tasks.size() * NOBS);
    std::vector<longlong2> ring(kSlots * slot / 16);
    EnsFlowArgs a{};
    a.fields = fields.data(), a.slabs = slabs.data(), a.tasks = tasks.data();
    a.ntasks = (int)tasks.size(), a.nslabs = ns, a.ctr = ctr.data(), a.part = part.data();
    a.ring = (char*)ring.data(), a.slot_bytes = slot, a.nfields = 5, a.gates = gates.data();
    const int mu[3] = {2, 1, 3}, nu[3] = {1, 3, 2}, sl[4] = {-1, 1, 0, 2}, dir[3] = {2, 1, 3};
    a.pa.np = 3, a.pa.nd = 3;
    for (int k = 0; k < 4; ++k) a.pa.slot[k] = sl[k], a.pa.dir[k] = k < 3 ? dir[k] : -1;
    for (int k = 0; k < 3; ++k) a.pa.mu[k] = mu[k], a.pa.nu[k] = nu[k];
    if (fixed)
        emu::launch_resident(3 * EF_BS, turns, [&] { k_ens_flow_fix<128>(a); });
    else
        emu::launch_resident(128, turns, [&] { k_ens_flow<FullLinks<double>, double, 128>(a); });
    if (ctr[1]) part.assign(part.size(), -1.0);  // a wait ran out
    return part;
}
}  // namespace flue
int main() {
    using namespace flue;
    std::vector<EnsTask> tasks;
    for (bool fixed : {true, false}) {
        const auto want = run({1}, fixed, tasks);
        std::vector<std::vector<int>> speeds{{1, 1}, {1, 30, 30}, {30, 1, 5}};
        for (int n = 40; n <= 400; n += 30) speeds.push_back({1, n}), speeds.push_back({n, 2, n});
        for (const std::vector<int>& turns : speeds) {
            const auto got = run(turns, fixed, tasks);
            for (size_t t = 0; t < tasks.size(); ++t)
                if (tasks[t].type == TASK_FWD && got[t * NOBS + 4] != want[t * NOBS + 4])
                    return printf("%s: slab %d, %zu blocks\n", fixed ? "fixed point" : "FP64", tasks[t].a, turns.size()), 1;
        }
    }
    return 0;
}
"""


def test_ensemble_ring_in_any_order_of_its_blocks(tmp_path):
    """Fields that a scheduler owns between fields that it skips, blocks of very
    different speed: no slab's lines are overwritten while they are read."""
    ens = _source("ensemble.cu")
    body = _cut(ens, "constexpr int NOBS = 6;\n", "// out[f*NOBS + o] = sum of the field's task partials")
    exe = _build(tmp_path, body + ENS_MAIN)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
