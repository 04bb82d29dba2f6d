"""The bounded compensated sums of the complex64 flow's reunitarisation against the
general ones, on the CPU (cuda_emu.h): links at any distance from 1 come out as
close to the exact result."""
import subprocess

from tests.test_schedules import LINKS, _build, _cut, _source

MAIN = LINKS + r"""
using Real = long double;
// FixSU3Matrix of rows 0 and 1; row 2 = conj(row 0 x row 1)
static void exact(Real r[3][3], Real i[3][3]) {
    auto unit = [&](int a) {
        Real n = 0;
        for (int c = 0; c < 3; ++c) n += r[a][c] * r[a][c] + i[a][c] * i[a][c];
        n = 1 / sqrtl(n);
        for (int c = 0; c < 3; ++c) r[a][c] *= n, i[a][c] *= n;
    };
    unit(0);
    Real dr = 0, di = 0;
    for (int c = 0; c < 3; ++c) dr += r[0][c] * r[1][c] + i[0][c] * i[1][c], di += r[0][c] * i[1][c] - i[0][c] * r[1][c];
    for (int c = 0; c < 3; ++c) {
        const Real p = r[0][c] * dr - i[0][c] * di, q = r[0][c] * di + i[0][c] * dr;
        r[1][c] -= p, i[1][c] -= q;
    }
    unit(1);
    for (int c = 0; c < 3; ++c) {
        const int j = (c + 1) % 3, k = (c + 2) % 3;
        r[2][c] = r[0][j] * r[1][k] - i[0][j] * i[1][k] - r[0][k] * r[1][j] + i[0][k] * i[1][j];
        i[2][c] = -(r[0][j] * i[1][k] + i[0][j] * r[1][k] - r[0][k] * i[1][j] - i[0][k] * r[1][j]);
    }
}
}  // namespace flue
int main() {
    using namespace flue;
    Rng rng{3};
    for (double dist = 0.5; dist > 1e-10; dist /= 2) {
        Real e_here = 0, e_general = 0;  // off the diagonal, squared
        for (int n = 0; n < 20000; ++n) {
            double m[3][3], mi[3][3];
            for (int a = 0; a < 3; ++a)  // 1 + an anti-Hermitian matrix
                for (int b = 0; b <= a; ++b) {
                    m[a][b] = a == b ? 1.0 : dist * rng(), mi[a][b] = dist * rng();
                    if (a != b) m[b][a] = -m[a][b], mi[b][a] = mi[a][b];
                }
            fix_su3_rows(m, mi);
            M3<float> w;
            float r[3][3], i[3][3];
            Real x[3][3], y[3][3];
            for (int a = 0; a < 3; ++a)
                for (int b = 0; b < 3; ++b) {
                    r[a][b] = w.r[3 * a + b] = (float)m[a][b], i[a][b] = w.i[3 * a + b] = (float)mi[a][b];
                    x[a][b] = r[a][b], y[a][b] = i[a][b];
                }
            exact(x, y);
            fix_su3_rows_f32<SumFF>(r, i);
            reunitarise(w);
            for (int a = 0; a < 3; ++a)
                for (int b = 0; b < 3; ++b)
                    if (a != b) {
                        const Real u = w.r[3 * a + b] - x[a][b], v = w.i[3 * a + b] - y[a][b];
                        const Real p = r[a][b] - x[a][b], q = i[a][b] - y[a][b];
                        e_here += u * u + v * v, e_general += p * p + q * q;
                    }
        }
        const double ratio = (double)sqrtl(e_here / e_general);
        if (!(ratio < 1.001)) return printf("at %g from 1: error %.3f of the general sums'\n", dist, ratio), 1;
    }
    return 0;
}
"""


def test_bounded_sums_are_as_exact_as_general_ones(tmp_path):
    """The rms error off the diagonal is that of the general sums, to a thousandth."""
    flow = _source("flow.cu")
    body = _cut(flow, "struct FF {", "// link u of direction mu at site s moved by")
    exe = _build(tmp_path, body + MAIN)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
