"""The bounds-checked build (test_gpu_bounds) on what complex128 fields take beside
the entry points run there: time slabs, the host-buffer call and ensembles, with
open gates, shut ones and both; planes of the intermediates are checked too."""
import ctypes

import numpy as np
import pytest

from flue_gb300 import _lib, ensemble, flow, forces, generate, gluonCalc as G
from flue_gb300.field import GaugeField
from tests.test_gpu_bounds import DIMS, checked  # noqa: F401 (fixture)

pytestmark = pytest.mark.gpu


def _field(dims, seed, shut):
    u = np.array(generate.random_field(dims, 0.5, seed))
    if shut:
        u[0, 0, 0, 0, 1] *= 1.01
    return np.asfortranarray(u)


def _run(monkeypatch):
    out = []
    for shut in (False, True):
        u = _field((8, 4, 6, 4), 5, shut)
        f = GaugeField.from_array(u)
        monkeypatch.setenv("FLUE_SLABS", "3")
        b, g = forces.magnetic_force(f)
        out += [b, float(g.abs().sum())]
        grad, e = np.empty_like(u, order="F"), ctypes.c_double()
        _lib.call("flue_magnetic_force_c", u.ctypes.data_as(ctypes.c_void_p), _lib.C128, *u.shape[:4], _lib.C128,
                  _lib.FORCE_LIE, ctypes.byref(e), grad.ctypes.data_as(ctypes.c_void_p))
        out += [e.value, float(np.abs(grad).sum())]
        monkeypatch.delenv("FLUE_SLABS")
        out.append(float(G.wmunu_table(f, 2, 1, 5, 3).sum()))
        h = f.clone()
        flow.wflow_step(h, 0.02)
        out.append(G.plaquette(h, 1, 4, 4)[0])
    for kinds in ((False,), (True,), (False, True)):  # shut or not, in turn
        monkeypatch.setenv("FLUE_ENS_SLAB_SITES", "1" if len(kinds) > 1 else "64")
        fs = [GaugeField.from_array(_field(d, 70 + i, kinds[i % len(kinds)])) for i, d in enumerate(DIMS)]
        for block in (128, 256):
            e = ensemble.Ensemble(fs, block=block)
            out += list(e.run(graph=False).ravel())
            e.close()  # with the library that created it
        e = ensemble.Ensemble(fs, mode="pipeline")
        out += list(e.run(graph=False).ravel())
        e.close()
    return np.array(out)


def test_complex128_stays_in_bounds(checked, monkeypatch):  # noqa: F811
    want = _run(monkeypatch)
    saved = _lib._lib
    _lib._lib = checked
    try:
        checked.flue_bounds_errors()
        got = _run(monkeypatch)
        assert checked.flue_bounds_errors() == 0
        checked.flue_release_host_cache()
    finally:
        _lib._lib = saved
    assert np.allclose(got, want, rtol=1e-12, atol=1e-12)
