"""Stage timing (flue_stage_timing) of the field strength: lines and forward, in
every precision and for both kinds; the FP32 clover has no lines stage to run."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from flue_gb300 import _lib, generate, gluonCalc as G
from flue_gb300.field import GaugeField

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["c128", "c64", "r12"])
@pytest.mark.parametrize("call", [G.cloverloopmunucoord, G.loop5munucoord])
def test_field_strength_records_its_stages(call, prec):
    L = _lib.load()
    f = GaugeField.from_array(generate.random_field((8, 4, 4, 4), 0.3, 2), prec=prec)
    L.flue_stage_timing(1)
    try:
        call(f, 2, 3)
        ms, n = (ctypes.c_double * 8)(), ctypes.c_int()
        assert L.flue_stage_times(ms, 8, ctypes.byref(n)) == 0
    finally:
        L.flue_stage_timing(0)
    assert n.value == 2 and ms[1] > 0.0 and np.isfinite(ms[0])
