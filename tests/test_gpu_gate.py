"""complex128 calls around the gate between fixed point and FP64 (csrc/fix.cuh):
fields and regions that have to stay in FP64, and what a shut gate costs."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from flue_gb300 import generate
from flue_gb300 import gluonCalc as G
from flue_gb300.ensemble import Ensemble
from flue_gb300.field import as_field

pytestmark = pytest.mark.gpu


# 16 chunks a slab and a slab a time slice: the four ring slots go round many
# times, past fields of either scheduler.  Tolerance as for one field alone (sums
# of V squares, test_gpu_fix).
@pytest.mark.parametrize("block", [128, 256])
def test_ensemble_of_open_and_shut_fields_reuses_its_ring(block, monkeypatch):
    monkeypatch.setenv("FLUE_ENS_SLAB_SITES", "1")
    fields = []
    for i, nt in enumerate([6, 5, 7, 11, 6, 2, 9]):
        u = np.array(generate.random_field((nt, 16, 16, 8), 0.4, 40 + i))
        if i % 2:
            u[0, 1, 2, 3, 1] *= 1.01
        fields.append(as_field(np.asfortranarray(u)))
    e = Ensemble(fields, block=block)
    first = e.run().copy()
    for _ in range(20):
        assert np.array_equal(first, e.run())
    for f, r in zip(fields, first):
        b2 = G.magnetic(f)
        assert abs(r[4] - b2) <= 1e-14 * abs(b2)
