"""Scratch of the Wilson flow: no more than the FP64 step's where a lattice fills the
32-site tiles, and a step that finds no memory for more runs in FP64."""
import numpy as np
import pytest

from flue_gb300 import _lib, generate


@pytest.mark.parametrize("dims", [(64, 32, 32, 32), (192, 96, 96, 96), (8, 4, 4, 4), (96, 5, 7, 3)])
def test_workspace_is_that_of_the_fp64_step(dims):
    n = _lib.load().flue_workspace_bytes
    assert n(_lib.OP_WFLOW, *dims, _lib.C128) <= n(_lib.OP_WFLOW, *dims, _lib.C64) + 256


@pytest.mark.gpu
def test_step_without_memory_for_fixed_point(monkeypatch):
    torch = pytest.importorskip("torch")
    from flue_gb300 import field, flow
    from tests.test_gpu_fix import _flow_both

    dims = (5, 3, 5, 7)
    u = generate.random_field(dims, 0.3, 4)
    fixed, fp64 = _flow_both(u, 0.02)
    asked = []

    def empty(n, **kw):
        asked.append(n)
        if len(asked) == 1:
            raise torch.cuda.OutOfMemoryError("no memory")
        return torch.empty(n, **kw)

    f = field.as_field(np.asfortranarray(u))
    field.Workspace.release()
    monkeypatch.setattr(field, "torch", type("T", (), {"empty": staticmethod(empty), "__getattr__": lambda s, k: getattr(torch, k)})())
    got = flow.wflow_step(f, 0.02).storage.permute(6, 5, 4, 3, 2, 1, 0).cpu().numpy()
    assert asked[1] < asked[0]
    assert np.array_equal(got, fp64) and not np.array_equal(got, fixed)
