"""The host-buffer gradient call and the pages of its output array: fresh from the
allocator, already written, or pinned."""
import ctypes
import mmap
import time

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from flue_gb300 import _lib, generate

pytestmark = pytest.mark.gpu

PRECS = {"c128": _lib.C128, "r12": _lib.R12}


def _force(u, grad, prec):
    b = ctypes.c_double()
    p = ctypes.c_void_p(grad if isinstance(grad, int) else grad.ctypes.data)
    _lib.call("flue_magnetic_force_c", u.ctypes.data_as(ctypes.c_void_p), _lib.C128, *u.shape[:4], PRECS[prec],
              _lib.FORCE_LIE, ctypes.byref(b), p)
    return b.value


# 8.4 MB and 17 MB: two and four threads map it; it starts and ends inside a page,
# and the bytes around it stay as they are.
@pytest.mark.parametrize("dims", [(16, 12, 10, 8), (13, 16, 12, 12)])
@pytest.mark.parametrize("prec", ["c128", "r12"])
def test_fresh_pageable_gradient(dims, prec):
    u = np.asfortranarray(generate.random_field(dims, 0.3, 3))
    pinned = torch.empty(u.size, dtype=torch.complex128, pin_memory=True).numpy()
    pinned[:] = np.nan
    e0 = _force(u, pinned, prec)
    assert np.isfinite(pinned).all()
    written = np.full(u.size, np.nan + 0j)
    assert _force(u, written, prec) == e0 and np.array_equal(written, pinned)
    off = 3 * 16
    m = mmap.mmap(-1, u.nbytes + 2 * mmap.PAGESIZE)
    base = ctypes.addressof(ctypes.c_char.from_buffer(m))
    assert _force(u, base + off, prec) == e0
    got = np.frombuffer(m, dtype=np.complex128, count=u.size, offset=off)
    assert np.array_equal(got, pinned)
    assert m[:off] == bytes(off) and not any(m[off + u.nbytes:])


# An array whose pages are there costs what it cost before they were looked after:
# a pinned one's time within the noise of calls this short.
@pytest.mark.parametrize("dims", [(16, 8, 8, 8), (48, 24, 24, 24)])
def test_written_pageable_gradient_costs_no_mapping(dims):
    f = torch.randn((3, 3, 4) + dims[:0:-1] + dims[:1], dtype=torch.complex128, device="cuda")
    from flue_gb300.field import GaugeField

    u = GaugeField(f, dims, "c128").reunitarise_().to_numpy()
    grads = {"pinned": torch.zeros(u.size, dtype=torch.complex128, pin_memory=True).numpy(),
             "written": np.full(u.size, 1.0 + 0j)}
    tries = []
    for _ in range(3):  # another user of the machine may hold one up
        times = {k: [] for k in grads}
        for _ in range(40):
            for k, g in grads.items():
                t = time.perf_counter()
                _force(u, g, "r12")
                times[k].append(time.perf_counter() - t)
        tries.append({k: np.median(v[8:]) for k, v in times.items()})
        if tries[-1]["written"] <= 1.2 * tries[-1]["pinned"]:
            break
    else:
        raise AssertionError(tries)
