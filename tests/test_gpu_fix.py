"""Fixed-point products of complex128 fields (csrc/fix.cuh): B^2, its gradient
and F_munu against the same entry points on a workspace that only holds the
FP64 intermediates, at the edges of the 32-site tiles and 128-site blocks, and
the fields that have to stay in FP64 (not unitary, not finite, close to 1).

Bounds.  A fixed-point product is off by 2e-18 an entry and an FP64 one by
2^-53 of its largest partial sum; the gradient passes about 40 products and the
sums of 28 weighted leaves, so the two agree to a few times 40 2^-53 = 4e-15
of the gradient's norm; B^2 sums V squares of either sign of error: 1e-14."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

import oracle
from flue_gb300 import _lib, flow, generate
from flue_gb300.field import as_field

pytestmark = pytest.mark.gpu

ALIGN = 256


def _a(x):
    return (x + ALIGN - 1) // ALIGN * ALIGN


def _fp64_only_bytes(dims, nplanes, ndirs, force):
    """What the FP64 intermediates take: lines, K, line cotangents, partials."""
    v = int(np.prod(dims))
    t = _a(3 * ndirs * v * 144)
    t = _a(t + (nplanes * v * 80 if force else 0))
    t = _a(t + (3 * ndirs * v * 144 if force else 0))
    return _a(t + nplanes * ((v + 127) // 128) * 8)


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def _energy(field, planes, form, nbytes):
    nt, nx, ny, nz = field.dims
    p = np.ascontiguousarray(np.asarray(planes, dtype=np.int32).reshape(-1))
    ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    e = torch.empty(1, dtype=torch.float64, device="cuda")
    g = torch.empty((3, 3, 4, nz, ny, nx, nt), dtype=torch.complex128, device="cuda")
    d = field.descriptor()
    _lib.call("flue_loop5_energy_force", ctypes.byref(d), p.ctypes.data_as(ctypes.c_void_p), len(planes), _ptr(e),
              _ptr(g), form, _ptr(ws), nbytes, ctypes.c_void_p(0))
    torch.cuda.synchronize()
    return e.item(), g.cpu().numpy()


def _both(field, planes, form):
    dirs = len({d for p in planes for d in p})
    small = _fp64_only_bytes(field.dims, len(planes), dirs, True)
    full = max(_lib.load().flue_workspace_bytes(op, *field.dims, _lib.C128)
               for op in (_lib.OP_MAGNETIC_FORCE, _lib.OP_ENERGY_FORCE))
    assert full > small
    return _energy(field, planes, form, full), _energy(field, planes, form, small)


B2 = ((3, 2), (2, 4), (4, 3))
ALL = ((1, 2), (1, 3), (1, 4), (2, 3), (2, 4), (3, 4))


# 31, 32, 33, 127, 128, 129 sites among the volumes; extents down to 1 and 2
@pytest.mark.parametrize("dims", [(31, 1, 1, 1), (4, 2, 2, 2), (3, 11, 1, 1), (127, 1, 1, 1), (8, 4, 2, 2), (43, 3, 1, 1),
                                  (5, 3, 4, 7), (16, 8, 8, 8)])
@pytest.mark.parametrize("planes", [B2, ALL, ((1, 4),)])
@pytest.mark.parametrize("eps", [0.0, 0.1, 0.4])
def test_fixed_point_against_fp64(dims, planes, eps):
    u = generate.haar_field(dims, 5) if eps == 0.0 else generate.random_field(dims, eps, 5)
    f = as_field(u)
    for form in (_lib.FORCE_LIE, _lib.FORCE_EUCLID):
        (e1, g1), (e0, g0) = _both(f, planes, form)
        assert abs(e1 - e0) <= 1e-14 * abs(e0) + 1e-28
        # (extents of 1 and 2 make some gradients vanish up to rounding)
        scale = max(np.linalg.norm(g0), np.sqrt(g0.size) * 1e-3 / np.prod(dims))
        assert np.linalg.norm(g1 - g0) <= 8e-15 * scale


@pytest.mark.parametrize("change", ["scaled", "nan", "inf", "not_orthogonal", "cold", "near_cold", "huge"])
def test_fields_that_stay_in_fp64(change):
    dims = (7, 5, 4, 3)
    u = np.array(generate.random_field(dims, 0.3, 9))
    if change == "scaled":
        u[3, 2, 1, 0, 2] *= 1.01
    elif change in ("nan", "inf"):
        u[3, 2, 1, 0, 2, 1, 1] = np.nan if change == "nan" else np.inf
    elif change == "not_orthogonal":
        u[0, 0, 0, 0, 1, 1] = u[0, 0, 0, 0, 1, 0]
    elif change == "huge":
        u[3, 2, 1, 0, 3, 0, 0] = 1e300
    elif change == "cold":
        u = np.array(generate.cold_field(dims))
    else:
        u = np.array(generate.random_field(dims, 1e-3, 9))
    (e1, g1), (e0, g0) = _both(as_field(np.asfortranarray(u)), B2, _lib.FORCE_LIE)
    assert np.array_equal(e1, e0, equal_nan=True) and np.array_equal(g1, g0, equal_nan=True)


def test_rough_fields_take_fixed_point():
    f = as_field(generate.random_field((8, 6, 4, 4), 0.3, 2))
    (_, g1), (_, g0) = _both(f, B2, _lib.FORCE_LIE)
    assert not np.array_equal(g1, g0)


def test_gauge_fixed_time_links_take_fixed_point():
    """A quarter of the links at 1 (temporal gauge) does not shut the gate."""
    u = np.array(generate.random_field((8, 6, 4, 4), 0.3, 2))
    u[..., 0, :, :] = np.eye(3)
    f = as_field(np.asfortranarray(u))
    (e1, g1), (e0, g0) = _both(f, ALL, _lib.FORCE_LIE)
    assert not np.array_equal(g1, g0)
    assert np.linalg.norm(g1 - g0) <= 8e-15 * np.linalg.norm(g0)
    assert abs(e1 - oracle.loop5_energy(u, ALL)) <= 1e-12 * abs(e0)


def _flow_step(field, eps, nbytes):
    f = field.clone()
    ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    d = f.descriptor()
    _lib.call("flue_wflow_step", ctypes.byref(d), eps, _ptr(ws), nbytes, ctypes.c_void_p(0))
    torch.cuda.synchronize()
    return f.to_numpy()


def _flow_both(u, eps):
    f = as_field(np.asfortranarray(u))
    v = f.volume
    small = _a(36 * v * 16) + _a(36 * v * 8) + _a((v + 127) // 128 * 4 * 8)
    full = _lib.load().flue_workspace_bytes(_lib.OP_WFLOW, *f.dims, _lib.C128)
    assert full > small
    return _flow_step(f, eps, full), _flow_step(f, eps, small)


# Entries are of order 1 and rounded to FP64 on both sides (2^-53 each); the
# FP64 step adds the rounding of its three exponentials: 8 x 2^-53.  eps = 0.1
# takes |X| past 1/2 (X is halved); 0.13 is past the fixed-point factors' range.
@pytest.mark.parametrize("dims", [(31, 1, 1, 1), (2, 2, 2, 2), (3, 11, 1, 1), (43, 3, 1, 1), (5, 3, 4, 7), (8, 4, 4, 8)])
@pytest.mark.parametrize("eps", [0.01, 0.1, 0.13])
@pytest.mark.parametrize("field_eps", [0.0, 0.3])
def test_flow_step_against_fp64(dims, eps, field_eps):
    u = generate.haar_field(dims, 5) if field_eps == 0.0 else generate.random_field(dims, field_eps, 5)
    a, b = _flow_both(u, eps)
    assert np.abs(a - b).max() <= 8 * 2.0**-53
    if eps > 0.12:
        assert np.array_equal(a, b)


@pytest.mark.parametrize("change", ["scaled", "nan", "cold"])
def test_flow_stays_in_fp64(change):
    dims = (7, 5, 4, 3)
    u = np.array(generate.cold_field(dims) if change == "cold" else generate.random_field(dims, 0.3, 9))
    if change == "scaled":
        u[3, 2, 1, 0, 2] *= 1.01
    elif change == "nan":
        u[3, 2, 1, 0, 2, 1, 1] = np.nan
    a, b = _flow_both(u, 0.02)
    assert np.array_equal(a, b, equal_nan=True)


def _loops(field, small):
    """Plaquette sums of the four kinds of range, the Polyakov sums and a W
    table on workspaces of the FP64 kernels' size, or of the full size."""
    L, st = _lib.load(), ctypes.c_void_p(0)
    nt, nx, ny, nz = field.dims
    v, d = field.volume, field.descriptor()
    out = torch.zeros(32, dtype=torch.float64, device="cuda")

    def ws(full, fp64):
        n = fp64 if small else full
        assert full > fp64
        return torch.empty(n, dtype=torch.uint8, device="cuda"), n

    w, n = ws(L.flue_workspace_bytes(_lib.OP_PLAQUETTE, *field.dims, _lib.C128), _a(min(1024, (v + 255) // 256) * 8))
    for k, r in enumerate(((1, 4, 4), (2, 4, 4), (1, 1, 4), (2, 2, 3), (3, 4, 4))):
        _lib.call("flue_plaquette", ctypes.byref(d), *r, ctypes.c_void_p(out.data_ptr() + 8 * k), _ptr(w), n, st)
    w, n = ws(L.flue_workspace_bytes(_lib.OP_POLYAKOV, *field.dims, _lib.C128),
              _a(min(1024, (v // nt + 7) // 8) * 16))
    _lib.call("flue_polyakov", ctypes.byref(d), ctypes.c_void_p(out.data_ptr() + 8 * 5), _ptr(w), n, st)
    nsb = (v + 127) // 128
    w, n = ws(L.flue_wmunu_table_bytes(*field.dims, _lib.C128, 5, 3), _a(8 * v * 144) + _a(15 * nsb * 8))
    _lib.call("flue_wmunu_table", ctypes.byref(d), 3, 1, 5, 3, ctypes.c_void_p(out.data_ptr() + 8 * 7), _ptr(w), n, st)
    torch.cuda.synchronize()
    return out.cpu().numpy()


# Sums over V sites of traces of order 1: each side rounds a trace to 2^-53 and
# a sum of n terms to at most n 2^-53 of its largest partial sum; 1e-13 a term.
@pytest.mark.parametrize("dims", [(31, 1, 1, 1), (4, 2, 2, 2), (3, 11, 1, 1), (127, 1, 1, 1), (129, 2, 1, 1), (16, 3, 3, 3),
                                  (33, 3, 4, 5), (1, 6, 5, 4), (64, 8, 4, 4), (1024, 2, 1, 1)])
@pytest.mark.parametrize("eps", [0.0, 0.1, 0.4])
def test_loops_against_fp64(dims, eps):
    u = generate.haar_field(dims, 5) if eps == 0.0 else generate.random_field(dims, eps, 5)
    f = as_field(u)
    a, b = _loops(f, False), _loops(f, True)
    v = f.volume
    terms = np.array([6 * v, 3 * v, 3 * v, v, v, v / dims[0], v / dims[0]] + [1.0] * 25)
    assert (np.abs(a - b) <= 1e-13 * np.maximum(terms, 1)).all()


@pytest.mark.parametrize("change", ["scaled", "nan", "cold", "near_cold"])
def test_loops_stay_in_fp64(change):
    dims = (18, 5, 4, 3)
    if change == "cold":
        u = np.array(generate.cold_field(dims))
    else:
        u = np.array(generate.random_field(dims, 1e-3 if change == "near_cold" else 0.3, 9))
    if change == "scaled":
        u[3, 2, 1, 0] *= 1.01
    elif change == "nan":
        u[3, 2, 1, 0, :, 1, 1] = np.nan
    f = as_field(np.asfortranarray(u))
    a, b = _loops(f, False), _loops(f, True)
    # (the FP64 partial sums are grouped by other blocks)
    assert np.allclose(a, b, rtol=1e-14, atol=1e-12, equal_nan=True)


def test_ensemble_mixes_fixed_point_and_fp64_fields():
    """Fields that pass the gate and fields that do not, in one evaluation: each
    as the device entry points give it (their own gate decides the same way);
    tolerance as in test_loops_against_fp64 and test_fixed_point_against_fp64."""
    from flue_gb300 import gluonCalc as G
    from flue_gb300.ensemble import Ensemble

    us = [np.array(generate.random_field(d, 0.3, 3 + i)) for i, d in enumerate([(8, 6, 5, 4), (5, 3, 3, 3), (17, 4, 4, 4)])]
    us.append(np.array(generate.cold_field((6, 4, 4, 4))))
    bad = us[0].copy()
    bad[3, 2, 1, 0] *= 1.01
    us.append(bad)
    fields = [as_field(np.asfortranarray(u)) for u in us]
    for block in (128, 256):
        e = Ensemble(fields, block=block)
        rows = e.run()
        assert np.array_equal(rows, e.run())
        for f, r in zip(fields, rows):
            v = f.volume
            assert abs(r[0] - G.plaquette(f, 2, 4, 4)[0]) <= 1e-13 * 3 * v
            assert abs(r[1] - G.plaquette(f, 1, 1, 4)[0]) <= 1e-13 * 3 * v
            re, _, _, im = G.polyakov(f, return_imag=True)
            assert abs(r[2] - re) <= 1e-13 * v and abs(r[3] - im) <= 1e-13 * v
            b2 = G.magnetic(f)
            assert abs(r[4] - b2) <= 1e-14 * abs(b2) + 1e-28


def _fix_su3_64(u):
    """FixSU3Matrix of every link in complex128; u: (..., 3, 3)."""
    r0 = u[..., 0, :] / np.linalg.norm(u[..., 0, :], axis=-1, keepdims=True)
    r1 = u[..., 1, :] - r0 * np.sum(r0.conj() * u[..., 1, :], axis=-1, keepdims=True)
    r1 = r1 / np.linalg.norm(r1, axis=-1, keepdims=True)
    return np.stack([r0, r1, np.cross(r0, r1).conj()], axis=-2)


# Rows of length^2 within 1/2 of 1 take sums of bounded size, others sums of any
# size: both sides of the two limits, and rows of different length.  The step is
# so short that it only reunitarises, three times.  Of an entry below 1 each time
# rounds at most 2^-24, the entries of row 2 once more by the errors of rows 0
# and 1 (two vectors of six such errors, 5 2^-24): 16 2^-24 in all.
@pytest.mark.parametrize("rows", [(1.0, 1.0), (1.22, 1.0), (1.23, 1.0), (0.71, 1.0), (0.70, 1.0), (1.0, 1.22), (1.0, 1.23),
                                  (1.0, 0.71), (1.0, 0.70), (3.0, 0.2)])
def test_fp32_flow_reunitarises(rows):
    u = generate.random_field((5, 3, 2, 3), 0.4, 11)
    v = (u * np.array([rows[0], rows[1], 1.0])[:, None]).astype(np.complex64)
    f = as_field(v, "c64")
    ref = _fix_su3_64(v.astype(np.complex128))
    flow.wflow_step(f, 1e-30)
    got = f.to_numpy()
    assert np.abs(got.astype(np.complex128) - ref).max() <= 16 * 2.0**-24
