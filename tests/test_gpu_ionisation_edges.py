"""Ionisation rates at the edges of their range, in the kernels of one CTA (the allocation-free entry
point) and of clusters of 4, 8 and 16 (rhs_device), against the FP64 oracle.
"""
import copy
import ctypes

import luna_b200_loader  # registers the luna.jl_b200 package

luna_b200_loader.load()

import numpy as np
import pytest

from luna_b200 import _lib
from luna_b200 import plan as P
from luna_b200.interface import prop_capillary_args
from oracle import uppe

pytestmark = pytest.mark.gpu

# one CTA for both entry points; one CTA against clusters of 4, 8 and 16; four samples a thread
TRANGES = [0.12e-12, 0.25e-12, 0.5e-12, 1e-12, 2e-12]


def _problem(trange, **kw):
    return prop_capillary_args(125e-6, 0.05, "Ar", 1.0, λ0=800e-9, τfwhm=10e-15, energy=80e-6, λlims=(150e-9, 4e-6),
                               trange=trange, saveN=5, **kw)


def _rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def _rhs(t, E):
    """The right-hand side by rhs (clusters from 4096 points) and by rhs_device_noalloc (one CTA), with
    their statuses."""
    torch = pytest.importorskip("torch")
    lib, plan = _lib.load(), P.Plan.from_transform(t)
    a = np.zeros_like(E)
    rc = lib.luna_b200_rhs(plan.handle, _lib.dptr(a.view(np.float64)), _lib.dptr(E.view(np.float64)), 0.0)
    d = torch.from_numpy(E.view(np.float64).copy()).cuda()
    o, st = torch.zeros_like(d), torch.full((1,), -1, dtype=torch.int32, device="cuda")
    _lib.check(lib.luna_b200_rhs_device_noalloc(plan.handle, ctypes.c_void_p(o.data_ptr()), ctypes.c_void_p(d.data_ptr()), 0.0,
                                                None, ctypes.c_void_p(st.data_ptr())))
    torch.cuda.synchronize()
    return (rc, a), (int(st.item()), o.cpu().numpy().view(np.complex128))


@pytest.mark.parametrize("trange", TRANGES)
def test_table_that_begins_at_a_zero_field(trange, monkeypatch):
    """A constant rate from E = 0 on, on a field whose every fourth sample is an exact zero (1 +
    cos(pi n / 2) on the oversampled grid): those samples ionise like the others."""
    p = _problem(trange)
    plasma = next(q for q in p.transform.resp if q.kind == "plasma")
    r = plasma.ratefunc = copy.copy(plasma.ratefunc)  # (tables are shared between problems)
    n, top = len(r.x), r.x[-1]
    r.x, r.y, r.D = np.linspace(0.0, top, n), np.full(n, np.log(1e13)), np.zeros(n)
    r.Emin = 0.0
    E = np.zeros(len(p.Eω), dtype=complex)
    E[0], E[-1] = 1.0, 0.5
    Et = uppe.to_time(p.grid, E)
    assert np.sum(Et == 0) == p.grid.No // 4
    E *= 1e-10 * top / Et.max()
    ref = uppe.trans_mode_avg(p.transform, E, 0.0)
    # what one rounding of each sample of the polarisation does to the result (a constant field's is far
    # from the window's frequencies), times the 3 sqrt(No) < 1000 of three running sums
    pol, rng = uppe.et_to_pt, np.random.default_rng(0)
    monkeypatch.setattr(uppe, "et_to_pt", lambda *a: pol(*a) * (1 + 2.0 ** -52 * rng.standard_normal(p.grid.No)))
    tol = 1000 * _rel(uppe.trans_mode_avg(p.transform, E, 0.0), ref)
    for rc, nl in _rhs(p.transform, E):
        assert rc == 0 and _rel(nl, ref) < tol


@pytest.mark.parametrize("trange", TRANGES)
def test_nan_field_gives_nan_and_field_above_the_table_is_reported(trange):
    p = _problem(trange)
    E = p.Eω.copy()
    E[len(E) // 3] = np.nan
    for rc, nl in _rhs(p.transform, E):
        assert rc == _lib.LUNA_OK and np.all(np.isnan(nl))
    for rc, _ in _rhs(p.transform, 50.0 * p.Eω):
        assert rc == _lib.LUNA_FIELD_ABOVE_EMAX


@pytest.mark.parametrize("trange", TRANGES)
def test_adk_rates_follow_the_oracle(trange):
    """The logarithmic form of the ADK rate against the power, from the threshold to ionisation of a
    visible part of the gas; 1e-11 as the parity tests have it for right-hand sides with plasma."""
    p = _problem(trange, plasma="ADK")
    assert next(q for q in p.transform.resp if q.kind == "plasma").ratefunc.kind == "adk"
    E = p.Eω * np.exp(1j * 0.2 * np.random.default_rng(3).standard_normal(len(p.Eω)))
    for f in (0.3, 1.0, 2.0):
        ref = uppe.trans_mode_avg(p.transform, f * E, 0.0)
        for rc, nl in _rhs(p.transform, f * E):
            assert rc == 0 and _rel(nl, ref) < 1e-11
