"""The modal transform on several clusters (FP64)."""
import ctypes

import luna_b200_loader  # registers the luna.jl_b200 package

luna_b200_loader.load()

import numpy as np
import pytest

from luna_b200 import _lib, fields, ionisation, modal, modes, raman
from luna_b200 import physdata as pd
from luna_b200.grid import RealGrid
from luna_b200.nonlinear import Kerr_field, PlasmaCumtrapz, RamanPolarField
from oracle import uppe

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


def _case(nm, trange, plasma=False, gas="Ar"):
    ms = tuple(modes.MarcatiliMode(50e-6, gas, 1.0, n=1, m=m + 1, loss=False) for m in range(nm))
    grid = RealGrid(1e-3, 800e-9, (160e-9, 3000e-9), trange)
    resp = [Kerr_field(pd.gamma3_gas(gas))]
    if gas == "H2":
        resp.append(RamanPolarField(grid.to, raman.raman_response(grid.to, gas)))
    if plasma:
        resp.append(PlasmaCumtrapz(grid.to, grid.to, ionisation.ionrate_PPTaccel("Ar", 800e-9, N=2 ** 12),
                                   pd.ionisation_potential("Ar")))
    E, t = modal.setup_modal(grid, pd.density(gas, 1.0), resp, fields.GaussField(800e-9, 10e-15, energy=20e-6), ms, "y")
    for m in range(1, nm):
        E[:, m] = 0.3 / m * E[:, 0]
    return grid, E, t, modal.make_const_linop_modes(grid, ms, 800e-9)


@pytest.mark.parametrize("nm,plasma", [(2, False), (3, True)])
def test_a_wait_that_runs_out_is_reported(nm, plasma):
    """Clusters that do not wait for one another at all: every entry point says so, and the plan works
    again when they do."""
    torch = pytest.importorskip("torch")
    grid, E, t, linop = _case(nm, 0.4e-12, plasma)
    lib, plan = _lib.load(), t.plan()
    ref = plan.rhs(np.zeros_like(E), E).copy()
    d = torch.from_numpy(np.ascontiguousarray(E.T).view(np.float64)).cuda()
    o = torch.zeros_like(d)
    assert lib.luna_b200_modal_set_wait(plan._h, 0) == 0
    with pytest.raises(_lib.LunaError) as e:
        plan.rhs(np.zeros_like(E), E)
    assert e.value.code == _lib.LUNA_WAIT_TIMEOUT
    _lib.check(lib.luna_b200_modal_rhs_device(plan._h, ctypes.c_void_p(o.data_ptr()), ctypes.c_void_p(d.data_ptr()), 0.0, None))
    torch.cuda.synchronize()
    assert o.isnan().all()
    with pytest.raises(_lib.LunaError) as e:
        plan.solve(linop, E, 0.0, 1e-5, 1e-4, saveN=2)
    assert e.value.code == _lib.LUNA_WAIT_TIMEOUT
    assert lib.luna_b200_modal_set_wait(plan._h, 1 << 24) == 0
    assert np.array_equal(plan.rhs(np.zeros_like(E), E), ref)
    assert plan.solve(linop, E, 0.0, 1e-5, 1e-4, saveN=2).status == 0


@pytest.mark.parametrize("nm,trange,plasma,gas", [(3, 0.2e-12, True, "Ar"), (1, 0.1e-12, True, "Ar"), (5, 0.4e-12, True, "Ar"), (2, 0.2e-12, False, "H2"),
                                                  (2, 1e-12, False, "H2"), (9, 0.2e-12, False, "H2")])
def test_several_modes_with_plasma_or_raman(nm, trange, plasma, gas):
    """Levels whose nodes the clusters share, fewer, as many and more modes than clusters, clusters of 4 to
    16; 1e-11 as the modal tests have it with plasma or Raman."""
    grid, E, t, _ = _case(nm, trange, plasma, gas)
    nl = np.zeros_like(E)
    t(nl, E, 0.0)
    assert _rel(nl, uppe.trans_modal(t, E, 0.0)) < 1e-11
    assert t.plan().nevals == t.oracle_nevals
