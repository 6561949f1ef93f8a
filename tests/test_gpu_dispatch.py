"""Which kernels calls take: CTAs of a right-hand side, instances of a batch on clusters."""
import luna_b200_loader  # registers the luna.jl_b200 package

luna_b200_loader.load()

import numpy as np
import pytest

from luna_b200 import _lib
from luna_b200 import plan as P
from luna_b200.interface import prop_capillary_args, prop_gnlse_args
from oracle import uppe

pytestmark = pytest.mark.gpu


def _capillary(trange, pressure=1.0, gas="Ar"):
    return prop_capillary_args(125e-6, 0.001, gas, pressure, λ0=800e-9, τfwhm=10e-15, energy=80e-6, λlims=(150e-9, 4e-6),
                               trange=trange, saveN=2)


def _gnlse(trange):
    return prop_gnlse_args(0.11, 0.001, [0.0, 0.0, -11.83e-27, 8.1e-41], λ0=835e-9, τfwhm=50e-15, power=10e3,
                           pulseshape="sech", λlims=(500e-9, 2400e-9), trange=trange, saveN=2)


def _ctas(p, precision=_lib.PREC_FP64):
    plan = P.Plan.from_transform(p.transform, precision)
    return _lib.load().luna_b200_plan_rhs_ctas(plan.handle)


@pytest.mark.parametrize("make,No,ctas", [(lambda: _capillary(0.12e-12), 2048, 1), (lambda: _capillary(0.25e-12), 4096, 4),
                                          (lambda: _capillary(0.5e-12), 8192, 8), (lambda: _capillary(1e-12), 16384, 16),
                                          (lambda: _capillary(2e-12), 32768, 16), (lambda: _capillary(2e-12, gas="H2"), 32768, 16),
                                          (lambda: _gnlse(1e-12), 1024, 1), (lambda: _gnlse(3e-12), 2048, 4),
                                          (lambda: _gnlse(6e-12), 4096, 8), (lambda: _gnlse(12.5e-12), 8192, 16),
                                          (lambda: _capillary(1e-12, (2.0, 0.2)), 16384, 1)])
def test_right_hand_sides_take_the_cluster_of_their_size(make, No, ctas):
    p = make()
    assert p.grid.No == No and _ctas(p) == ctas
    assert _ctas(p, _lib.PREC_MIXED) == 1


@pytest.mark.parametrize("make,precision,on", [(lambda: _capillary(0.25e-12), _lib.PREC_FP64, 0), (lambda: _capillary(0.5e-12), _lib.PREC_FP64, 1),
                                               (lambda: _capillary(2e-12, gas="H2"), _lib.PREC_FP64, 1), (lambda: _gnlse(3e-12), _lib.PREC_FP64, 0),
                                               (lambda: _gnlse(6e-12), _lib.PREC_FP64, 1), (lambda: _capillary(0.5e-12), _lib.PREC_MIXED, 0),
                                               (lambda: _capillary(1e-12), _lib.PREC_MIXED, 1), (lambda: _gnlse(12.5e-12), _lib.PREC_MIXED, 0),
                                               (lambda: _capillary(1e-12, (2.0, 0.2)), _lib.PREC_FP64, 0)])
def test_solves_from_the_smallest_grids_that_go_to_clusters(make, precision, on):
    """Real grids from 8192 points (16384 in mixed precision) and envelope grids from 4096 (full
    precision alone); no pressure gradients. NO_DIST keeps all on one CTA."""
    p = make()
    for flags, expect in ((0, on), (_lib.SOLVE_NO_DIST | _lib.SOLVE_NO_CLUSTERS, 0)):
        b = P.Batch([P.Plan.from_transform(p.transform, precision)], 2, np.array([0.0, p.grid.zmax]), flags=flags)
        assert b.info()[1:] == (expect, expect)


@pytest.mark.parametrize("make,No", [(lambda: _capillary(0.06e-12), 1024), (lambda: _capillary(0.12e-12, gas="H2"), 2048),
                                     (lambda: _capillary(0.25e-12), 4096), (lambda: _gnlse(1e-12), 1024)])
def test_smallest_mixed_right_hand_sides(make, No):
    """Sub-transforms of 512 and 1024 points in radix-2 passes, the next size in radix 4; the bound is the
    parity tests' for mixed precision."""
    p = make()
    assert p.grid.No == No
    E = p.Eω * np.exp(1j * 0.2 * np.random.default_rng(5).standard_normal(len(p.Eω)))
    nl = P.Plan.from_transform(p.transform, _lib.PREC_MIXED).rhs(np.zeros_like(E), E)
    ref = uppe.trans_mode_avg(p.transform, E, 0.0)
    assert np.linalg.norm(nl - ref) <= 1e-5 * np.linalg.norm(ref)
