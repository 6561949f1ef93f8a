"""What several objects and threads of one process share: kernel attributes, kept device memory."""
import ctypes
import threading
import time

import luna_b200_loader  # registers the luna.jl_b200 package

luna_b200_loader.load()

import numpy as np
import pytest

from luna_b200 import _lib
from luna_b200 import plan as P
from luna_b200.interface import prop_capillary_args

pytestmark = pytest.mark.gpu


def _capillary(trange, gas="Ar", flength=0.001):
    return prop_capillary_args(125e-6, flength, gas, 1.0, λ0=800e-9, τfwhm=10e-15, energy=80e-6, λlims=(150e-9, 4e-6),
                               trange=trange, saveN=2)


def _batch(p, precision, flags):
    b = P.Batch([P.Plan.from_transform(p.transform, precision)], 2, np.array([0.0, p.grid.zmax]), flags=flags)
    b.upload([p.linop], [p.Eω], [0.0], [1e-4], [p.grid.zmax])
    return b


@pytest.mark.parametrize("precision,flags,gas", [(_lib.PREC_FP64, _lib.SOLVE_NO_DIST, "Ar"), (_lib.PREC_FP64, 0, "Ar"),
                                                 (_lib.PREC_MIXED, _lib.SOLVE_NO_DIST | _lib.SOLVE_NO_CLUSTERS, "Ar"),
                                                 (_lib.PREC_MIXED, _lib.SOLVE_NO_DIST, "H2")])
def test_a_small_batch_created_between_leaves_a_large_one_as_it_was(precision, flags, gas):
    """Create a batch of a large grid, then one of a small grid, then run the large one: on single
    CTAs, on clusters, and on clusters with a Raman response apart."""
    large, small = _capillary(1e-12, gas), _capillary(0.06e-12, gas)
    a = _batch(large, precision, flags)
    b = _batch(small, precision, flags)
    a.run()
    first = a.results()[0]
    b.run()
    assert first.status == b.results()[0].status == 0
    a.run()
    assert np.array_equal(a.results()[0].y, first.y)
