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


# ------------------------------------------------------------------ kept device memory
@pytest.mark.parametrize("mode", ["relaxed", "thread_local"])
@pytest.mark.parametrize("what", ["destroy", "create", "solve"])
def test_objects_come_and_go_beside_a_capture(mode, what):
    """Destroying or creating a plan and a whole solve, while the caller captures a right-hand side: in the
    capturing thread (relaxed mode) or another one."""
    torch = pytest.importorskip("torch")
    lib = _lib.load()
    p = _capillary(0.25e-12)
    plan = P.Plan.from_transform(p.transform)
    E = torch.from_numpy(p.Eω.view(np.float64).copy()).cuda()
    ref, out = torch.zeros_like(E), torch.zeros_like(E)
    rhs = lambda o: _lib.check(lib.luna_b200_rhs_device(plan.handle, ctypes.c_void_p(o.data_ptr()), ctypes.c_void_p(E.data_ptr()), 0.0,
                                                        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    solve = lambda: P.solve_precon(p.transform, p.linop, p.Eω, 0.0, 1e-4, p.grid.zmax, saveN=2, max_dt=1e-4).y
    rhs(ref)
    keep = {"other": P.Plan.from_transform(p.transform), "y": solve()}
    torch.cuda.synchronize()

    def act():
        if what == "destroy":
            keep["other"] = None
        elif what == "create":
            keep["other"] = P.Plan.from_transform(p.transform)
        else:
            keep["y2"] = solve()

    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode=mode):
        rhs(out)
        if mode == "relaxed":
            act()
        else:
            th = threading.Thread(target=act)
            th.start()
            th.join()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, ref)
    assert what != "solve" or np.array_equal(keep["y2"], keep["y"])


def test_giving_memory_back_does_not_wait_for_another_threads_batch():
    """A solve ends, gives its memory back, and another one begins and ends, while a third thread's batch
    of some seconds runs on one SM."""
    p, big = _capillary(0.25e-12), _capillary(2e-12)
    solve = lambda: P.solve_precon(p.transform, p.linop, p.Eω, 0.0, 1e-4, p.grid.zmax, saveN=2, max_dt=1e-4).y
    long = P.Batch([P.Plan.from_transform(big.transform)], 2, np.array([0.0, big.grid.zmax]), flags=_lib.SOLVE_NO_DIST,
                   max_steps=2000, max_dt=1e-8)  # 2000 steps of 1.5 ms
    long.upload([big.linop], [big.Eω], [0.0], [1e-8], [big.grid.zmax])
    ref = solve()
    out = []

    def work():
        for _ in range(3):
            out.append(solve())

    runner = threading.Thread(target=long.run)
    runner.start()
    time.sleep(0.1)
    th = [threading.Thread(target=work) for _ in range(2)]
    [t.start() for t in th]
    [t.join() for t in th]
    beside = runner.is_alive()
    runner.join()
    assert beside, "the solves ended after the batch"
    assert len(out) == 6 and all(np.array_equal(y, ref) for y in out)
    assert long.download()[2][0].steps == 2000
