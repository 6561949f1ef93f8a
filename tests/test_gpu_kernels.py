"""Kernels chosen by size: each choice at the edges of its range against the FP64 oracle, a matrix
product, or the general kernel.

Tolerances: right-hand sides as in the parity tests (1e-12, with plasma or Raman 1e-11: the
transforms and running integrals round in another order); matrix products of K terms in FP64 within
K 2^-52 of the sum of magnitudes; BF16 products accumulated in FP32, 16 terms at a time and
truncated, K/16 2^-23 / 2 (at least 1e-5); BF16 results 5e-3 (2^-9 a rounding, two roundings); results of the same operations in the same order are equal.
"""
import ctypes
import threading

import luna_b200_loader  # registers the luna.jl_b200 package

luna_b200_loader.load()

import numpy as np
import pytest

from luna_b200 import _lib, fields, modal, modes
from luna_b200 import physdata as pd
from luna_b200 import plan as P
from luna_b200.grid import RealGrid
from luna_b200.interface import prop_capillary_args, prop_gnlse_args
from luna_b200.nonlinear import Kerr_field
from luna_b200.radial import prop_radial_args
from luna_b200.radial_plan import RadialPlan
from oracle import uppe

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


def _capillary(gas, trange, flength=0.05):
    return prop_capillary_args(125e-6, flength, gas, 1.0, λ0=800e-9, τfwhm=10e-15, energy=80e-6,
                               λlims=(150e-9, 4e-6), trange=trange, saveN=5)


def _gnlse(trange, flength=0.002):
    return prop_gnlse_args(0.11, flength, [0.0, 0.0, -11.83e-27, 8.1e-41], λ0=835e-9, τfwhm=50e-15,
                           power=10e3, pulseshape="sech", λlims=(500e-9, 2400e-9), trange=trange, saveN=5)


def _perturbed(p):
    rng = np.random.default_rng(11)
    return p.Eω * np.exp(1j * 0.2 * rng.standard_normal(p.Eω.shape))


# ------------------------------------------------------------------ one right-hand side on a cluster
@pytest.mark.parametrize("gas,trange", [(g, t) for g in ("Ar", "H2") for t in (0.12e-12, 0.25e-12, 0.5e-12, 1e-12, 2e-12)]
                         + [("Ar", 4e-12)])  # (a Raman response takes grids of up to 32768 points)
def test_rhs_on_every_cluster_size(gas, trange):
    """Real grids from 2048 points (one CTA) over clusters of 4, 8 and 16 to several samples a
    thread, with Kerr and plasma, and with Raman as well."""
    p = _capillary(gas, trange)
    E = _perturbed(p)
    nl = p.transform.plan().rhs(np.zeros_like(E), E)
    assert _rel(nl, uppe.trans_mode_avg(p.transform, E, 0.0)) < 1e-11


@pytest.mark.parametrize("trange", [1e-12, 3e-12, 6e-12, 12.5e-12, 50e-12])
def test_envelope_rhs_on_every_cluster_size(trange):
    p = _gnlse(trange)
    E = _perturbed(p)
    nl = p.transform.plan().rhs(np.zeros_like(E), E)
    assert _rel(nl, uppe.trans_mode_avg(p.transform, E, 0.0)) < 1e-11


@pytest.mark.parametrize("make", [lambda: _capillary("Ar", 0.25e-12), lambda: _capillary("H2", 0.5e-12),
                                  lambda: _gnlse(12.5e-12), lambda: _gnlse(50e-12)])
def test_cluster_solve_follows_the_oracle(make):
    """The smallest grids that go to clusters and envelope grids, on the oracle's step sequence."""
    p = make()
    ores = uppe.run(p.transform, p.grid, p.linop, p.Eω, saveN=3)
    replay = np.array(ores.steps_all, dtype=np.float64).ravel()
    r = P.solve_precon(p.transform, p.linop, p.Eω, 0.0, 1e-4, p.grid.zmax, saveN=3, replay=replay)
    for a, b in zip(r.Eω, ores.Eω):
        assert _rel(a, b) < 1e-10


def test_batch_on_clusters_and_single_ctas_agrees():
    """More instances than clusters run at one time, real and envelope: the shapes chosen by the
    work estimates against one CTA each, on the same step sequences."""
    probs = [_capillary("Ar", t, 0.01) for t in (0.25e-12, 0.5e-12, 1e-12) * 8] + [_gnlse(12.5e-12, 0.001)] * 4
    plans = [P.Plan.from_transform(p.transform) for p in probs]

    def run(shapes, logs=None):
        b = P.Batch(plans, 3, np.linspace(0, 1, 3), steplog_cap=200)
        if logs:
            for i, g in enumerate(logs):
                b.set_replay(i, g[:, [1, 3]].ravel())
        b.upload([p.linop for p in probs], [p.Eω for p in probs], [0.0] * len(probs), [1e-4] * len(probs),
                 [p.grid.zmax for p in probs], [np.linspace(0, p.grid.zmax, 3) for p in probs],
                 [p.grid.zmax / 4 for p in probs])
        b.set_shapes(shapes)
        b.set_priority([1.0] * len(probs))
        b.run()
        return b.results()

    ref = run([1] * len(probs))
    for r, q in zip(run([0] * len(probs), [r.steplog for r in ref]), ref):
        assert r.status == q.status == 0 and r.steps == q.steps
        assert _rel(r.Eω[-1], q.Eω[-1]) < 1e-10


# ------------------------------------------------------------------ radial products
@pytest.mark.parametrize("N,trange", [(31, 0.2e-12), (33, 0.2e-12), (64, 0.2e-12), (65, 0.2e-12), (200, 0.5e-12)])
def test_qdht_products_in_both_tiles(N, trange):
    torch = pytest.importorskip("torch")
    p = prop_radial_args("Ar", 1.2, R=1e-3, N=N, flength=0.01, λ0=800e-9, λlims=(400e-9, 2000e-9), trange=trange,
                         τfwhm=20e-15, energy=20e-6, w0=40e-6, propz=0.0, plasma=False, saveN=3)
    plan = RadialPlan.from_transform(p.transform)
    rng = np.random.default_rng(N)
    X = rng.standard_normal((N, plan.Nw)) + 1j * rng.standard_normal((N, plan.Nw))
    dX = torch.from_numpy(X.view(np.float64).copy()).cuda()
    for fwd, M in ((0, p.transform.q.Mi), (1, p.transform.q.Mf)):
        dY = torch.zeros_like(dX)
        _lib.check(_lib.load().luna_b200_qdht_device(plan.handle, ctypes.c_void_p(dY.data_ptr()),
                                                     ctypes.c_void_p(dX.data_ptr()), fwd,
                                                     ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        Y = dY.cpu().numpy().view(np.complex128)
        bound = N * 2.0 ** -52 * (np.abs(M) @ (np.abs(X.real) + np.abs(X.imag)))
        assert np.all(np.abs(Y - M @ X) <= 2 * bound)


@pytest.mark.parametrize("N", [33, 90])
def test_radial_fused_steps_follow_the_oracle(N):
    """Rejected and accepted steps of the fused stages, for sizes that are no multiple of a tile."""
    p = prop_radial_args("Ar", 1.2, R=1e-3, N=N, flength=0.002, λ0=800e-9, λlims=(400e-9, 2000e-9), trange=0.2e-12,
                         τfwhm=20e-15, energy=20e-6, w0=40e-6, propz=0.0, plasma="PPT", saveN=3)
    ores = uppe.run(p.transform, p.grid, p.linop, p.Eω, saveN=3)
    replay = np.array(ores.steps_all, dtype=np.float64).ravel()
    r = RadialPlan.from_transform(p.transform).solve(p.linop, p.Eω, 0.0, 1e-4, p.grid.zmax, saveN=3, replay=replay)
    for a, b in zip(r.Eω, ores.Eω):
        assert _rel(a, b) < 1e-10


# ------------------------------------------------------------------ modal transform
@pytest.mark.parametrize("nm,trange", [(1, 0.1e-12), (1, 0.4e-12), (3, 0.4e-12), (5, 0.4e-12), (10, 0.4e-12)])
def test_modal_rhs_over_mode_counts(nm, trange):
    """One CTA a mode (small grids), one cluster, several clusters, more modes than are held in
    registers, and more modes than clusters of 16 are resident."""
    ms = tuple(modes.MarcatiliMode(50e-6, "Ar", 1.0, n=1, m=m + 1, loss=False) for m in range(nm))
    grid = RealGrid(1e-3, 800e-9, (160e-9, 3000e-9), trange)
    E, t = modal.setup_modal(grid, pd.density("Ar", 1.0), [Kerr_field(pd.gamma3_gas("Ar"))],
                             fields.GaussField(800e-9, 10e-15, energy=20e-6), ms, "y")
    for m in range(1, nm):
        E[:, m] = 0.3 / m * E[:, 0]
    nl = np.zeros_like(E)
    t(nl, E, 0.0)
    assert _rel(nl, uppe.trans_modal(t, E, 0.0)) < 1e-12
    assert t.plan().nevals == t.oracle_nevals


# ------------------------------------------------------------------ kept device memory
def test_solves_on_threads_share_kept_memory():
    """Buffers pass from solve to solve and thread to thread; every result is the first one's."""
    probs = [_capillary("Ar", 0.25e-12, 0.01), _gnlse(12.5e-12, 0.001)]
    solve = lambda p: P.solve_precon(p.transform, p.linop, p.Eω, 0.0, 1e-4, p.grid.zmax, saveN=3).Eω
    ref = [solve(p) for p in probs]
    out = {}

    def work(i):
        out[i] = [solve(probs[i]) for _ in range(4)]

    th = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    [t.start() for t in th]
    [t.join() for t in th]
    assert all(np.array_equal(e, ref[i]) for i in range(2) for e in out[i])


# ------------------------------------------------------------------ surrogate
def _sg():
    torch = pytest.importorskip("torch")
    from luna_b200 import surrogate as S
    return torch, S, S.load(), (lambda t: ctypes.c_void_p(t.data_ptr())), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


@pytest.mark.parametrize("B,K,N,members", [(128, 128, 128, 1), (128, 128, 384, 3), (384, 512, 256, 2), (2560, 128, 128, 8),
                                           (9600, 128, 256, 4), (19072, 256, 256, 1)])
def test_surrogate_products_in_every_tile(B, K, N, members):
    """64-, 128- and 256-wide tiles, fewer and more tiles than SMs, one to several K chunks, and the
    transposed operands of both backward products."""
    torch, S, lib, p, st = _sg()
    g = torch.Generator(device="cuda").manual_seed(B + N)
    bf = torch.bfloat16
    X = torch.randn(members, B, K, device="cuda", generator=g).to(bf)
    W = (torch.randn(members, N, K, device="cuda", generator=g) / K ** 0.5).to(bf)
    b = torch.randn(members, N, device="cuda", generator=g)
    dZ = torch.randn(members, B, N, device="cuda", generator=g).to(bf)
    Zp = torch.randn(members, B, K, device="cuda", generator=g).to(bf)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    Y, dX = torch.empty(members, B, N, device="cuda", dtype=bf), torch.empty(members, B, K, device="cuda", dtype=bf)
    dW, db = torch.empty(members, N, K, device="cuda"), torch.empty(members, N, device="cuda")
    assert lib.luna_sg_linear_fwd(p(X), B * K, p(W), p(b), B, K, N, 1, p(Y), None, None, members, p(err), st) == 0
    assert lib.luna_sg_linear_bwd_data(p(dZ), p(W), p(Zp), B, K, N, p(dX), members, p(err), st) == 0
    assert lib.luna_sg_linear_bwd_weight(p(dZ), p(X), B * K, B, K, N, p(dW), p(db), members, p(err), st) == 0
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    d = torch.float64
    z = torch.bmm(X.to(d), W.to(d).transpose(1, 2)) + b[:, None, :].to(d)
    s = torch.sigmoid(Zp.to(d))
    ref = lambda a, r: float((a.to(d) - r).norm() / r.norm())
    assert ref(Y, z * torch.sigmoid(z)) < 5e-3
    assert ref(dX, torch.bmm(dZ.to(d), W.to(d)) * (s * (1 + Zp.to(d) * (1 - s)))) < 5e-3
    assert ref(dW, torch.bmm(dZ.to(d).transpose(1, 2), X.to(d))) < max(1e-5, B / 16 * 2.0 ** -24)
    assert ref(db, dZ.to(d).sum(dim=1)) < 1e-5


@pytest.mark.parametrize("B,N,nspec,members", [(128, 128, 100, 1), (256, 256, 128, 3), (640, 768, 512, 4), (20480, 128, 0, 2)])
def test_last_layer_leaves_the_statistics_of_its_outputs(B, N, nspec, members):
    """The fused last layer against the layer and the statistics kernel: the same operations."""
    torch, S, lib, p, st = _sg()
    g = torch.Generator(device="cuda").manual_seed(B)
    K = 128
    X = torch.randn(members, B, K, device="cuda", generator=g).to(torch.bfloat16)
    W = (torch.randn(members, N, K, device="cuda", generator=g) / K ** 0.5).to(torch.bfloat16)
    b = torch.randn(members, N, device="cuda", generator=g)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    Y = torch.empty(members, B, N, device="cuda")
    m0, s0, m1, s1 = (torch.full(sh, 7.0, device="cuda") for sh in ((B, N), (B,), (B, N), (B,)))
    assert lib.luna_sg_linear_fwd(p(X), B * K, p(W), p(b), B, K, N, 0, None, None, p(Y), members, p(err), st) == 0
    assert lib.luna_sg_ensemble(p(Y), members, B, N, nspec, p(m0), p(s0), st) == 0
    assert lib.luna_sg_linear_ensemble(p(X), B * K, p(W), p(b), B, K, N, nspec, p(m1), p(s1), members, p(err), st) == 0
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    assert torch.equal(m0, m1) and torch.equal(s0, s1)


@pytest.mark.parametrize("n,chunk", [(1, 1 << 17), (129, 128), (1000, 300), (384, 128)])
def test_predict_in_chunks_equals_one_call(n, chunk):
    torch, S, lib, p, st = _sg()
    m = S.Ensemble(members=2, seed=3, batch=128)
    x = torch.randn(n, 8, device="cuda", generator=torch.Generator(device="cuda").manual_seed(n))
    pad = torch.cat([x, x[:1].expand((-n) % 128, -1)]) if n % 128 else x
    mu, sp = m.predict(pad.contiguous())
    a, b = S.predict(m, x, chunk)
    assert a.shape == (n, S.NOUT) and b.shape == (n,)
    assert torch.equal(a, mu[:n]) and torch.equal(b, sp[:n])
    for y, c in ((x, 0), (x, -128), (x[:0], chunk)):  # no chunk to take, nothing to return
        with pytest.raises((RuntimeError, ValueError)):
            S.predict(m, y, c)
