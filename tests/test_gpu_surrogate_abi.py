"""The surrogate library's C entry points on what their header allows beyond the package's own calls.
Where the same operations run, results are equal; what is refused is refused before a launch."""
import ctypes

import luna_b200_loader  # registers the luna.jl_b200 package

luna_b200_loader.load()

import pytest

pytestmark = pytest.mark.gpu


def _sg():
    torch = pytest.importorskip("torch")
    from luna_b200 import surrogate as S
    return torch, S.load(), (lambda t: ctypes.c_void_p(t.data_ptr())), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def _layer(torch, members, B, K, N, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    bf = torch.bfloat16
    return dict(X=torch.randn(members, B, K, device="cuda", generator=g).to(bf),
                W=(torch.randn(members, N, K, device="cuda", generator=g) / K ** 0.5).to(bf),
                b=torch.randn(members, N, device="cuda", generator=g),
                dZ=torch.randn(members, B, N, device="cuda", generator=g).to(bf),
                Zp=torch.randn(members, B, K, device="cuda", generator=g).to(bf),
                err=torch.zeros(1, dtype=torch.int32, device="cuda"))


def _offset(torch, t, n):
    """A copy of t that starts n elements behind a 16-byte boundary."""
    flat = torch.zeros(t.numel() + 16, dtype=t.dtype, device="cuda")
    v = flat[n:n + t.numel()].view(t.shape)
    v.copy_(t)
    return v


@pytest.mark.parametrize("off", [1, 2, 3])
def test_bias_as_a_slice_of_a_flat_parameter_buffer(off):
    torch, lib, p, st = _sg()
    members, B, K, N = 2, 128, 64, 128
    d = _layer(torch, members, B, K, N)
    b = _offset(torch, d["b"], off)
    assert b.data_ptr() % 16 == 4 * off
    out = []
    for bias in (d["b"], b):
        Y, m, s = torch.zeros(members, B, N, device="cuda"), torch.zeros(B, N, device="cuda"), torch.zeros(B, device="cuda")
        assert lib.luna_sg_linear_fwd(p(d["X"]), B * K, p(d["W"]), p(bias), B, K, N, 1, None, None, p(Y), members, p(d["err"]), st) == 0
        assert lib.luna_sg_linear_ensemble(p(d["X"]), B * K, p(d["W"]), p(bias), B, K, N, N, p(m), p(s), members, p(d["err"]), st) == 0
        out.append((Y, m, s))
    torch.cuda.synchronize()
    assert int(d["err"].item()) == 0
    assert all(torch.equal(x, y) for x, y in zip(*out))


def test_misaligned_outputs_are_refused():
    """Return codes only: nothing is launched."""
    torch, lib, p, st = _sg()
    members, B, K, N = 1, 128, 128, 128
    d = _layer(torch, members, B, K, N)
    bf = torch.bfloat16
    big = torch.zeros(B * N + 64, device="cuda")
    q = lambda nbytes: ctypes.c_void_p(big.data_ptr() + nbytes)
    X, W, b, dZ, Zp, err = (p(d[k]) for k in ("X", "W", "b", "dZ", "Zp", "err"))
    for k in (4, 8):
        for Y, Z, Yf in ((q(k), None, None), (None, q(k), None), (None, None, q(k))):
            assert lib.luna_sg_linear_fwd(X, B * K, W, b, B, K, N, 1, Y, Z, Yf, members, err, st) == 16
        assert lib.luna_sg_linear_bwd_data(dZ, W, Zp, B, K, N, q(k), members, err, st) == 16
        assert lib.luna_sg_linear_bwd_data(dZ, W, q(k), B, K, N, q(0), members, err, st) == 16
        assert lib.luna_sg_linear_bwd_weight(dZ, X, B * K, B, K, N, q(k), b, members, err, st) == 16
    assert lib.luna_sg_linear_fwd(X, B * K, W, q(2), B, K, N, 1, None, None, q(16), members, err, st) == 16
    torch.cuda.synchronize()
    assert not big.any()


@pytest.mark.parametrize("off,gap", [(0, 2), (2, 0), (4, 6), (6, 0)])
def test_backward_operands_at_four_byte_alignment(off, gap):
    """dZ, X and W of the transposed roles as slices of larger buffers (`off` elements behind a 16-byte
    boundary) and X with a member stride of an even number of elements."""
    torch, lib, p, st = _sg()
    members, B, K, N = 2, 128, 128, 256
    d = _layer(torch, members, B, K, N)
    Xb = torch.zeros(members * (B * K + gap) + 16, dtype=torch.bfloat16, device="cuda")
    for m in range(members):
        Xb[off + m * (B * K + gap):][:B * K].copy_(d["X"][m].flatten())
    moved = dict(X=(Xb[off:], B * K + gap), dZ=_offset(torch, d["dZ"], off), W=_offset(torch, d["W"], off))
    out = []
    for X, sX, dZ, W in ((d["X"], B * K, d["dZ"], d["W"]), (*moved["X"], moved["dZ"], moved["W"])):
        dX, dW, db = (torch.zeros(members, B, K, device="cuda", dtype=torch.bfloat16), torch.zeros(members, N, K, device="cuda"),
                      torch.zeros(members, N, device="cuda"))
        assert lib.luna_sg_linear_bwd_data(p(d["dZ"]), p(W), p(d["Zp"]), B, K, N, p(dX), members, p(d["err"]), st) == 0
        assert lib.luna_sg_linear_bwd_weight(p(dZ), p(X), sX, B, K, N, p(dW), p(db), members, p(d["err"]), st) == 0
        out.append((dX, dW, db))
    torch.cuda.synchronize()
    assert int(d["err"].item()) == 0 and out[0][1].any()
    assert all(torch.equal(x, y) for x, y in zip(*out))


def test_members_in_reverse_order():
    """A negative member stride: member z reads the matrix before member z - 1's."""
    torch, lib, p, st = _sg()
    members, B, K, N = 3, 128, 64, 128
    d = _layer(torch, members, B, K, N)
    Y = torch.zeros(2, members, B, N, device="cuda")
    last = ctypes.c_void_p(d["X"][-1].data_ptr())
    assert lib.luna_sg_linear_fwd(last, -B * K, p(d["W"]), p(d["b"]), B, K, N, 1, None, None, p(Y[0]), members, p(d["err"]), st) == 0
    X = d["X"].flip(0).contiguous()
    assert lib.luna_sg_linear_fwd(p(X), B * K, p(d["W"]), p(d["b"]), B, K, N, 1, None, None, p(Y[1]), members, p(d["err"]), st) == 0
    torch.cuda.synchronize()
    assert torch.equal(Y[0], Y[1]) and int(d["err"].item()) == 0


@pytest.mark.parametrize("B,nf", [(1, 1), (65, 252), (4095, 129), (4096, 128), (4100, 128), (22000, 24), (131072, 23), (5000, 896), (70, 897), (4097, 2000)])
def test_features_of_every_width(B, nf):
    """Both kernels at the edges of their rule, and rows that do not fit in shared memory. Bound: the
    projection's eight rounded products and sums (|f . x| < 60: 16 2^-24 60 of a turn, times 2 pi 3.6e-4)
    and the rounding to BF16 (2^-9)."""
    torch, lib, p, st = _sg()
    g = torch.Generator(device="cuda").manual_seed(nf)
    x, f = torch.randn(B, 8, device="cuda", generator=g), torch.randn(nf, 8, device="cuda", generator=g)
    ld = 8 + 2 * nf
    out = torch.full((B, ld), 9.0, device="cuda", dtype=torch.bfloat16)
    assert lib.luna_sg_features(p(x), B, p(f), nf, p(out), ld, st) == 0
    torch.cuda.synchronize()
    d = x.double() @ f.double().T
    assert d.abs().max() < 60
    a = 2 * torch.pi * (d - d.round())
    assert torch.equal(out[:, :8], x.to(torch.bfloat16))
    assert (out[:, 8:8 + nf].double() - a.sin()).abs().max() < 2.0 ** -9 + 4e-4
    assert (out[:, 8 + nf:].double() - a.cos()).abs().max() < 2.0 ** -9 + 4e-4


@pytest.mark.parametrize("B,N,nspec,members", [(1, 512, 512, 12), (2048, 768, 100, 3), (2049, 768, 100, 3), (300, 511, 511, 2), (300, 513, 257, 5),
                                               (77, 4099, 0, 1), (130, 7, 7, 40)])
def test_statistics_with_a_warp_or_a_block_a_row(B, N, nspec, members):
    """Mean and spread against 64-bit values: the sums of `members` FP32 terms and one division within
    members 2^-23 of the sum of magnitudes, a variance within 4 members 2^-23 of the mean square."""
    torch, lib, p, st = _sg()
    Y = torch.randn(members, B, N, device="cuda", generator=torch.Generator(device="cuda").manual_seed(N)) + 1
    mean, spread = torch.full((B, N), 7.0, device="cuda"), torch.full((B,), 7.0, device="cuda")
    assert lib.luna_sg_ensemble(p(Y), members, B, N, nspec, p(mean), p(spread), st) == 0
    torch.cuda.synchronize()
    d = Y.double()
    assert ((mean - d.mean(0)).abs() <= members * 2.0 ** -23 * d.abs().mean(0)).all()
    var = d.var(0, unbiased=False)[:, :nspec].amax(1) if nspec and members > 1 else torch.zeros(B, device="cuda").double()
    msq = (d ** 2).mean(0)[:, :max(nspec, 1)].amax(1)
    assert ((spread.double() ** 2 - var).abs() <= 4 * members * 2.0 ** -23 * msq).all()


def _blocks(torch, values, bad):
    """Columns of 32 values, the first of each block replaced by `bad` in a second copy: 31 of 32 columns
    are the same values once in the range of the common case and once beside one outside."""
    a = values.view(-1, 32).clone()
    a[:, 0] = 0.5
    b = a.clone()
    b[:, 0] = bad
    return a.flatten(), b.flatten()


@pytest.mark.parametrize("bad,act", [(-70.0, 0.0), (1e31, 1e31), (float("inf"), float("inf")), (float("-inf"), float("nan")),
                                     (float("nan"), float("nan"))])
def test_silu_is_the_same_beside_values_out_of_its_common_range(bad, act):
    """act(v) of biases over all exponents from 2^-126 to 2^99 and both signs (v > -69): the division
    without a range check gives the operator's bits, and the operator's form takes what lies
    outside. Against 64-bit values: __expf within 2 + 1.173 |v| ulp and three roundings of 2^-24."""
    torch, lib, p, st = _sg()
    g = torch.Generator(device="cuda").manual_seed(1)
    n = 1 << 17
    mant, ex = 1 + torch.rand(n, device="cuda", generator=g), torch.randint(-126, 100, (n,), device="cuda", generator=g)
    v = torch.ldexp(mant, ex)
    w = torch.where(torch.rand(n, device="cuda", generator=g) < 0.5, torch.ldexp(mant, ex.clamp(max=5)), 68.9 * torch.rand(n, device="cuda", generator=g))
    v = torch.cat([v, -w.clamp(max=68.9), torch.tensor([0.0, -0.0] * 16, device="cuda"), 80 * torch.rand(n - 32, device="cuda", generator=g)])
    B, K = 128, 64
    X, W = torch.zeros(B, K, dtype=torch.bfloat16, device="cuda"), torch.zeros(v.numel(), K, dtype=torch.bfloat16, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    out = []
    for b in _blocks(torch, v, bad):
        Y = torch.empty(B, b.numel(), device="cuda")
        assert lib.luna_sg_linear_fwd(p(X), 0, p(W), p(b), B, K, b.numel(), 1, None, None, p(Y), 1, p(err), st) == 0
        torch.cuda.synchronize()
        assert torch.equal(Y[0].view(torch.int32), Y[-1].view(torch.int32))
        out.append(Y[0].view(-1, 32))
    a, b = out
    assert int(err.item()) == 0 and torch.equal(a[:, 1:].view(torch.int32), b[:, 1:].view(torch.int32))
    x = v.view(-1, 32)[:, 1:].double()
    ref = x * torch.sigmoid(x)
    tol = ((2 + 1.173 * x.abs().clamp(max=100)) * 2.0 ** -23 + 3 * 2.0 ** -24) * ref.abs() + 2.0 ** -149
    assert ((a[:, 1:].double() - ref).abs() <= tol).all()
    assert torch.allclose(b[:, 0].double(), torch.full_like(b[:, 0], act).double(), rtol=1e-6, atol=1e-27, equal_nan=True)


@pytest.mark.parametrize("bad", [-70.0, 1e31, float("inf"), float("nan")])
def test_silu_derivative_is_the_same_beside_values_out_of_its_common_range(bad):
    """v silu'(z) for every BF16 z above -69, v = 1: a warp's rows share eight columns, so a value out of
    range in one row sends the others through the operator's form."""
    torch, lib, p, st = _sg()
    bits = torch.arange(1 << 16, device="cuda", dtype=torch.int32).to(torch.int16)
    z = bits.view(torch.bfloat16)
    z = z[torch.isfinite(z) & (z > -69) & (z < 1e30)]
    z = torch.cat([z, z[: (-z.numel()) % (4 * 31 * 128)]]).view(-1, 4, 31, 128)  # 31 of a warp's 32 rows
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    B, K, N = 128, 128, 128
    dZ, W = (torch.zeros(B, N, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    dZ[:, 0] = 1
    W[0, :] = 1  # dZ W = 1 everywhere
    for block in z:
        out = []
        for q in (0.5, bad):
            Zp = torch.cat([block, torch.full((4, 1, K), q, dtype=torch.bfloat16, device="cuda")], 1).contiguous()
            dX = torch.empty(B, K, dtype=torch.bfloat16, device="cuda")
            assert lib.luna_sg_linear_bwd_data(p(dZ), p(W), p(Zp), B, K, N, p(dX), 1, p(err), st) == 0
            out.append(dX.view(4, 32, K)[:, :-1])
        torch.cuda.synchronize()
        assert torch.equal(out[0].view(torch.int16), out[1].view(torch.int16))
        x = block.double()
        s = torch.sigmoid(x)
        ref = s * (1 + x * (1 - s))
        assert ((out[0].double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-5).all()
    assert int(err.item()) == 0
