"""Products of matrices that fit on the chip (csrc/linear_resident.cu): every epilogue, against 64 bits and the clusters of linear_tc.cu."""
import pytest
import torch

from bitnet_c_b200.csrc import ops

pytestmark = pytest.mark.gpu

SIZES = [
    (1, 16, 8),        # one block, lanes without a piece
    (3, 48, 72),       # an inner dimension that ends within the first warps
    (8, 2048, 2048),   # eight tokens, whole turns
    (9, 1008, 1032),   # a second group of tokens; an inner dimension that ends within a warp's share
    (16, 3072, 2048),
    (16, 64, 6144),    # the longest rows: three turns
    (7, 96, 3000),
]


@pytest.fixture
def by(monkeypatch):
    def choose(resident):
        monkeypatch.setattr(ops, "linear_resident_pays", lambda *a: resident)
    return choose


def _case(M, N, K):
    g = torch.Generator().manual_seed(M * 100 + N + K)
    return (torch.randn(M, K, generator=g).bfloat16().cuda(), (torch.randn(N, K, generator=g) * K ** -0.5).bfloat16().cuda(),
            torch.randn(N, generator=g).cuda())


@pytest.mark.parametrize("M,N,K", SIZES)
def test_plain_bias_and_unit(by, M, N, K):
    x, w, b = _case(M, N, K)
    want, size = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
    err = []
    for resident in (True, False):
        by(resident)
        got = ops.linear_tc(x, w, out_dtype=torch.float32)
        assert ((got.double() - want).abs() <= K * 2.0 ** -23 * size).all()  # sums of K numbers, each cut off or rounded at 2^-23
        err.append(float((got.double() - want).norm()))
    assert err[0] <= 1.1 * err[1] + 1e-7 * float(want.norm())  # no less exact than the other kernel
    by(True)
    got = ops.linear_tc(x, w, out_dtype=torch.float32, bias=b)
    assert ((got.double() - want - b.double()).abs() <= K * 2.0 ** -23 * (size + b.double().abs())).all()
    # the square of the positive part, in bfloat16
    got = ops.linear_tc(x, w, bias=b, act=ops.ACT_RELU2).double()
    y = (want + b.double()).clamp(min=0) ** 2
    assert ((got - y).abs() <= 2.0 ** -8 * y + 1e-4).all()


@pytest.mark.parametrize("M,N,K", [s for s in SIZES if s[1] % 16 == 0])
@pytest.mark.parametrize("act", [ops.ACT_SILU, ops.ACT_GELU_TANH])
def test_gated(by, M, N, K, act):
    x, w, _ = _case(M, N, K)
    by(True)
    got = ops.linear_tc(x, w, swiglu=True, act=act).double()
    z = (x.double() @ w.double().t()).view(M, N // 16, 2, 8)
    gate, up = z[:, :, 0].reshape(M, N // 2), z[:, :, 1].reshape(M, N // 2)
    want = (gate * torch.sigmoid(gate) if act == ops.ACT_SILU else torch.nn.functional.gelu(gate, approximate="tanh")) * up
    assert ((got - want).abs() <= 2.0 ** -8 * want.abs() + 1e-4).all()


@pytest.mark.parametrize("M,N,K", [s for s in SIZES if s[1] % 8 == 0])
def test_residual_and_norm(by, M, N, K):
    """Residual, rows for the next norm and their sums of squares; the rows are then read by either kernel."""
    x, w, b = _case(M, N, K)
    gain, start = b.abs() + 0.5, torch.randn(M, N, device="cuda")
    nxt = _case(M, 40, N)[1]
    res = (start.double() + x.double() @ w.double().t())
    for resident in (True, False):
        by(resident)
        got = start.clone()
        rows = ops.linear_tc(x, w, sink=ops.NormSink(got, gain, 1e-5))
        assert ((got.double() - res).abs() <= 1e-4).all()
        assert ((rows.ss.double().sum(0) - res.square().sum(1)).abs() <= 1e-4 * res.square().sum(1)).all()
        h = res * torch.rsqrt(res.square().mean(1, keepdim=True) + 1e-5) * gain.double()
        for reader in (True, False):
            by(reader)
            z = ops.linear_tc(rows, nxt, out_dtype=torch.float32).double()
            assert ((z - h @ nxt.double().t()).abs() <= 2.0 ** -8 * (h.abs() @ nxt.double().abs().t())).all()


def test_tokens_do_not_depend_on_the_batch(by):
    x, w, _ = _case(8, 512, 1024)
    by(True)
    whole = ops.linear_tc(x, w)
    for m in range(8):
        assert torch.equal(ops.linear_tc(x[m:m + 1].contiguous(), w), whole[m:m + 1])


@pytest.mark.parametrize("M,N,K", [(1, 256, 256), (16, 2048, 2048), (17, 2048, 2048), (8, 2048, 6144), (8, 2048, 6152), (8, 32000, 2048), (2, 8, 64)])
def test_both_sides_of_the_choice(M, N, K):
    x, w, _ = _case(M, N, K)
    want = x.double() @ w.double().t()
    assert (ops.linear(x, w, out_dtype=torch.float32).double() - want).norm() <= 1e-5 * want.norm()
