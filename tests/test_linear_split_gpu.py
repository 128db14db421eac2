"""Float32 products of many rows from split operands (csrc/linear_split.cu), against 64 bits and plain float32."""
import pytest
import torch

from bitnet_c_b200.csrc import ops

pytestmark = pytest.mark.gpu


def _pair(M, N, K, seed, spread=0.0):
    g = torch.Generator().manual_seed(seed)
    x, w = torch.randn(M, K, generator=g), torch.randn(N, K, generator=g) * K ** -0.5
    if spread:  # columns of very different sizes: the small ones are the low parts' business
        x = x * torch.exp(spread * torch.randn(K, generator=g))
    return x.cuda(), w.cuda()


@pytest.mark.parametrize("M,N,K,spread", [
    (17, 128, 128, 0.0),     # the fewest rows, one tile, the smallest inner dimension
    (17, 130, 132, 0.0),     # a tile of two rows of w; an inner dimension that ends within a stage
    (192, 256, 512, 0.0),    # one full tile of rows of x
    (193, 72, 1000, 0.0),    # two of them, the second nearly empty
    (520, 1000, 516, 0.0),
    (33, 8, 2048, 0.0),
    (1000, 64, 192, 0.0),    # more tiles of rows than SMs have tiles of w
    (400, 20000, 160, 0.0),  # several tiles per block
    (300, 384, 4096, 3.0),
    (17, 2048, 288, 0.0),    # nine steps a tile: the groups that split w change places from tile to tile
    (100, 19100, 160, 0.0),  # the same with several tiles per block, and the fewest steps but one
])
@pytest.mark.parametrize("with_bias", [False, True])
def test_linear_split(M, N, K, spread, with_bias):
    x, w = _pair(M, N, K, M + N + K, spread)
    b = torch.randn(N, device="cuda") if with_bias else None
    got = ops.linear_split(x, w, b)
    ops.check_tc_status(x.device)
    want, size = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
    if with_bias:
        want, size = want + b.double(), size + b.double().abs()
    # A sum of 32 numbers in the tensor cores is cut off some twelve times at 2^-23 of its size at most, the sums of those are rounded at
    # 2^-24 each, and the three products that the split leaves out are below 2^-24 + 2^-23 + 2^-32 < 2 * 2^-23 of each product.
    bound = (12 + K / 64 + 2) * 2.0 ** -23 * size
    assert ((got.double() - want).abs() <= bound).all()
    plain = torch.matmul(x, w.t()) if b is None else torch.addmm(b, x, w.t())
    err = lambda y: float((y.double() - want).norm() / want.norm())
    assert err(got) <= max(1.05 * err(plain), 1.5e-7)  # no less exact than float32 sums (below, both are at one rounding of the result)


def test_linear_split_what_does_not_split():
    """Infinities and what is not a number come out as float32 sums give them, numbers near the largest one stay finite, and other rows are
    not touched."""
    x, w = _pair(40, 200, 256, 3)
    clean = ops.linear_split(x, w)
    x[3, 7], x[5, 9], x[6, 1], x[8, 2], w[100, 5], w[7, 7] = float("inf"), float("nan"), 3.39e38, 1e-39, -float("inf"), 0.0
    got, want = ops.linear_split(x, w), torch.matmul(x.double(), w.double().t())
    finite = want.isfinite() & (want.abs() < 3.4e38)
    assert torch.equal(got.isnan(), want.isnan())
    assert torch.equal(got.isinf() & want.isinf(), want.isinf()) and torch.equal(got[want.isinf()].sign().double(), want[want.isinf()].sign())
    assert got[finite].isfinite().all()
    assert ((got.double() - want).abs()[finite] <= 1e-5 * (x.double().abs() @ w.double().abs().t())[finite]).all()
    rows, cols = [m for m in range(40) if m not in (3, 5, 6, 8)], [n for n in range(200) if n not in (7, 100)]
    assert torch.equal(got[rows][:, cols], clean[rows][:, cols])


def test_float32_products_go_by_one_rule(monkeypatch):
    """``linear`` takes whichever kernel the sizes choose, refuses TF32 on both, and both agree."""
    x, w = _pair(70, 256, 512, 9)
    out = {}
    for chosen in (True, False):
        monkeypatch.setattr(ops, "linear_split_pays", lambda *a: chosen)
        out[chosen] = ops.linear(x, w)
        monkeypatch.setattr(torch.backends.cuda.matmul, "allow_tf32", True)
        with pytest.raises(ops.KernelError):
            ops.linear(x, w)
        monkeypatch.setattr(torch.backends.cuda.matmul, "allow_tf32", False)
    assert (out[True] - out[False]).norm() <= 3e-6 * out[False].norm()


def test_profile_counts_a_product_once(monkeypatch):
    """While kernel classes are timed, a float32 product stands under the kernel that ran it and nowhere else."""
    x, w = _pair(70, 256, 512, 9)
    for chosen, key in ((True, "linear_split.bn_linear_split"), (False, "library.matmul")):
        monkeypatch.setattr(ops, "linear_split_pays", lambda *a: chosen)
        monkeypatch.setattr(ops, "PROFILE", {})
        ops.linear(x, w)
        assert {k: len(v) for k, v in ops.PROFILE.items()} == {key: 1}


def test_linear_split_of_a_matrix_that_was_just_written():
    """W, like x, may be what the kernel in front of the product writes."""
    x, w = _pair(64, 8192, 2048, 4)
    clean = ops.linear_split(x, w)
    for i in range(1, 21):
        w1 = w.clone()
        torch.cuda.synchronize()
        ops.scale_softcap(w1, 2.0 ** i, 0.0)  # a kernel of the library, which lets the next one start early
        got = ops.linear_split(x, w1)
        assert torch.equal(got, clean * 2.0 ** i)


def _as_exact_as_float32(x, w, K):
    """``linear_split`` against 64 bits: within its bound (numbers below the smallest normal one are rounded at 2^-149), and no less exact than the
    float32 product."""
    got, plain = ops.linear_split(x, w), torch.matmul(x, w.t())
    ops.check_tc_status(x.device)
    want, size = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
    assert ((got.double() - want).abs() <= (12 + K / 64 + 2) * 2.0 ** -23 * size + 2.0 ** -149).all()
    err = lambda y: float((y.double() - want).norm() / want.norm())
    assert err(got) <= max(1.05 * err(plain), 1.5e-7)


@pytest.mark.parametrize("x_scale,w_scale", [(1e-33, 1.0), (1e-34, 1.0), (1e-35, 30.0), (1.0, 1e-34), (1.0, 1e-35), (3e6, 1e-38), (1e-19, 1e-15),
                                             (1e9, 1.0), (1e20, 1e-20), (1e37, 1e-3), (1e30, 1e-38), (1.0, 1e8)])
def test_linear_split_of_very_small_and_large_numbers(x_scale, w_scale):
    """Operands far below and above one keep all their bits."""
    x, w = _pair(40, 200, 256, 6)
    _as_exact_as_float32(x * x_scale, w * w_scale, 256)


def test_linear_split_of_rows_of_all_sizes():
    """Rows, and numbers within a row, of very different sizes; where the large ones of x meet zeros, the small ones alone make the result."""
    x, w = _pair(48, 200, 256, 7)
    x[::3] *= 1e-35
    x[1::6] *= 1e25
    w[::2] *= 1e-34
    got, want = ops.linear_split(x, w).double(), x.double() @ w.double().t()
    size = x.double().abs() @ w.double().abs().t()
    assert ((got - want).abs() <= (12 + 4 + 2) * 2.0 ** -23 * size + 2.0 ** -149).all()
    for large in (1.0, 1e12, 1e30):  # 1e30 beside 1e-35: too far apart to be split
        x, w = _pair(40, 200, 256, 8)
        x[:, :128] *= large
        x[:, 128:] *= 1e-35
        w[:, :128] = 0
        _as_exact_as_float32(x, w, 256)
    x, w = _pair(40, 200, 256, 8)
    w[5, 9], w[7, 3] = 3e9, -1e30  # weights that are not split
    _as_exact_as_float32(x, w, 256)


@pytest.mark.parametrize("M,N,K", [(17, 130, 132), (193, 300, 1000), (100, 19100, 160)])
@pytest.mark.parametrize("of_x,of_w", [([0], []), ([], [0]), ([3, 16], [5, 129]), (slice(None), []), ([], slice(None))])
def test_linear_split_marked_rows(M, N, K, of_x, of_w):
    """Rows that do not split, at the edges of tiles and all at once: what float32 sums give, and the others' bits untouched."""
    x, w = _pair(M, N, K, M)
    b = torch.randn(N, device="cuda")
    clean = ops.linear_split(x, w, b)
    x1, w1 = x.clone(), w.clone()
    x1[of_x, K // 2] = 3e38
    x1[of_x, K // 3] = 1e-38  # too far apart
    w1[of_w, K - 1] = 2e9
    got, want = ops.linear_split(x1, w1, b).double(), torch.addmm(b.double(), x1.double(), w1.double().t())
    size = x1.double().abs() @ w1.double().abs().t() + b.double().abs()
    fits = size < 3e38  # (sums may become infinite on the way, in any order)
    assert ((got - want).abs()[fits] <= (K / 32 + 8) * 2.0 ** -23 * size[fits]).all()
    x1[of_x, 1], w1[of_w, 2] = float("nan"), float("inf")
    got = ops.linear_split(x1, w1, b)
    rows, cols = torch.ones(M, dtype=torch.bool, device="cuda"), torch.ones(N, dtype=torch.bool, device="cuda")
    rows[of_x], cols[of_w] = False, False
    assert torch.equal(got[rows][:, cols], clean[rows][:, cols])
    assert got[~rows].isnan().all() and not got[rows][:, ~cols].isfinite().any()



@pytest.mark.parametrize("rows", [1, 192, 299, 300])
def test_linear_split_in_bands(monkeypatch, rows):
    """Working space for so many rows only: the same bits, and no more space is asked for."""
    x, w = _pair(300, 200, 516, 5)
    b = torch.randn(200, device="cuda")
    whole = ops.linear_split(x, w, b)
    most = rows * (6 * 520 + 4)
    monkeypatch.setattr(ops, "LINEAR_SPLIT_SCRATCH", most)
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    got = ops.linear_split(x, w, b)
    assert torch.cuda.max_memory_allocated() - before <= most + 300 * 200 * 4 + 2 * 512  # (sizes are rounded up to 512 bytes)
    assert torch.equal(got, whole)


@pytest.mark.parametrize("numbers", [1, 128])
def test_linear_split_leaves_out_no_more_than_it_says(numbers):
    """The significands whose products lose most to the split, of one sign, so that nothing cancels."""
    x, w = torch.zeros(17, 128, device="cuda"), torch.zeros(128, 128, device="cuda")
    x[:, :numbers] = torch.tensor(0x3f807f40, dtype=torch.int32).view(torch.float32)
    w[:, :numbers] = torch.tensor(0x3f80ffff, dtype=torch.int32).view(torch.float32)
    got, want = ops.linear_split(x, w).double(), x.double() @ w.double().t()
    # of one product: its six kept parts are added up with five cuts at 2^-23; of 128, as above
    cuts = 5 if numbers == 1 else 12 + 128 / 64
    assert ((got - want).abs() <= (cuts + 1.51) * 2.0 ** -23 * want).all()
