"""The expert products for few tokens that read every chosen expert once (csrc/moe_few.cu), against the same sums in 64 bits."""
import pytest
import torch

from bitnet_c_b200.csrc import ops

pytestmark = pytest.mark.gpu


def _case(tokens, width, ff, experts, top, act, identity, seed):
    g = torch.Generator().manual_seed(seed)
    draw = lambda *shape, std=1.0: (torch.randn(*shape, generator=g) * std).bfloat16().cuda()
    per = 1 if act == ops.ACT_RELU2 else 2
    h = draw(tokens, width)
    up, down = draw(experts, per * ff, width, std=width ** -0.5), draw(experts, width, ff, std=ff ** -0.5)
    score = torch.rand(tokens, experts + identity, generator=g)
    score[:, : max(1, experts // 3)] += 0.5  # some experts are chosen by many tokens, some by none
    ids = score.topk(top, 1).indices.to(torch.int32).cuda()
    weights = torch.rand(tokens, top, generator=g).cuda() + 0.1
    return h, ids, weights, up, down


def _expected(h, ids, weights, up, down, limit, slope, scale_input, add, act, add_scale):
    """The sums in 64 bits, rounded to bfloat16 where the kernels store or hand on bfloat16; and the sum of the absolute values of
    the last product's terms."""
    experts, ff = up.shape[0], down.shape[2]
    out = torch.zeros(h.shape, dtype=torch.float64, device=h.device)
    size = torch.zeros_like(out)
    for t in range(h.shape[0]):
        for k in range(ids.shape[1]):
            e, wt = int(ids[t, k]), weights[t, k]
            if e >= experts:
                out[t] += h[t].double() * wt.double()
                continue
            x = (h[t].float() * wt).bfloat16() if scale_input else h[t]
            z = (up[e].double() @ x.double()).bfloat16()
            if act == ops.ACT_RELU2:
                y = z.double().clamp_min(0) ** 2
            else:
                a, b = z[:ff].double(), z[ff:].double()
                if act < 0:
                    a = a.clamp(max=limit)
                    y = a * torch.sigmoid(slope * a) * (b.clamp(-limit, limit) + 1)
                else:
                    y = (a * torch.sigmoid(a) if act == 0 else torch.nn.functional.gelu(a, approximate="tanh")) * b
            y, w = y.bfloat16().double(), (1.0 if scale_input else wt.double())
            out[t] += w * (down[e].double() @ y)
            size[t] += w * (down[e].double().abs() @ y.abs())
    if add is not None:
        out += add.double() * (1.0 if add_scale is None else add_scale.double()[:, None])
    return out, size


@pytest.mark.parametrize("tokens,width,ff,experts,top,act,scale_input,identity", [
    (1, 64, 40, 4, 2, 0, False, 0),       # one token; an inner dimension that ends within a group of 32
    (3, 72, 264, 5, 1, -1, True, 0),      # warps without a share of the inner dimension; weights on the input
    (8, 1024, 512, 8, 2, 0, False, 0),
    (16, 512, 1024, 16, 4, 1, False, 0),  # one full tile of tokens
    (17, 256, 136, 3, 2, 0, False, 2),    # a second tile; identity experts
    (33, 128, 2048, 4, 3, ops.ACT_RELU2, False, 0),
    (64, 520, 264, 6, 2, -1, True, 0),    # the most items of one launch; experts with more than 32 of them
    (8, 128, 40, 12, 16, 0, False, 4),    # as many experts per token as there are, identity experts among them
    (70, 256, 128, 8, 2, 0, False, 1),    # two launches
    (9, 128, 64, 40, 32, 0, False, 0),    # many experts per token: 4 tokens per launch
])
@pytest.mark.parametrize("with_add", [False, True])
def test_moe_experts_few_bfloat16(tokens, width, ff, experts, top, act, scale_input, identity, with_add):
    h, ids, weights, up, down = _case(tokens, width, ff, experts, top, act, identity, seed=tokens * 1000 + ff)
    add = torch.randn(tokens, width, device="cuda") if with_add else None
    add_scale = torch.rand(tokens, device="cuda") if with_add and act == 0 else None
    got = ops.moe_experts_few(h, ids, weights, up, down, 3.0, 1.5, scale_input, add=add, act=act, add_scale=add_scale)
    want, size = _expected(h, ids, weights, up, down, 3.0, 1.5, scale_input, add, act, add_scale)
    # A stored value may round the other way where a sum of another order falls on the other side: the gate, the up value and the
    # activation each by one part in 2^8, the gate's through a slope of the activation of at most 2 of its own size.
    bound = (4 * 2.0 ** -8) * size + 1e-5 * want.abs() + 1e-6
    assert ((got.double() - want).abs() <= bound).all()
    assert (got.double() - want).norm() <= 2.0 ** -8 * want.norm()  # and on the whole far fewer than all of them
    for t in (0, tokens - 1):  # a token's result does not depend on the batch around it
        one = slice(t, t + 1)
        alone = ops.moe_experts_few(h[one], ids[one], weights[one], up, down, 3.0, 1.5, scale_input,
                                    add=None if add is None else add[one], act=act, add_scale=None if add_scale is None else add_scale[one])
        assert torch.equal(alone, got[one])


def test_moe_experts_few_repeated_expert():
    """A token whose entries name one expert twice (a table's entry out of range stands for expert 0 with weight 0)."""
    h, ids, weights, up, down = _case(5, 64, 64, 3, 2, 0, 0, seed=5)
    ids[:, 1] = ids[:, 0]
    weights[::2, 1] = 0.0
    got = ops.moe_experts_few(h, ids, weights, up, down, 0.0, 0.0, False, act=0)
    want, size = _expected(h, ids, weights, up, down, 0.0, 0.0, False, None, 0, None)
    assert ((got.double() - want).abs() <= (4 * 2.0 ** -8) * size + 1e-6).all()


@pytest.mark.parametrize("tokens,width,ff,experts,top", [(1, 1024, 2048, 8, 2), (8, 2048, 7168, 4, 2), (33, 1024, 1408, 8, 2)])
def test_moe_experts_few_is_as_exact_as_float32(tokens, width, ff, experts, top):
    """The last product's sums stay float32: no further from 64 bits than the kernel that multiplies and adds in float32 (sums that stay
    in the tensor cores' accumulators, which cut off instead of rounding, were 2 to 7 times as far).  An input of a single one makes
    the first product exact."""
    h, ids, weights, up, down = _case(tokens, width, ff, experts, top, ops.ACT_RELU2, 0, seed=tokens + ff)
    h = torch.zeros_like(h)
    h[:, 3] = 1.0
    weights = torch.ones_like(weights)
    want, _ = _expected(h, ids, weights, up, down, 0.0, 0.0, False, None, ops.ACT_RELU2, None)
    err = [float((ops.moe_experts_few(h, ids, weights, up, down, 0.0, 0.0, False, act=ops.ACT_RELU2, read_once=once).double() - want).norm())
           for once in (True, False)]
    assert err[0] <= 1.1 * err[1]


@pytest.mark.parametrize("tokens,width,ff,experts,top", [(2, 512, 256, 32, 1), (3, 512, 256, 32, 1), (3, 512, 256, 17, 1), (16, 512, 256, 32, 8), (17, 512, 256, 32, 8),
                                                         (43, 1024, 512, 42, 4), (33, 1024, 512, 43, 4), (65, 1024, 512, 64, 2), (65, 1024, 512, 64, 1),
                                                         (32, 1024, 512, 65, 1), (33, 1024, 512, 65, 1)])
def test_moe_experts_few_on_both_sides_of_the_choice(monkeypatch, tokens, width, ff, experts, top):
    """Whichever kernels the sizes choose (each expert once for all tokens, or per token), the results agree."""
    h, ids, weights, up, down = _case(tokens, width, ff, experts, top, 0, 0, seed=tokens + experts)
    run = lambda: ops.moe_experts_few(h, ids, weights, up, down, 0.0, 0.0, False, act=0)
    got = run()
    want, size = _expected(h, ids, weights, up, down, 0.0, 0.0, False, None, 0, None)
    for chosen in (None, True, False):
        if chosen is not None:
            monkeypatch.setattr(ops, "moe_once_pays", lambda *a: chosen)
        assert ((run().double() - want).abs() <= (4 * 2.0 ** -8) * size + 1e-6).all()  # as above
    monkeypatch.undo()
    assert torch.equal(run(), got)


@pytest.mark.parametrize("tokens,width,ff,experts,top,act,scale_input,identity", [
    (1, 64, 64, 3, 2, 0, False, 0),
    (5, 72, 200, 4, 2, 0, False, 0),      # lanes without a last piece; runs that end within a unit of rows
    (3, 4104, 264, 2, 1, 1, False, 0),
    (33, 128, 2048, 4, 3, ops.ACT_RELU2, False, 0),  # experts passed over several times
    (64, 520, 264, 6, 2, -1, True, 0),    # the most items of one launch; weights on the input
    (64, 264, 128, 1, 1, 0, True, 0),     # one expert for all
    (8, 128, 40, 12, 16, 0, False, 4),    # identity experts
    (9, 128, 64, 40, 32, 0, False, 0),    # several launches
    (3, 40960, 64, 4, 2, 0, False, 0),    # the longest rows: few beside the ring
    (12, 64, 40960, 3, 1, 0, False, 0),
])
@pytest.mark.parametrize("with_add", [False, True])
def test_moe_experts_few_in_order(monkeypatch, tokens, width, ff, experts, top, act, scale_input, identity, with_add):
    """Without ``read_once`` the sums are those of the kernels that read an expert per item, bit for bit, whichever kernels run."""
    h, ids, weights, up, down = _case(tokens, width, ff, experts, top, act, identity, seed=tokens * 1000 + ff)
    add = torch.randn(tokens, width, device="cuda") if with_add else None
    add_scale = torch.rand(tokens, device="cuda") if with_add and act == 0 else None
    out = []
    for once in (True, False):
        monkeypatch.setattr(ops, "moe_in_order_pays", lambda *a: once)
        out.append(ops.moe_experts_few(h, ids, weights, up, down, 3.0, 1.5, scale_input, add=add, act=act, add_scale=add_scale, read_once=False))
    assert torch.equal(*out)


def test_moe_experts_few_in_order_again_and_again(monkeypatch):
    """Experts without a gate run one kernel for both products: the larger shared memory of the one is still granted when the other has asked for
    less, in every later call."""
    wide, narrow = (_case(8, w, f, 8, 2, ops.ACT_RELU2, 0, seed=w) for w, f in ((4096, 1024), (1024, 4096)))
    for case in (wide, narrow, wide, wide):
        out = []
        for once in (True, False):
            monkeypatch.setattr(ops, "moe_in_order_pays", lambda *a: once)
            out.append(ops.moe_experts_few(*case, 3.0, 1.5, False, act=ops.ACT_RELU2, read_once=False))
        assert torch.equal(*out)
