"""The products per head around attention in a latent space, for few tokens (csrc/latent.cu), against 64 bits."""
import pytest
import torch

from bitnet_c_b200.csrc import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens,heads,dim,rot,rank,vdim", [
    (1, 1, 8, 0, 8, 8),
    (3, 5, 40, 8, 72, 36),        # parts of blocks: columns, rows and numbers of a head
    (4, 16, 128, 64, 192, 128),
    (5, 3, 256, 64, 512, 160),    # the largest; a second, nearly empty turn of tokens
    (64, 2, 129, 2, 264, 33),
])
def test_latent_products(tokens, heads, dim, rot, rank, vdim):
    g = torch.Generator().manual_seed(tokens + rank)
    draw = lambda *s, std=1.0: (torch.randn(*s, generator=g) * std).bfloat16().cuda()
    wide = draw(tokens, 8 + heads * (dim + rot))
    q, uk, uv = wide[:, 8:], draw(heads, dim, rank, std=dim ** -0.5), draw(heads, vdim, rank, std=rank ** -0.5)  # a view with rows of its own
    assert ops.latent_few(tokens, q, uk, uv)
    got = ops.latent_queries(q, uk, rot)
    q3 = q.reshape(tokens, heads, dim + rot)
    want = torch.einsum("thd,hdr->thr", q3[..., :dim].double(), uk.double())
    size = torch.einsum("thd,hdr->thr", q3[..., :dim].double().abs(), uk.double().abs())
    assert ((got[..., :rank].double() - want).abs() <= 2.0 ** -8 * want.abs() + dim * 2.0 ** -24 * size).all()  # one rounding to bfloat16
    assert torch.equal(got[..., rank:], q3[..., dim:])
    x = draw(tokens, heads * rank)
    got = ops.latent_values(x, uv).view(tokens, heads, vdim)
    x3 = x.view(tokens, heads, rank).double()
    want, size = torch.einsum("thr,hvr->thv", x3, uv.double()), torch.einsum("thr,hvr->thv", x3.abs(), uv.double().abs())
    assert ((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + rank * 2.0 ** -24 * size).all()


def test_latent_few_refuses_what_the_kernels_cannot_hold():
    z = lambda *s, dtype=torch.bfloat16: torch.zeros(*s, dtype=dtype, device="cuda")
    fits = lambda tokens=4, dim=64, rank=64, dtype=torch.bfloat16: ops.latent_few(tokens, z(tokens, 2 * dim, dtype=dtype), z(2, dim, rank, dtype=dtype),
                                                                                 z(2, 32, rank, dtype=dtype))
    assert fits() and not fits(tokens=65) and not fits(dim=257) and not fits(rank=520) and not fits(rank=60) and not fits(dtype=torch.float32)
