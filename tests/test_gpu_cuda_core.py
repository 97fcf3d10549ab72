"""The CUDA-core kernels (fp32, and the widths no tensor-core kernel covers) at the edges of their tiles,
against the oracle, and over the chunked plane layouts."""

import pytest
import torch

from oracle import trimul_oracle as O
from tests._util import forward_kwargs, weights_dict

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    from miniworld_engine_b200 import _lib
    _lib.load()
    return torch.device("cuda", 0)


def block64(z, mask, w, outgoing):
    """The block in 64 bits (reference.py:66-83); the oracle's LayerNorm computes in fp32."""
    d = lambda t: t.double()
    ln = lambda x, g, b, eps: torch.nn.functional.layer_norm(x, x.shape[-1:], d(g), d(b), eps)
    x = ln(d(z), w.ln_pair_weight, w.ln_pair_bias, w.eps_in)
    keep = d((mask[:, :, None] & mask[:, None, :])[..., None])
    left = torch.sigmoid(x @ d(w.to_left_gate).T) * (x @ d(w.to_left).T) * keep
    right = torch.sigmoid(x @ d(w.to_right_gate).T) * (x @ d(w.to_right).T) * keep
    tri = torch.einsum("bikd,bjkd->bijd" if outgoing else "bkid,bkjd->bijd", left, right)
    return torch.sigmoid(x @ d(w.to_gate).T) * (ln(tri, w.ln_out_weight, w.ln_out_bias, w.eps_out) @ d(w.to_out).T)


# token counts around the 32 / 64 / 128-position tiles and a row length below one tile; widths around the 64-channel
# blocks and the 32-wide K slices; N = 200 and 250 are enough planes of little enough padding for the contraction's
# 128 x 128 tiles
@pytest.mark.parametrize("outgoing", [True, False], ids=["outgoing", "incoming"])
@pytest.mark.parametrize("c,B,N", [(128, 1, 1), (128, 1, 5), (128, 2, 33), (128, 1, 96), (128, 1, 131), (64, 1, 65),
                                   (8, 3, 17), (40, 1, 70), (72, 2, 64), (136, 1, 40), (256, 1, 67), (128, 1, 200),
                                   (128, 1, 250)])
def test_fp32_block_at_tile_edges(dev, c, B, N, outgoing):
    from miniworld_engine_b200 import read_status, trimul_forward
    w = O.make_weights(c, 11, affine="random")
    z = O.make_input(B, N, c, 12)
    g = torch.Generator().manual_seed(13)
    m = torch.rand(B, N, generator=g) > 0.2
    ds = (torch.rand(B, 1, N, c, generator=g) > 0.25).float() / 0.75
    kw = forward_kwargs(w, torch.float32, dev)
    zd = z.to(dev)
    y = trimul_forward(zd, m.to(dev), outgoing=outgoing, residual=zd, drop_scale=ds.to(dev), **kw).cpu().double()
    assert read_status(dev)[0] == 0
    ref = block64(z, m, w, outgoing) * ds.double()
    # the roundings of an fma chain of length k add up like sqrt(k) u (u = 2^-24; the worst case, k u, is never near): three
    # chains of up to 256, 250 and 256 and two LayerNorms stay below 2e-6, 1e-5 is what the path is held to; the sum with the
    # residual is rounded once more
    tol = 2e-6 + 2.0 ** -24 * float(y.norm() / ref.norm())
    assert float((y - z.double() - ref).norm() / ref.norm()) <= tol


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16], ids=["fp32", "bf16"])
@pytest.mark.parametrize("chunk", ["rows16", "cols16", "cols6"])
def test_chunked_planes_give_the_plain_layouts_result(dev, dtype, chunk):
    """Every output is one fma chain over ascending k, so the layout of the planes must not change a bit."""
    from miniworld_engine_b200 import stages as S
    N, c = 48, 40
    w = O.make_weights(c, 21, affine="random")
    kw = weights_dict(w, dtype, dev)
    z = O.make_input(1, N, c, 22).to(dtype).to(dev)
    layout = {"rows16": dict(row_chunk=16), "cols16": dict(col_chunk=16), "cols6": dict(col_chunk=6)}[chunk]

    def run(**lay):
        a, b, t = (S.alloc_planes(c, N, N, dtype, dev, fill=float("nan"), **lay) for _ in range(3))
        S.tm1(z, None, kw, a, b, outgoing=False, plain_kernels=True)
        S.contract(a, b, t, plain_kernels=True)
        return (*(S.planes_to_dense(s) for s in (a, b, t)), S.tm2(z, t, kw, plain_kernels=True))

    for got, ref in zip(run(**layout), run()):
        assert not torch.isnan(ref.float()).any()
        assert torch.equal(got, ref)
