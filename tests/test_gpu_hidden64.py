"""64 hidden channels: the stacked-operand tensor-core kernels (c = 64 and 128) against the CUDA-core kernels of
the same stage, at the edges of the 128-position tiles, over masks, chunked planes and unaligned LayerNorm
vectors."""

import pytest
import torch

from oracle import trimul_oracle as O
from tests._util import weights_dict

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    from miniworld_engine_b200 import _lib
    _lib.load()
    return torch.device("cuda", 0)


def shifted(t):
    """The same values at an address that is 4-byte but not 16-byte aligned."""
    buf = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    buf[1:].copy_(t)
    return buf[1:]


@pytest.mark.parametrize("outgoing", [True, False], ids=["outgoing", "incoming"])
@pytest.mark.parametrize("c", [64, 128])
@pytest.mark.parametrize("B,N,mask_kind,layout", [
    (1, 1, None, {}), (2, 31, "pair", {}), (1, 128, "token", {}), (3, 129, "token", {}), (1, 200, None, {}),
    (1, 257, "pair", {}), (2, 256, "token", dict(row_chunk=128)), (1, 256, "pair", dict(col_chunk=64))])
def test_stage1_matches_the_cuda_core_kernel(dev, c, B, N, mask_kind, layout, outgoing):
    from miniworld_engine_b200 import read_status, stages as S
    w = O.make_weights(c, 31, affine="random", h=64)
    kw = weights_dict(w, torch.bfloat16, dev)
    kw["ln_in_w"], kw["ln_in_b"] = shifted(kw["ln_in_w"]), shifted(kw["ln_in_b"])
    z = O.make_input(B, N, c, 32).bfloat16().to(dev)
    g = torch.Generator().manual_seed(33)
    mask = {None: None, "token": torch.rand(B, N, generator=g) > 0.2,
            "pair": torch.rand(B, N, N, generator=g) > 0.2}[mask_kind]
    mask = None if mask is None else mask.to(dev)

    def run(plain):
        a, b = (S.alloc_planes(B * 64, N, N, torch.bfloat16, dev, fill=float("nan"), **layout) for _ in range(2))
        S.tm1(z, mask, kw, a, b, outgoing=outgoing, plain_kernels=plain)
        return S.planes_to_dense(a).float(), S.planes_to_dense(b).float()

    for got, ref in zip(run(False), run(True)):
        # same rounding points (x_n, the stored product); the gate's hardware tanh is good to 2.5e-4, a bf16 ulp is 2^-8
        assert not torch.isnan(got).any()
        assert O.rel_rms(got.cpu(), ref.cpu()) <= 4e-3
        assert ((got - ref).abs() <= 2 ** -7 * ref.abs() + 1e-3 * ref.abs().max()).all()
    assert read_status(dev)[0] == 0
