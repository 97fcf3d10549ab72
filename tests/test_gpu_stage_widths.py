"""Stages 1 and 3 on the tensor cores at widths other than c = h = 128: stage 1 against the CUDA-core kernel of the
same stage, stage 3 against 64 bits, at the edges of the 128-position tiles (odd tile counts among them), over masks,
residuals, dropout scales, chunked planes and unaligned LayerNorm vectors."""

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
        # same rounding points (x_n, the stored product); the gate's hardware tanh (c = 64) is good to 4e-6, a bf16 ulp is 2^-8
        assert not torch.isnan(got).any()
        assert O.rel_rms(got.cpu(), ref.cpu()) <= 4e-3
        assert ((got - ref).abs() <= 2 ** -7 * ref.abs() + 1e-3 * ref.abs().max()).all()
    assert read_status(dev)[0] == 0


@pytest.mark.parametrize("c,h", [(64, 64), (128, 64), (128, 128), (128, 256), (256, 256)])
@pytest.mark.parametrize("B,N,residual,scale", [
    (1, 1, "z", False), (2, 33, None, False), (1, 128, "z", True), (1, 129, None, True), (3, 127, "z", False),
    (1, 255, "other", False), (1, 300, "z", True), (3, 130, "z", True), (1, 385, None, False)])
def test_stage3_against_64_bits(dev, c, h, B, N, residual, scale):
    """The folded last stage, with LayerNorm vectors at any float address, and what takes over for another residual,
    against the stage in 64 bits on the same bf16 operands."""
    from miniworld_engine_b200 import _lib, read_status, stages as S
    from miniworld_engine_b200.functional import _status_words
    import ctypes as C
    w = O.make_weights(c, 41, affine="random", h=h).to(torch.bfloat16)
    kw = weights_dict(w, torch.bfloat16, dev)
    g = torch.Generator().manual_seed(42)
    z = torch.randn(B, N, N, c, generator=g).bfloat16()
    tri = (torch.randn(B * h, N, N, generator=g) + 0.5).bfloat16()
    ds = ((torch.rand(B, 1, N, c, generator=g) > 0.25).float() / 0.75).bfloat16() if scale else None
    res = {None: None, "z": z, "other": torch.randn(B, N, N, c, generator=g).bfloat16()}[residual]

    d64 = lambda t: t.double()
    ln = lambda x, gm, bt, eps: torch.nn.functional.layer_norm(x, x.shape[-1:], d64(gm), d64(bt), eps)
    zn = ln(d64(z), w.ln_pair_weight, w.ln_pair_bias, w.eps_in)
    tn = ln(d64(tri).view(B, h, N, N).permute(0, 2, 3, 1), w.ln_out_weight, w.ln_out_bias, w.eps_out)
    upd = torch.sigmoid(zn @ d64(w.to_gate).T) * (tn @ d64(w.to_out).T)
    if ds is not None:
        upd = upd * d64(ds)

    t = S.alloc_planes(B * h, N, N, torch.bfloat16, dev, fill=float("nan"))
    S.dense_to_planes(t, tri.to(dev))
    zd, lib = z.to(dev), _lib.load()
    rd = zd if residual == "z" else None if res is None else res.to(dev)
    dsd = None if ds is None else ds.to(dev)
    errs = []
    for move in (False, True):
        k = dict(kw)
        if move:
            for n in ("ln_in_w", "ln_in_b", "ln_out_w", "ln_out_b"):
                k[n] = shifted(k[n])
        ws, _ = S._weights_struct(c, z.dtype, device=dev, c_hidden=h, c_proj=h, **k)
        desc = _lib.make_desc(B, N, c, c_hidden=h, dtype=_lib.DTYPE_BF16, direction=_lib.OUTGOING, eps_in=w.eps_in,
                              eps_out=w.eps_out, drop_scale=None if dsd is None else dsd.data_ptr())
        out = torch.full_like(zd, float("nan"))
        _lib.check(lib.trimul_b200_tm2(C.byref(desc), zd.data_ptr(), C.byref(t.struct()), C.byref(ws), out.data_ptr(),
                                       None if rd is None else rd.data_ptr(),
                                       torch.cuda.current_stream(dev).cuda_stream, _status_words(dev).data_ptr()), "tm2")
        y = out.cpu().double()
        ref = upd if res is None else upd + d64(res)
        errs.append(float((y - ref).norm() / ref.norm()))
    assert read_status(dev)[0] == 0
    # roundings to bf16 (1.1e-3 rms each): the folded weights or the normalised operands, twice; the output, with a
    # scale and a residual once more each
    assert max(errs) <= 5e-3, errs


@pytest.mark.parametrize("residual", [False, True], ids=["bare", "residual"])
@pytest.mark.parametrize("c,h", [(64, 64), (128, 64), (128, 128), (128, 256), (256, 256)])
def test_stage3_of_a_row_slab_is_that_part_of_the_whole(dev, c, h, residual):
    """Rows 37 .. 126 of 200 with a dropout scale, whose tiles are walked in column order (rows != N): the same bits."""
    from miniworld_engine_b200 import _lib, read_status, stages as S
    from miniworld_engine_b200.functional import _status_words
    import ctypes as C
    B, N, row0, rows = 2, 200, 37, 90
    kw = weights_dict(O.make_weights(c, 91, affine="random", h=h), torch.bfloat16, dev)
    g = torch.Generator().manual_seed(92)
    z = torch.randn(B, N, N, c, generator=g).bfloat16().to(dev)
    tri = torch.randn(B * h, N, N, generator=g).bfloat16().to(dev)
    ds = ((torch.rand(B, 1, N, c, generator=g) > 0.25).float() / 0.75).bfloat16().to(dev)
    ws, _ = S._weights_struct(c, z.dtype, device=dev, c_hidden=h, c_proj=h, **kw)

    def run(first, count):
        zs = z[:, first:first + count].contiguous()
        t = S.alloc_planes(B * h, count, N, torch.bfloat16, dev, fill=float("nan"))
        S.dense_to_planes(t, tri[:, first:first + count])
        desc = _lib.make_desc(B, N, c, c_hidden=h, dtype=_lib.DTYPE_BF16, direction=_lib.OUTGOING, rows=count, row0=first,
                              drop_scale=ds.data_ptr())
        out = torch.full_like(zs, float("nan"))
        _lib.check(_lib.load().trimul_b200_tm2(C.byref(desc), zs.data_ptr(), C.byref(t.struct()), C.byref(ws), out.data_ptr(),
                                               zs.data_ptr() if residual else None,
                                               torch.cuda.current_stream(dev).cuda_stream,
                                               _status_words(dev).data_ptr()), "tm2")
        return out

    whole, slab = run(0, N), run(row0, rows)
    assert read_status(dev)[0] == 0
    assert not torch.isnan(whole.float()).any()
    assert torch.equal(slab, whole[:, row0:row0 + rows])


@pytest.mark.parametrize("single_cta", [False, True], ids=["pair", "lone"])
@pytest.mark.parametrize("c", [64, 128, 256])
def test_stage1_takes_layernorm_vectors_at_any_float_address(dev, c, single_cta):
    """c = h: the same values at an address that is not 16-byte aligned give the same bits."""
    from miniworld_engine_b200 import read_status, stages as S
    B, N = 2, 130
    kw = weights_dict(O.make_weights(c, 51, affine="random"), torch.bfloat16, dev)
    z = O.make_input(B, N, c, 52).bfloat16().to(dev)
    outs = []
    for move in (False, True):
        k = {n: shifted(v) if move and n.startswith("ln_") else v for n, v in kw.items()}
        assert k["ln_in_w"].data_ptr() % 16 == (4 if move else 0)
        a, b = (S.alloc_planes(B * c, N, N, torch.bfloat16, dev, fill=float("nan")) for _ in range(2))
        S.tm1(z, None, k, a, b, outgoing=False, single_cta=single_cta)
        outs.append([S.planes_to_dense(s) for s in (a, b)])
    assert read_status(dev)[0] == 0
    for ref, got in zip(*outs):
        assert not torch.isnan(ref.float()).any() and torch.equal(got, ref)


@pytest.mark.parametrize("c", [64, 128, 256])
def test_a_block_takes_layernorm_vectors_at_any_float_address(dev, c):
    from miniworld_engine_b200 import read_status, trimul_forward
    kw = forward_kwargs(O.make_weights(c, 53, affine="random"), torch.bfloat16, dev)
    z = O.make_input(1, 70, c, 54).bfloat16().to(dev)
    ref, got = (trimul_forward(z, None, outgoing=True, residual=z,
                               **{n: shifted(v) if move and n.startswith("ln_") else v for n, v in kw.items()})
                for move in (False, True))
    assert read_status(dev)[0] == 0
    assert torch.equal(got, ref)


def closed_gates(c, h):
    """Weights whose gate logits are about -15 (sigmoid 3.1e-7): LayerNorm_in has a bias of one, the gate rows a mean of -15/c."""
    w = O.make_weights(c, 61, affine="random", h=h)
    w.ln_pair_weight[:], w.ln_pair_bias[:] = 1.0, 1.0
    g = torch.Generator().manual_seed(62)
    for m in (w.to_left_gate, w.to_right_gate, w.to_gate):
        m.copy_(-15.0 / c + 0.05 * torch.randn(m.shape, generator=g) / c ** 0.5)
    return w.to(torch.bfloat16)


@pytest.mark.parametrize("mask_kind", [None, "pair"])
def test_stage1_keeps_the_bits_of_nearly_shut_gates_at_64_hidden_channels(dev, mask_kind):
    """c = 128, h = 64.  Against the CUDA-core kernel (the same rounding of x_n, expf).  A hardware tanh is off by 6e-8 to 1e-7 of the
    gate's full scale here, which is a fifth to a third of the value."""
    from miniworld_engine_b200 import read_status, stages as S
    B, N = 2, 70
    kw = weights_dict(closed_gates(128, 64), torch.bfloat16, dev)
    z = O.make_input(B, N, 128, 63).bfloat16().to(dev)
    mask = None if mask_kind is None else (torch.rand(B, N, N, generator=torch.Generator().manual_seed(64)) > 0.2).to(dev)

    def run(plain):
        a, b = (S.alloc_planes(B * 64, N, N, torch.bfloat16, dev, fill=float("nan")) for _ in range(2))
        S.tm1(z, mask, kw, a, b, outgoing=True, plain_kernels=plain)
        return S.planes_to_dense(a).float().cpu(), S.planes_to_dense(b).float().cpu()

    for got, ref in zip(run(False), run(True)):
        # one rounding to bf16 each (1.1e-3 rms of the value) and now and then another rounding of an x_n
        assert 0 < float(ref.abs().max()) < 1e-3
        assert O.rel_rms(got, ref) <= 4e-3
    assert read_status(dev)[0] == 0


@pytest.mark.parametrize("scale", [False, True], ids=["bare", "scaled"])
def test_stage3_keeps_the_bits_of_nearly_shut_gates_at_64_hidden_channels(dev, scale):
    """c = 128, h = 64, against the stage in 64 bits on the same bf16 operands."""
    from miniworld_engine_b200 import _lib, read_status, stages as S
    from miniworld_engine_b200.functional import _status_words
    import ctypes as C
    B, N, c, h = 1, 130, 128, 64
    w = closed_gates(c, h)
    kw = weights_dict(w, torch.bfloat16, dev)
    g = torch.Generator().manual_seed(65)
    z = torch.randn(B, N, N, c, generator=g).bfloat16()
    tri = torch.randn(B * h, N, N, generator=g).bfloat16()
    ds = ((torch.rand(B, 1, N, c, generator=g) > 0.25).float() / 0.75).bfloat16()
    ln = lambda x, gm, bt, eps: torch.nn.functional.layer_norm(x, x.shape[-1:], gm.double(), bt.double(), eps)
    zn = ln(z.double(), w.ln_pair_weight, w.ln_pair_bias, w.eps_in)
    tn = ln(tri.double().view(B, h, N, N).permute(0, 2, 3, 1), w.ln_out_weight, w.ln_out_bias, w.eps_out)
    ref = torch.sigmoid(zn @ w.to_gate.double().T) * (tn @ w.to_out.double().T)
    if scale:
        ref = ref * ds.double()
    t = S.alloc_planes(B * h, N, N, torch.bfloat16, dev, fill=float("nan"))
    S.dense_to_planes(t, tri.to(dev))
    zd, dsd = z.to(dev), ds.to(dev)
    ws, _ = S._weights_struct(c, z.dtype, device=dev, c_hidden=h, c_proj=h, **kw)
    desc = _lib.make_desc(B, N, c, c_hidden=h, dtype=_lib.DTYPE_BF16, direction=_lib.OUTGOING, eps_in=w.eps_in,
                          eps_out=w.eps_out, drop_scale=dsd.data_ptr() if scale else None)
    out = torch.full_like(zd, float("nan"))
    _lib.check(_lib.load().trimul_b200_tm2(C.byref(desc), zd.data_ptr(), C.byref(t.struct()), C.byref(ws), out.data_ptr(),
                                           None, torch.cuda.current_stream(dev).cuda_stream,
                                           _status_words(dev).data_ptr()), "tm2")
    # roundings to bf16 of the folded weights (in the logit 15 * 1.1e-3 / sqrt(c), in the projection 1.1e-3), of the output and
    # of the scaled output
    assert read_status(dev)[0] == 0
    assert float((out.cpu().double() - ref).norm() / ref.norm()) <= 5e-3


@pytest.mark.parametrize("residual", [None, "z", "other"])
@pytest.mark.parametrize("c,h", [(256, 256), (128, 64), (128, 256)])
def test_stage3_with_the_layernorms_in_place_on_request(dev, c, h, residual):
    """The flag's rounding points (LN(x) to bf16, unchanged weights) are those of the CUDA-core kernel: the outputs are the same
    but for values that lie on a rounding boundary.  Folded weights (another rounding of every product) change far more."""
    from miniworld_engine_b200 import read_status, stages as S
    B, N = 2, 70
    kw = weights_dict(O.make_weights(c, 71, affine="random", h=h), torch.bfloat16, dev)
    g = torch.Generator().manual_seed(72)
    z = torch.randn(B, N, N, c, generator=g).bfloat16().to(dev)
    t = S.alloc_planes(B * h, N, N, torch.bfloat16, dev, fill=float("nan"))
    S.dense_to_planes(t, torch.randn(B * h, N, N, generator=g).bfloat16().to(dev))
    res = {None: None, "z": z, "other": torch.randn(B, N, N, c, generator=g).bfloat16().to(dev)}[residual]
    plain = S.tm2(z, t, kw, residual=res, plain_kernels=True)
    asked = S.tm2(z, t, kw, residual=res, inplace_norm=True)
    assert read_status(dev)[0] == 0
    # fp32 sums in another order differ by about 1e-6 of the value and a bf16 step is 4e-3 of it: a few in ten thousand of
    # the roundings of LN(x), and of the outputs, go the other way
    assert (asked != plain).float().mean() <= 0.02


@pytest.mark.parametrize("outgoing", [True, False], ids=["outgoing", "incoming"])
def test_stage1_leaves_what_is_past_a_ragged_last_chunk_alone(dev, outgoing):
    """c = 128, h = 64, column chunks of 64 over 100 columns: the last chunk holds 36."""
    from miniworld_engine_b200 import read_status, stages as S
    B, N = 1, 100
    kw = weights_dict(O.make_weights(128, 81, affine="random", h=64), torch.bfloat16, dev)
    z = O.make_input(B, N, 128, 82).bfloat16().to(dev)
    outs = []
    for layout in ({}, dict(col_chunk=64)):
        a, b = (S.alloc_planes(B * 64, N, N, torch.bfloat16, dev, fill=float("nan"), **layout) for _ in range(2))
        S.tm1(z, None, kw, a, b, outgoing=outgoing)
        outs.append([S.planes_to_dense(s).float().cpu() for s in (a, b)])
        if layout:
            for s in (a, b):
                last = s.buf[s.chunk_stride:].view(64, N, s.pitch)
                assert torch.isnan(last[..., N - 64:]).all()
    assert read_status(dev)[0] == 0
    for ref, got in zip(*outs):
        assert not torch.isnan(got).any()
        assert O.rel_rms(got, ref) <= 4e-3      # two kernels, the same rounding points
