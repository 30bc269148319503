"""3 x 3 layers of 33 to 64 channels that march down the image (conv_march.cu): against double precision at the edges of slabs,
columns and runs, with every storage type, and an image alone gives the bits it has in a batch."""
import ctypes

import pytest

import test_conv_tc_gpu as tc

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


class MarchPlan(ctypes.Structure):
    _fields_ = [("tma_a", ctypes.c_uint64 * 16), ("tma_b", ctypes.c_uint64 * 16), ("shape", tc.ConvShape),
                ("operand_bf16", ctypes.c_int), ("segments", ctypes.c_int), ("segment_w", ctypes.c_int), ("column_h", ctypes.c_int),
                ("pad_top", ctypes.c_int), ("total", ctypes.c_int), ("pool", ctypes.c_int)]


def march(L, x, w, *, in_bf16, out_bf16, scale, shift, act, slope, prelu, pool=0):
    n, c, h, wd = x.shape
    cout = w.shape[0]
    s = tc.ConvShape(n, h, wd, c, c, cout, 3, 3, 1, 1, 1, 1, 1, 1, 1, 0, 0)
    L.mcb200_conv_march_packed_weight_bytes.restype = ctypes.c_size_t
    packed = torch.empty(L.mcb200_conv_march_packed_weight_bytes(ctypes.byref(s), in_bf16), dtype=torch.uint8, device="cuda")
    wdev = w.contiguous().cuda()
    assert L.mcb200_conv_march_pack_weights(ctypes.byref(s), in_bf16, ctypes.c_void_p(wdev.data_ptr()),
                                            ctypes.c_void_p(packed.data_ptr()), None) == 0
    nhwc = x.permute(0, 2, 3, 1).contiguous().cuda().to(torch.bfloat16 if in_bf16 else torch.float32)
    raw = ctypes.create_string_buffer(ctypes.sizeof(MarchPlan) + 128)
    plan = MarchPlan.from_address((ctypes.addressof(raw) + 63) & ~63)
    rc = L.mcb200_conv_march_plan(ctypes.byref(s), in_bf16, ctypes.c_void_p(nhwc.data_ptr()), ctypes.c_void_p(packed.data_ptr()),
                                  pool, ctypes.byref(plan))
    assert rc == 0, rc
    if pool:
        h, wd = (h + 1) // 2, (wd + 1) // 2
    out = torch.full((n, h, wd, cout), float("nan"), device="cuda", dtype=torch.bfloat16 if out_bf16 else torch.float32)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    ep = tc.Epilogue()
    ep.residual_coeff, ep.act, ep.slope = 1.0, act, slope
    keep = [t.cuda() if t is not None else None for t in (scale, shift, prelu)]
    for name, t in zip(("scale", "shift", "prelu"), keep):
        if t is not None:
            setattr(ep, name, t.data_ptr())
    for flags in (0, 1):
        rc = L.mcb200_conv_march_launch(ctypes.byref(plan), ctypes.c_void_p(out.data_ptr()), out_bf16, cout, ctypes.byref(ep), flags,
                                        ctypes.c_void_p(status.data_ptr()), None)
        assert rc == 0, rc
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    return out.permute(0, 3, 1, 2).float()


CASES = [
    # name, N, C, H, W, Cout, activation, negative slope
    ("one_image_56", 1, 64, 56, 56, 64, 1, 0.0),
    ("one_row", 3, 64, 1, 48, 64, 0, 0.0),
    ("widest_slab", 2, 64, 7, 62, 64, 1, 0.1),
    ("five_columns", 2, 64, 9, 300, 64, 1, 0.0),
    ("ragged_last_column", 1, 36, 33, 121, 48, 2, 0.0),              # two columns of 61 and 60, 36 of 64 channels
    ("odd_channels_out", 2, 40, 12, 55, 33, 1, 0.0),                 # element-wise stores
    ("long_runs", 24, 64, 56, 56, 64, 1, 0.0),                       # five rows a slab: accumulators in turn
    ("many_rows_a_slab", 6, 64, 300, 180, 64, 1, 0.0),               # eighteen rows a slab, all slots twice
]


@pytest.mark.parametrize("storage", ["fp32", "fp32_to_bf16", "bf16_to_fp32", "bf16"])
@pytest.mark.parametrize("case", CASES, ids=[c[0] for c in CASES])
def test_march_matches_double(kernels, case, storage):
    name, n, c, h, w, cout, act, slope = case
    in_bf16, out_bf16 = int(storage.startswith("bf16")), int(storage in ("bf16", "fp32_to_bf16"))
    if in_bf16:
        c = (c + 7) // 8 * 8
    g = torch.Generator().manual_seed(51)
    x = torch.randn((n, c, h, w), generator=g)
    wt = torch.randn((cout, c, 3, 3), generator=g) * (2.0 / (9 * c)) ** 0.5
    kw = dict(scale=torch.rand(cout, generator=g) + 0.5, shift=torch.randn(cout, generator=g), act=act, slope=slope,
              prelu=torch.rand(cout, generator=g) * 0.3 if act == 2 else None)
    got = march(kernels, x, wt, in_bf16=in_bf16, out_bf16=out_bf16, **kw)
    assert torch.isfinite(got).all()
    if in_bf16:
        x, wt = x.bfloat16().float(), wt.bfloat16().float()
    alone = march(kernels, x[n - 1:], wt, in_bf16=in_bf16, out_bf16=out_bf16, **kw)
    assert torch.equal(alone, got[n - 1:])
    # The general kernel's halo mode makes the same sums: which of the two runs may depend on the batch.
    tail = dict(scale=kw["scale"], shift=kw["shift"], act=act)
    if in_bf16 and act == 1 and slope == 0.0:
        other = tc._with_planner(64, "0", lambda: tc.run_conv_bf16(kernels, x[n - 1:], wt, out_bf16=bool(out_bf16), pad=1, **tail)[0], halo="1")
        assert torch.equal(other.float().cpu(), alone.cpu())
    elif storage == "fp32":
        other, plan = tc._with_planner(64, "0", lambda: tc.run_conv(kernels, x[n - 1:].cuda(), wt, pad=1, slope=slope, prelu=kw["prelu"], **tail),
                                       halo="1")
        assert plan.im2col == 3 and torch.equal(other.cpu(), alone.cpu())
    if n * h * w > 100000:      # the last image stands for the batch
        got, x = got[n - 1:], x[n - 1:]
    want = tc.reference(x, wt, stride=1, pad=1, dil=1, residual=None, res_coeff=1.0, **kw)
    # TF32 operands have 10 bits: cut off (activations) or rounded (weights), their errors spread by 2^-10 / sqrt(12) of a
    # product each, 5.6e-4 of the results' sqrt(2) together, 8.5e-4 behind the scale: 2^-7 is nine times that; the cut
    # also takes up to 2^-10 of the result.  bfloat16 values are exact here, which leaves fp32 sums of 576
    # products; a result stored as bfloat16 adds 2^-9 of itself.
    err = (got.cpu() - want).abs()
    bound = (2.0 ** -14 if in_bf16 else 2.0 ** -7) + ((2.0 ** -8 if out_bf16 else 0) + (2.0 ** -14 if in_bf16 else 2.0 ** -10)) * want.abs()
    assert (err <= bound).all(), float((err - bound).max())


@pytest.mark.parametrize("storage", ["fp32", "bf16"])
@pytest.mark.parametrize("size", [(1, 56, 56), (2, 9, 61), (3, 7, 121), (2, 1, 49), (5, 30, 300), (40, 48, 48)], ids=str)
def test_march_with_pooling_is_march_then_pooling(kernels, size, storage):
    """Odd heights and widths (windows cut at the last row and pixel), single rows, several columns: the same bits as
    pooling the unpooled result."""
    n, h, w = size
    half = int(storage == "bf16")
    g = torch.Generator().manual_seed(52)
    x = torch.randn((n, 64, h, w), generator=g)
    wt = torch.randn((64, 64, 3, 3), generator=g) * 0.06
    for act in (0, 1):
        kw = dict(in_bf16=half, out_bf16=half, scale=None, shift=torch.randn(64, generator=g), act=act, slope=0.0, prelu=None)
        want = torch.nn.functional.max_pool2d(march(kernels, x, wt, **kw), 2, 2, ceil_mode=True)
        assert torch.equal(march(kernels, x, wt, pool=1, **kw), want)


def test_march_leaves_other_layers_alone(kernels):
    """Rows that would leave more than a quarter of the slabs empty, too few rows for all of them, other filters and counts."""
    for n, c, h, w, cout, k, stride, pad, want in (
            (64, 64, 56, 56, 64, 3, 1, 1, 1), (64, 64, 40, 40, 64, 3, 1, 1, 0), (64, 64, 63, 63, 64, 3, 1, 1, 0),
            (64, 32, 56, 56, 64, 3, 1, 1, 0), (64, 64, 56, 56, 65, 3, 1, 1, 0), (64, 64, 56, 56, 64, 3, 2, 1, 0),
            (64, 64, 56, 56, 64, 1, 1, 0, 0), (64, 64, 56, 56, 64, 3, 1, 0, 0), (1, 64, 300, 300, 64, 3, 1, 1, 1),
            (1, 64, 56, 56, 64, 3, 1, 1, 0)):
        s = tc.ConvShape(n, h, w, c, c, cout, k, k, stride, stride, pad, pad, 1, 1, 1, 0, 0)
        assert kernels.mcb200_conv_march_pays(ctypes.byref(s), 0) == want, (n, c, h, w, cout, k, stride, pad)
