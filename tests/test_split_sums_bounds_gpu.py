"""Layers whose sum over K is made in segments against double precision, with every storage type and a bound for each."""
import pytest

import test_conv_tc_gpu as tc
import test_split_sums_gpu as split

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["by the plan", "in turn"])
@pytest.mark.parametrize("storage", ["fp32", "bf16_in", "bf16_in_out"])
@pytest.mark.parametrize("case", split.CASES, ids=[c[0] for c in split.CASES])
def test_segments_match_double(kernels, case, storage, form):
    name, n, c, h, w, cout, k, stride, pad, dil, with_res, act = case
    half, half_out = storage != "fp32", storage == "bf16_in_out"
    act = min(act, 1) if half else act
    g = torch.Generator().manual_seed(42)
    x = torch.randn((n, c, h, w), generator=g)
    wt = torch.randn((cout, c, k, k), generator=g) * (2.0 / (c * k * k)) ** 0.5
    ho, wo = (h + 2 * pad - dil * (k - 1) - 1) // stride + 1, (w + 2 * pad - dil * (k - 1) - 1) // stride + 1
    res = torch.randn((n, cout, ho, wo), generator=g) if with_res else None
    kw = dict(stride=stride, pad=pad, dil=dil, scale=torch.rand(cout, generator=g) + 0.5, shift=torch.randn(cout, generator=g))
    prelu = torch.linspace(0.1, 0.3, cout) if act == 2 else None
    if half:
        x, wt = x.bfloat16().float(), wt.bfloat16().float()
        res = res.bfloat16().float() if with_res else None

    def run():
        if half:
            return tc.run_conv_bf16(kernels, x, wt, out_bf16=half_out, residual=res, act=act, **kw)[0]
        return tc.run_conv(kernels, x.cuda(), wt, residual=res, act=act, prelu=prelu, **kw)[0]

    got = split._run({"MCB200_SPLIT": "0"}, run) if form == "in turn" else run()
    want = tc.reference(x, wt, residual=res, res_coeff=1.0, act=act, slope=0.0, prelu=prelu, **kw)
    # The sums' deviation is sqrt(2) whatever K.  TF32 operands, as for shorter sums: 5.6e-4 of that, 8.5e-4 behind the scale,
    # of which 2^-7 is nine times, and the cut takes up to 2^-10 of the result.  bfloat16 operands are exact here: what is
    # left are fp32 sums, of at most 4608 products a segment, added up sixteen at a time: 288 additions, each off by 2^-23 of a
    # partial sum of at most 6, behind a scale of 1.5: 3.1e-4, less than 2^-11.  A result in bfloat16 adds 2^-9 of itself.
    err = (got.float().cpu() - want).abs()
    bound = (2.0 ** -11 if half else 2.0 ** -7) + ((2.0 ** -8 if half_out else 0) + (2.0 ** -14 if half else 2.0 ** -10)) * want.abs()
    assert torch.isfinite(got).all() and (err <= bound).all(), float((err - bound).max())
