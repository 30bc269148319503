"""Layers whose sum over K is made in segments: a cluster of CTAs that makes them side by side, one CTA that makes them one
after the other and the tiles of a large batch give the same bits, and they are what double precision gives."""
import os

import pytest

import test_conv_tc_gpu as tc

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

CASES = [
    # name, N, C, H, W, Cout, k, stride, pad, dil, residual, activation
    ("inner_product", 1, 2048, 1, 1, 1000, 1, 1, 0, 1, False, 0),
    ("odd_columns", 3, 1088, 1, 1, 21, 1, 1, 0, 1, False, 2),            # 34 k-blocks in four segments, 3 rows, 21 columns
    ("matrix_14", 1, 1024, 14, 14, 256, 1, 1, 0, 1, True, 1),
    ("matrix_7_many", 5, 2048, 7, 7, 520, 1, 1, 0, 1, True, 1),          # 245 rows, last tile of eight columns
    ("im2col_14", 1, 256, 14, 14, 256, 3, 1, 1, 1, False, 1),
    ("im2col_stride", 2, 120, 13, 11, 72, 3, 2, 1, 1, True, 2),          # 36 k-blocks, the last of each tap with 24 channels
    ("one_by_one_stride", 1, 1024, 14, 14, 512, 1, 2, 0, 1, False, 1),
    ("halo_7", 1, 512, 7, 7, 512, 3, 1, 1, 1, False, 1),
    ("halo_19", 1, 1024, 19, 19, 24, 3, 1, 1, 1, True, 1),
    ("halo_19_126", 1, 256, 19, 19, 126, 3, 1, 1, 1, False, 0),
    ("im2col_dilated", 1, 160, 19, 19, 320, 3, 1, 6, 6, False, 1),
]


def _run(env, fn):
    saved = {k: os.environ.get(k) for k in env}
    os.environ.update(env)
    try:
        return fn()
    finally:
        for k, v in saved.items():
            if v is None:
                del os.environ[k]
            else:
                os.environ[k] = v


@pytest.mark.parametrize("storage", ["fp32", "bf16_in", "bf16_in_out"])
@pytest.mark.parametrize("case", CASES, ids=[c[0] for c in CASES])
def test_segments_side_by_side_and_in_turn(kernels, case, storage):
    name, n, c, h, w, cout, k, stride, pad, dil, with_res, act = case
    g = torch.Generator().manual_seed(41)
    large = 24
    x = torch.randn((large, c, h, w), generator=g)
    wt = torch.randn((cout, c, k, k), generator=g) * (2.0 / (c * k * k)) ** 0.5
    ho, wo = (h + 2 * pad - dil * (k - 1) - 1) // stride + 1, (w + 2 * pad - dil * (k - 1) - 1) // stride + 1
    res = torch.randn((large, cout, ho, wo), generator=g) if with_res else None
    kw = dict(stride=stride, pad=pad, dil=dil, scale=torch.rand(cout, generator=g) + 0.5, shift=torch.randn(cout, generator=g))

    def run(images):
        r = res[:images] if with_res else None
        if storage == "fp32":
            return tc.run_conv(kernels, x[:images].cuda(), wt, residual=r, act=act,
                               prelu=torch.linspace(0.1, 0.3, cout) if act == 2 else None, **kw)[0]
        return tc.run_conv_bf16(kernels, x[:images], wt, out_bf16=storage == "bf16_in_out", residual=r, act=min(act, 1), **kw)[0]

    split = run(n)
    in_turn = _run({"MCB200_SPLIT": "0"}, lambda: run(n))
    assert torch.isfinite(split).all() and torch.equal(split, in_turn)
    assert torch.equal(run(large)[:n], split)
    if storage == "fp32":
        want = tc.reference(x[:n], wt, residual=res[:n] if with_res else None, res_coeff=1.0, act=act, slope=0.0,
                            prelu=torch.linspace(0.1, 0.3, cout) if act == 2 else None, **kw)
        err = (split.cpu() - want).abs()
        assert (err <= 2e-2 + 1e-2 * want.abs()).all(), float(err.max())
