"""64-row M tiles (tcgen05.mma at M = 64, 64 or 32 columns) cut a layer up differently and sum in the same order:
the same bits as 128-row tiles of 64 columns, which the other tests compare with double precision."""
import os

import pytest

import test_conv_tc_gpu as tc

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

CASES = [
    # name, N, C, H, W, Cout, k, stride, pad, dil, residual, halo
    ("one_pixel", 1, 64, 1, 1, 8, 1, 1, 0, 1, False, "0"),
    ("edge_64", 1, 64, 8, 8, 64, 1, 1, 0, 1, True, "0"),
    ("edge_65", 1, 64, 5, 13, 32, 1, 1, 0, 1, True, "0"),
    ("ragged_columns", 2, 96, 7, 7, 72, 1, 1, 0, 1, True, "0"),
    ("many_chunks", 1, 512, 14, 14, 1000, 1, 1, 0, 1, True, "0"),
    ("im2col_3x3", 1, 128, 14, 14, 96, 3, 1, 1, 1, True, "0"),
    ("im2col_stride2", 3, 64, 15, 11, 40, 3, 2, 1, 1, False, "0"),
    ("one_by_one_stride2", 1, 64, 14, 14, 64, 1, 2, 0, 1, False, "0"),
    ("plain_stores", 1, 32, 9, 11, 21, 3, 1, 1, 1, True, "0"),
    ("persistent", 8, 32, 40, 40, 64, 3, 1, 1, 1, True, "0"),        # more tiles than SMs: both accumulators in turn
    ("halo_7", 1, 512, 7, 7, 512, 3, 1, 1, 1, False, "1"),           # 63 virtual positions: one tile
    ("halo_19", 2, 64, 19, 19, 24, 3, 1, 1, 1, True, "1"),
    ("halo_dilated", 1, 64, 19, 19, 64, 3, 1, 6, 6, False, "1"),
    ("halo_5x5", 1, 32, 20, 17, 66, 5, 1, 2, 1, True, "1"),
]


def _with(block_m, block_n, halo, fn):
    env = {"MCB200_BLOCK_M": block_m, "MCB200_BLOCK_N": block_n, "MCB200_CTA_PAIR": "0", "MCB200_HALO": halo}
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


@pytest.mark.parametrize("half", [False, True], ids=["tf32", "bf16"])
@pytest.mark.parametrize("case", CASES, ids=[c[0] for c in CASES])
def test_small_tiles_give_the_same_bits(kernels, case, half):
    name, n, c, h, w, cout, k, stride, pad, dil, with_res, halo = case
    g = torch.Generator().manual_seed(17)
    x = torch.randn((n, c, h, w), generator=g)
    wt = torch.randn((cout, c, k, k), generator=g) * (2.0 / (c * k * k)) ** 0.5
    ho, wo = (h + 2 * pad - dil * (k - 1) - 1) // stride + 1, (w + 2 * pad - dil * (k - 1) - 1) // stride + 1
    kw = dict(stride=stride, pad=pad, dil=dil, scale=torch.rand(cout, generator=g) + 0.5,
              shift=torch.randn(cout, generator=g), act=1,
              residual=torch.randn((n, cout, ho, wo), generator=g) if with_res else None)

    def run(out_bf16):
        if half:
            return tc.run_conv_bf16(kernels, x, wt, out_bf16=out_bf16, **kw)
        return tc.run_conv(kernels, x.cuda(), wt, **kw)

    for out_bf16 in ((False, True) if half else (False,)):
        base, plan = _with("128", "64", halo, lambda: run(out_bf16))
        assert plan.block_n == 64 and plan.strip_rows in (0, 128 + (k - 1) * dil)
        for width in ("64", "32"):
            got, plan = _with("64", width, halo, lambda: run(out_bf16))
            assert plan.block_n == int(width) and plan.cta_pair == 0
            assert plan.strip_rows == 64 + ((k - 1) * dil if plan.im2col == 3 else 0)
            assert torch.isfinite(got).all() and torch.equal(got, base), (width, float((got - base).abs().max()))


def test_planner_cuts_the_layers_of_one_image(kernels):
    """Without overrides: small layers run in small tiles, large ones do not, and halo mode stays a matter of geometry."""
    for n, c, hw, cout, k, rows in ((1, 256, 14, 256, 3, 64), (1, 512, 7, 512, 3, 66), (1, 1024, 14, 256, 1, 64),
                                    (64, 256, 14, 256, 3, 0), (64, 64, 56, 256, 1, 0)):
        x = torch.zeros((n, c, hw, hw), device="cuda")
        _, plan = tc.run_conv(kernels, x, torch.zeros((cout, c, k, k)), stride=1, pad=k // 2, dil=1)
        assert plan.strip_rows == rows, (n, c, hw, cout, k, plan.strip_rows, plan.block_n)
