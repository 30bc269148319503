"""The two ways results leave the convolution kernel, straight from registers and as staged TMA tiles: the same bits, at the
edges of tiles, chunks and column groups, for every storage type (other tests compare the staged form with double precision)."""
import os

import pytest

import test_conv_tc_gpu as tc

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

CASES = [
    # name, N, C, H, W, Cout, k, tile width, pair, residual, activation
    ("one_row", 1, 32, 1, 1, 8, 1, 64, "0", True, 1),
    ("rows_127", 1, 64, 127, 1, 64, 1, 64, "0", True, 0),
    ("rows_129_ragged_groups", 1, 64, 43, 3, 72, 1, 64, "0", True, 2),       # 72 = a tile and one group of eight
    ("last_chunk_of_eight", 2, 32, 11, 13, 136, 1, 128, "0", False, 1),
    ("second_warp_without_chunk", 1, 64, 12, 12, 24, 3, 256, "0", True, 1),
    ("wide_3x3", 1, 64, 18, 18, 256, 3, 256, "0", True, 1),
    ("pair_odd_tiles", 1, 256, 19, 19, 256, 3, 128, "1", True, 1),
    ("persistent", 4, 64, 80, 80, 64, 1, 64, "0", True, 1),                  # 200 tiles: the residual of the next tile
]


def _with(staged, block_n, pair, fn):
    env = {"MCB200_STAGED": staged, "MCB200_BLOCK_N": str(block_n), "MCB200_CTA_PAIR": pair, "MCB200_HALO": "0",
           "MCB200_BLOCK_M": "128"}
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
def test_both_ways_out_give_the_same_bits(kernels, case, storage):
    name, n, c, h, w, cout, k, block_n, pair, with_res, act = case
    g = torch.Generator().manual_seed(31)
    x = torch.randn((n, c, h, w), generator=g)
    wt = torch.randn((cout, c, k, k), generator=g) * (2.0 / (c * k * k)) ** 0.5
    kw = dict(stride=1, pad=k // 2, dil=1, scale=torch.rand(cout, generator=g) + 0.5, shift=torch.randn(cout, generator=g),
              residual=torch.randn((n, cout, h, w), generator=g) if with_res else None, act=act)
    if storage == "fp32":
        kw.update(prelu=torch.rand(cout, generator=g) if act == 2 else None)
        run = lambda: tc.run_conv(kernels, x.cuda(), wt, **kw)
    else:
        kw.update(act=min(act, 1))
        run = lambda: tc.run_conv_bf16(kernels, x, wt, out_bf16=storage == "bf16_in_out", **kw)
    staged, plan = _with("1", block_n, pair, run)
    direct, _ = _with("0", block_n, pair, run)
    assert plan.block_n == block_n and plan.cta_pair == int(pair)
    assert torch.isfinite(direct).all() and torch.equal(staged, direct)
