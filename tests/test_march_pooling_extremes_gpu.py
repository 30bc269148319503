"""The pooling in the march's store against the pooling kernels on the march's own unpooled result, where windows hold nothing
but -infinity, NaN or the lowest value: the same bits."""
import ctypes

import pytest

import test_conv_march_gpu as tm

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("act,slope", [(0, 0.0), (1, 0.1), (1, 0.0)], ids=["none", "leaky", "relu"])
@pytest.mark.parametrize("cout,storage", [(64, "fp32"), (64, "bf16"), (40, "bf16"), (36, "fp32"), (42, "fp32"), (33, "fp32")])
@pytest.mark.parametrize("size", [(2, 56, 56), (3, 7, 61), (1, 1, 49), (1, 9, 121)], ids=str)
def test_windows_without_an_ordinary_value(kernels, size, cout, storage, act, slope):
    n, h, w = size
    half = int(storage == "bf16")
    g = torch.Generator().manual_seed(53)
    x = torch.randn((n, 64, h, w), generator=g)
    wt = torch.randn((cout, 64, 3, 3), generator=g) * 0.06
    shift = torch.randn(cout, generator=g)
    shift[0:32:4] = float("-inf")
    shift[1:32:4] = float("nan")
    shift[2:32:8] = float("inf")
    shift[6] = torch.finfo(torch.bfloat16 if half else torch.float32).min
    x[-1, 0, h // 2, w // 2] = float("nan")      # three windows or fewer with ordinary neighbours
    x[-1, 0, 0, 0] = float("-inf")
    kw = dict(in_bf16=half, out_bf16=half, scale=None, shift=shift, act=act, slope=slope, prelu=None)
    whole = tm.march(kernels, x, wt, **kw).permute(0, 2, 3, 1).contiguous()
    oh, ow = (h + 1) // 2, (w + 1) // 2
    if half:
        whole = whole.bfloat16().contiguous()
    want = torch.empty((n, oh, ow, cout), device="cuda", dtype=whole.dtype)
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    if half:
        rc = kernels.mcb200_pool_max_nhwc_bf16(p(whole), p(want), n, h, w, cout, 2, 2, 2, 2, 0, 0, oh, ow, None)
    else:
        rc = kernels.mcb200_pool_nhwc(p(whole), p(want), n, h, w, cout, 2, 2, 2, 2, 0, 0, oh, ow, 0, None)
    assert rc == 0, rc
    torch.cuda.synchronize()
    got = tm.march(kernels, x, wt, pool=1, **kw).permute(0, 2, 3, 1).contiguous()
    want = want.float()
    assert torch.equal(got.isnan(), want.isnan())
    assert torch.equal(got.nan_to_num(nan=7.0, posinf=float("inf"), neginf=float("-inf")),
                       want.nan_to_num(nan=7.0, posinf=float("inf"), neginf=float("-inf")))
