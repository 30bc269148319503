"""Two layers in one launch whose results leave through shared memory: the bits of the launch that stores from registers and of
each layer in a launch of its own, where tiles hold columns of both, of one, and of neither (the zero columns between)."""
import ctypes
import os

import pytest

import test_conv_tc_gpu as tc

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


class Second(ctypes.Structure):
    _fields_ = [("begin", ctypes.c_int), ("first_cout", ctypes.c_int), ("out", ctypes.c_void_p), ("out_ld", ctypes.c_int),
                ("act", ctypes.c_int)]


CASES = [
    # name, N, C, H, W, first columns, second columns, k, tile width, pair
    ("tile_of_both", 1, 64, 11, 13, 40, 24, 1, 64, "0"),             # first columns 0-39, zeros to 63; the second tile the other's
    ("chunk_by_chunk", 2, 96, 15, 9, 32, 96, 1, 128, "0"),           # a tile whose chunks alternate between warps and layers
    ("one_wide_tile", 3, 64, 20, 20, 8, 200, 1, 256, "0"),           # 24 zero columns behind eight
    ("im2col", 2, 32, 14, 15, 72, 56, 3, 128, "0"),                  # first ends in the second chunk group of a tile
    ("pair", 1, 256, 19, 19, 136, 120, 3, 128, "1"),                 # odd M tiles
    ("pair_wide", 4, 64, 20, 20, 256, 64, 1, 256, "1"),              # one layer per tile
    ("persistent", 4, 32, 90, 90, 16, 48, 1, 64, "0"),               # 507 tiles
]


def _run(L, x, wt, first, second, k, half, half_out, acts, tail, staged, block_n, pair, both):
    """Output of the first and the second layer: from one launch of two (both) or from a launch each."""
    sfx = "_bf16" if half else ""
    count = getattr(L, "mcb200_conv_packed_weight_count" + sfx)
    count.restype = ctypes.c_size_t
    n, c, h, w = x.shape
    dt, odt = (torch.bfloat16 if f else torch.float32 for f in (half, half_out))
    nhwc = x.permute(0, 2, 3, 1).contiguous().cuda().to(dt)
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    begin = (first + 31) // 32 * 32
    env = {"MCB200_STAGED": staged, "MCB200_BLOCK_N": str(block_n), "MCB200_CTA_PAIR": pair, "MCB200_HALO": "0", "MCB200_BLOCK_M": "128"}
    saved = {key: os.environ.get(key) for key in env}
    os.environ.update(env)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    try:
        def launch(weights, scale, shift, act, out, two):
            s = tc.ConvShape(n, h, w, c, c, weights.shape[0], k, k, 1, 1, k // 2, k // 2, 1, 1, 1, 0, 0)
            assert L.mcb200_conv_out_shape(ctypes.byref(s)) == 0
            wdev, sc, sh = weights.contiguous().cuda(), scale.cuda(), shift.cuda()
            packed = torch.empty(count(ctypes.byref(s)), device="cuda", dtype=dt)
            assert getattr(L, "mcb200_conv_pack_weights" + sfx)(ctypes.byref(s), p(wdev), p(packed), None) == 0
            plan = tc.aligned_plan()
            assert getattr(L, "mcb200_conv_tc_plan" + sfx)(ctypes.byref(s), p(nhwc), p(packed), ctypes.byref(plan)) == 0
            if two:
                assert plan.block_n == block_n and plan.cta_pair == int(pair)
            ep = tc.Epilogue()
            ep.residual_coeff, ep.act, ep.scale, ep.shift = 1.0, act, sc.data_ptr(), sh.data_ptr()
            if two:
                more = Second(begin, first, out[1].data_ptr(), second, acts[1])
                rc = L.mcb200_conv_tc_launch_two(ctypes.byref(plan), p(out[0]), int(half_out), first, ctypes.byref(ep),
                                                 ctypes.byref(more), 0, p(status), None)
            else:
                rc = L.mcb200_conv_tc_launch_flags(ctypes.byref(plan), p(out[0]), int(half_out), weights.shape[0], ctypes.byref(ep), 0,
                                                   p(status), None)
            assert rc == 0, rc
            torch.cuda.synchronize()
            assert int(status.item()) == 0

        out = [torch.full((n, h, w, m), float("nan"), device="cuda", dtype=odt) for m in (first, second)]
        if both:
            weights = torch.zeros((begin + second,) + wt.shape[1:])
            weights[:first], weights[begin:] = wt[:first], wt[first:]
            scale, shift = torch.ones(begin + second), torch.zeros(begin + second)
            for whole, part in ((scale, tail[0]), (shift, tail[1])):
                whole[:first], whole[begin:] = part[:first], part[first:]
            launch(weights, scale, shift, acts[0], out, True)
        else:
            launch(wt[:first], tail[0][:first], tail[1][:first], acts[0], out[:1], False)
            launch(wt[first:], tail[0][first:], tail[1][first:], acts[1], out[1:], False)
        return out
    finally:
        for key, v in saved.items():
            if v is None:
                del os.environ[key]
            else:
                os.environ[key] = v


@pytest.mark.parametrize("acts", [(1, 0), (0, 1)], ids=["relu_first", "relu_second"])
@pytest.mark.parametrize("storage", ["fp32", "bf16_in", "bf16_in_out"])
@pytest.mark.parametrize("case", CASES, ids=[c[0] for c in CASES])
def test_two_layers_staged_and_from_registers(kernels, case, storage, acts):
    name, n, c, h, w, first, second, k, block_n, pair = case
    half, half_out = storage != "fp32", storage == "bf16_in_out"
    g = torch.Generator().manual_seed(81)
    x = torch.randn((n, c, h, w), generator=g)
    wt = torch.randn((first + second, c, k, k), generator=g) * (2.0 / (c * k * k)) ** 0.5
    tail = torch.rand(first + second, generator=g) + 0.5, torch.randn(first + second, generator=g)
    run = lambda staged, both: _run(kernels, x, wt, first, second, k, half, half_out, acts, tail, staged, block_n, pair, both)
    staged, direct, alone = run("1", True), run("0", True), run("0", False)
    for a, b, want in zip(staged, direct, alone):
        assert torch.isfinite(want).all()
        assert torch.equal(a, b) and torch.equal(a, want)
