"""One launch plan for launches of two layers, of one layer and of one with a residual, to the same addresses: the tile maps
cached in the plan have to follow."""
import ctypes

import pytest

import test_conv_tc_gpu as tc

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


class Second(ctypes.Structure):
    _fields_ = [("begin", ctypes.c_int), ("first_cout", ctypes.c_int), ("out", ctypes.c_void_p), ("out_ld", ctypes.c_int),
                ("act", ctypes.c_int)]


def test_cached_tile_maps_follow_the_kind_of_launch(monkeypatch, kernels):
    L = kernels
    L.mcb200_conv_packed_weight_count.restype = ctypes.c_size_t
    monkeypatch.setenv("MCB200_BLOCK_M", "128")      # the form that stores through shared memory
    monkeypatch.setenv("MCB200_STAGED", "1")
    first, begin, columns, m = 40, 64, 96, 3 * 20 * 20
    g = torch.Generator().manual_seed(71)
    x = torch.randn((3, 20, 20, 64), generator=g).cuda()
    wt = torch.randn((columns, 64, 1, 1), generator=g) * 0.1
    wt[first:begin] = 0
    s = tc.ConvShape(3, 20, 20, 64, 64, columns, 1, 1, 1, 1, 0, 0, 1, 1, 1, 0, 0)
    assert L.mcb200_conv_out_shape(ctypes.byref(s)) == 0
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    wdev = wt.cuda()
    packed = torch.empty(L.mcb200_conv_packed_weight_count(ctypes.byref(s)), device="cuda")
    assert L.mcb200_conv_pack_weights(ctypes.byref(s), p(wdev), p(packed), None) == 0
    plan = tc.aligned_plan()
    assert L.mcb200_conv_tc_plan(ctypes.byref(s), p(x), p(packed), ctypes.byref(plan)) == 0
    a, b = torch.empty((m, columns), device="cuda"), torch.empty((m, columns), device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    ep = tc.Epilogue()
    ep.residual_coeff = 1.0
    res = tc.Epilogue()
    res.residual_coeff, res.residual, res.residual_ld = 1.0, b.data_ptr(), columns
    second = Second(begin, first, b.data_ptr(), columns, 0)

    def one(epilogue):
        assert L.mcb200_conv_tc_launch(ctypes.byref(plan), p(a), columns, ctypes.byref(epilogue), p(status), None) == 0

    def two():
        assert L.mcb200_conv_tc_launch_two(ctypes.byref(plan), p(a), 0, columns, ctypes.byref(ep), ctypes.byref(second), 0,
                                           p(status), None) == 0

    a.zero_()
    one(ep)
    torch.cuda.synchronize()
    want = a.clone()
    assert float(want[:, :first].abs().max()) > 0 and float(want[:, begin:].abs().max()) > 0
    for _ in range(2):
        a.fill_(7.0)
        b.fill_(5.0)
        two()
        torch.cuda.synchronize()
        assert torch.equal(a[:, :first], want[:, :first]) and bool((a[:, first:] == 7.0).all())
        assert torch.equal(b[:, :columns - begin], want[:, begin:]) and bool((b[:, columns - begin:] == 5.0).all())
        b.fill_(5.0)
        one(res)
        torch.cuda.synchronize()
        assert torch.equal(a, want + 5.0)
        a.fill_(7.0)
        one(ep)
        torch.cuda.synchronize()
        assert torch.equal(a, want)
    assert int(status.item()) == 0
