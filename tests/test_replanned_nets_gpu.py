"""What the net's schedule fuses and merges, and nets that are planned again after they have run (another set of
outputs, another batch): what the layers keep from pass to pass has to follow."""
import ctypes

import numpy as np
import pytest

from conftest import pkg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu_engine(engine):
    engine.set_mode(True, 0)
    return engine


def _launches(engine):
    engine.lib.mcb200_launch_count.restype = ctypes.c_longlong
    return engine.lib.mcb200_launch_count()


def _equal(a, b):
    return np.array_equal(np.ascontiguousarray(a).view(np.uint32), np.ascontiguousarray(b).view(np.uint32))


@pytest.mark.parametrize("parts", ["1", "3"])
@pytest.mark.parametrize("precision", ["fp32", "bf16"])
def test_a_blob_in_front_of_a_fused_pooling_is_marked_after_a_pass(monkeypatch, capi, gpu_engine, precision, parts):
    """Enough rows that the layer marches with its pooling and without: the first plan pools in the store, the second may
    not, on the same input buffer, weights and shape."""
    wl = pkg("workloads")
    b = wl.NetBuilder("marked_later")
    b.input([("data", (9, 3, 101, 62))])
    b.conv("conv1", "data", "conv1", 3, 64, 3, pad=1)
    b.relu("conv1_relu", "conv1")
    b.conv("conv2", "conv1", "conv2", 64, 64, 3, pad=1)
    b.relu("conv2_relu", "conv2")
    b.pool("pool", "conv2", "pool", "MAX", k=2, stride=2)
    b.conv("conv3", "pool", "conv3", 64, 48, 1)
    b.pool("last", "conv3", "last", "AVE", global_pooling=True)
    weights = wl.init_params(b.params, seed=61)
    rng = np.random.default_rng(61)
    images = [rng.standard_normal((9, 3, 101, 62)).astype(np.float32) for _ in range(4)]
    monkeypatch.setenv("MINICAFFE_PRECISION", precision)
    monkeypatch.setenv("MCB200_INPUT_PARTS", parts)

    def run(marked_after):
        net = capi.Net(gpu_engine, b.text(), None, from_buffer=True)
        net.set_params(weights)
        got = []
        for i, x in enumerate(images):
            if i == marked_after:
                net.mark_output("conv2")
            net.forward(data=x)
            got.append([net.blob("last").data.copy()] + ([net.blob("conv2").data.copy()] if i >= marked_after else []))
        net.close()
        return got

    before, after = run(0), run(2)
    for i in (2, 3):
        assert np.isfinite(before[i][0]).all() and np.abs(before[i][0]).max() > 0
        assert _equal(before[i][0], after[i][0]) and _equal(before[i][1], after[i][1]), i


@pytest.mark.parametrize("pooled_first", [False, True])
@pytest.mark.parametrize("precision", ["fp32", "bf16"])
@pytest.mark.parametrize("batch,cout", [(1, 64), (2, 128), (16, 128), (16, 64)])
def test_a_layer_with_a_fused_pooling_stays_out_of_its_neighbours_launch(monkeypatch, capi, gpu_engine, batch, cout, precision,
                                                                         pooled_first):
    """Two 3 x 3 layers of one 64-channel input, the result of one read by a pooling only: the other marches or not, by its
    columns and the batch."""
    wl = pkg("workloads")
    b = wl.NetBuilder("pooled_sibling")
    b.input([("data", (batch, 3, 56, 56))])
    b.conv("conv1", "data", "conv1", 3, 64, 3, pad=1)
    b.relu("conv1_relu", "conv1")

    def plain():
        b.conv("plain", "conv1", "plain", 64, cout, 3, pad=1)
        b.relu("plain_relu", "plain")

    def pooled():
        b.conv("pooled", "conv1", "pooled", 64, 64, 3, pad=1)
        b.relu("pooled_relu", "pooled")
        b.pool("pool", "pooled", "pool", "MAX", k=2, stride=2)

    for add in (pooled, plain) if pooled_first else (plain, pooled):
        add()
    b.conv("next", "pool", "next", 64, 40, 1)
    b.pool("last", "plain", "last", "AVE", global_pooling=True)
    weights = wl.init_params(b.params, seed=62)
    rng = np.random.default_rng(62)
    images = [rng.standard_normal((batch, 3, 56, 56)).astype(np.float32) for _ in range(3)]
    monkeypatch.setenv("MINICAFFE_PRECISION", precision)

    def run(siblings, march):
        monkeypatch.setenv("MCB200_SIBLINGS", siblings)
        monkeypatch.setenv("MCB200_MARCH", march)
        net = capi.Net(gpu_engine, b.text(), None, from_buffer=True)
        net.set_params(weights)
        net.mark_output("next")
        got = []
        for x in images:
            net.forward(data=x)
            got.append([net.blob(name).data.copy() for name in ("next", "last")])
        net.close()
        return got

    for alone, together in zip(run("0", "0"), run("1", "1")):
        for want, got in zip(alone, together):
            assert np.isfinite(want).all() and np.abs(want).max() > 0 and _equal(want, got)


@pytest.mark.parametrize("parts", ["1", "3"])
@pytest.mark.parametrize("stride,kernel", [(9, 3), (16, 16), (2, 3)])
def test_a_refused_launch_of_two_stays_two_layers(monkeypatch, capi, gpu_engine, stride, kernel, parts):
    """Strides above 8 are refused by the tensor map: both layers run on the plain kernel, in this pass and in all later
    ones, with new weights and another batch too."""
    wl = pkg("workloads")
    b = wl.NetBuilder("refused")
    b.input([("data", (5, 3, 48, 48))])
    b.conv("trunk", "data", "trunk", 3, 16, 3, pad=1)
    b.relu("trunk_relu", "trunk")
    b.conv("left", "trunk", "left", 16, 24, kernel, stride=stride)
    b.relu("left_relu", "left")
    b.conv("right", "trunk", "right", 16, 40, kernel, stride=stride)
    b.pool("last", "left", "last", "AVE", global_pooling=True)
    weights = wl.init_params(b.params, seed=63)
    rng = np.random.default_rng(63)
    images = [rng.standard_normal((n, 3, 48, 48)).astype(np.float32) for n in (5, 5, 5, 5, 3, 3)]
    monkeypatch.setenv("MCB200_INPUT_PARTS", parts)

    def run(siblings):
        monkeypatch.setenv("MCB200_SIBLINGS", siblings)
        net = capi.Net(gpu_engine, b.text(), None, from_buffer=True)
        net.set_params(weights)
        net.mark_output("right")
        got = []
        for i, x in enumerate(images):
            if i == 3:
                net.set_params({"right_0": weights["right_0"] * 0.5, "left_1": weights["left_1"] + 0.25})
            net.forward(data=x)
            got.append([net.blob(name).data.copy() for name in ("right", "last")])
        net.close()
        return got

    for i, (alone, together) in enumerate(zip(run("0"), run("1"))):
        for want, got in zip(alone, together):
            assert np.isfinite(want).all() and np.abs(want).max() > 0 and _equal(want, got), i


def test_the_last_layers_top_comes_to_the_host_from_another_layers_launch(capi, gpu_engine):
    """The last layer runs in the launch of an earlier one, and the last step is a layer that nobody asked for: a pass still
    ends with the last layer's top on the host, so that reading it launches nothing."""
    wl = pkg("workloads")
    b = wl.NetBuilder("last_merged")
    b.input([("data", (2, 8, 14, 14))])
    b.conv("trunk", "data", "trunk", 8, 64, 3, pad=1)
    b.relu("trunk_relu", "trunk")
    b.conv("first", "trunk", "first", 64, 24, 3, pad=1)
    b.pool("between", "trunk", "between", "AVE", global_pooling=True)
    b.conv("last", "trunk", "last", 64, 40, 3, pad=1)
    net = capi.Net(gpu_engine, b.text(), None, from_buffer=True)
    net.set_params(wl.init_params(b.params, seed=64))
    rng = np.random.default_rng(64)
    for i in range(3):
        net.forward(data=rng.standard_normal((2, 8, 14, 14)).astype(np.float32))
        before = _launches(gpu_engine)
        assert np.isfinite(net.blob("last").data).all()
        assert _launches(gpu_engine) == before, i


def test_the_batch_before_does_not_decide_what_is_merged(capi, gpu_engine):
    """Two 3 x 3 layers that share a launch where few rows are left for each of the march's slabs, and march on their own
    with more images: a net that was planned for two images first runs 72 as one that was planned for 72."""
    wl = pkg("workloads")
    images = np.random.default_rng(65).standard_normal((72, 64, 56, 56)).astype(np.float32)
    got = {}
    for planned in (2, 72):
        b = wl.NetBuilder("history")
        b.input([("data", (planned, 64, 56, 56))])
        b.conv("left", "data", "left", 64, 64, 3, pad=1)
        b.conv("right", "data", "right", 64, 64, 3, pad=1)
        b.pool("pool", "left", "pool", "AVE", global_pooling=True)
        b.pool("last", "right", "last", "AVE", global_pooling=True)
        net = capi.Net(gpu_engine, b.text(), None, from_buffer=True)
        net.set_params(wl.init_params(b.params, seed=65))
        net.mark_output("pool")
        counts = []
        for x in (images[:planned], images, images[:2], images):
            net.forward(data=x)      # (packs weights where the form changes)
            before = _launches(gpu_engine)
            net.forward(data=x)
            counts.append(_launches(gpu_engine) - before)
        got[planned] = counts[1:], net.blob("pool").data.copy(), net.blob("last").data.copy()
        net.close()
    assert got[2][0] == got[72][0] and got[2][0][0] == got[2][0][2] > got[2][0][1]
    assert _equal(got[2][1], got[72][1]) and _equal(got[2][2], got[72][2])


@pytest.mark.parametrize("precision", ["fp32", "bf16"])
@pytest.mark.parametrize("batch", [16, 24, 71])
@pytest.mark.parametrize("couts", [(64, 64), (64, 128), (128, 64), (40, 48)], ids=str)
def test_marching_layers_give_the_same_bits_merged_and_alone(monkeypatch, capi, gpu_engine, batch, couts, precision):
    """Around the rows at which layers that march on their own share a launch, in either order."""
    wl = pkg("workloads")
    b = wl.NetBuilder("marching_siblings")
    b.input([("data", (batch, 64, 52, 50))])
    b.conv("trunk", "data", "trunk", 64, 64, 1)
    b.conv("left", "trunk", "left", 64, couts[0], 3, pad=1)
    b.relu("left_relu", "left")
    b.conv("right", "trunk", "right", 64, couts[1], 3, pad=1)
    b.conv("next", "left", "next", couts[0], 24, 1)
    b.pool("pool", "next", "pool", "AVE", global_pooling=True)
    b.pool("last", "right", "last", "AVE", global_pooling=True)
    weights = wl.init_params(b.params, seed=66)
    x = np.random.default_rng(66).standard_normal((batch, 64, 52, 50)).astype(np.float32)
    monkeypatch.setenv("MINICAFFE_PRECISION", precision)

    def run(siblings, march):
        monkeypatch.setenv("MCB200_SIBLINGS", siblings)
        monkeypatch.setenv("MCB200_MARCH", march)
        net = capi.Net(gpu_engine, b.text(), None, from_buffer=True)
        net.set_params(weights)
        net.mark_output("pool")
        for _ in range(2):
            net.forward(data=x)
        got = [net.blob(name).data.copy() for name in ("pool", "last")]
        net.close()
        return got

    want = run("0", "0")
    assert all(np.isfinite(w).all() and np.abs(w).max() > 0 for w in want)
    for got in (run("1", "1"), run("0", "1")):
        assert _equal(want[0], got[0]) and _equal(want[1], got[1])


@pytest.mark.parametrize("precision", ["fp32", "bf16"])
def test_a_pooling_is_taken_in_the_store_where_that_pays(monkeypatch, capi, gpu_engine, precision):
    """5 images of 58 rows are fewer than 296 slabs, 6 are more: in fp32 the pooling keeps its launch with five, with the same
    bits as everywhere."""
    wl = pkg("workloads")
    b = wl.NetBuilder("pool_pays")
    b.input([("data", (6, 64, 56, 56))])
    b.conv("trunk", "data", "trunk", 64, 64, 1)
    b.conv("conv", "trunk", "conv", 64, 64, 3, pad=1)
    b.relu("conv_relu", "conv")
    b.pool("pool", "conv", "pool", "MAX", k=2, stride=2)
    b.conv("next", "pool", "next", 64, 24, 1)
    b.pool("last", "next", "last", "AVE", global_pooling=True)
    weights = wl.init_params(b.params, seed=67)
    images = np.random.default_rng(67).standard_normal((6, 64, 56, 56)).astype(np.float32)
    monkeypatch.setenv("MINICAFFE_PRECISION", precision)

    def run(march):
        monkeypatch.setenv("MCB200_MARCH", march)
        net = capi.Net(gpu_engine, b.text(), None, from_buffer=True)
        net.set_params(weights)
        got = []
        for n in (6, 5, 6, 1):
            net.forward(data=images[:n])
            before = _launches(gpu_engine)
            net.forward(data=images[:n])
            got.append((_launches(gpu_engine) - before, net.blob("last").data.copy()))
        net.close()
        return got

    alone, fused = run("0"), run("1")
    saved = [a[0] - f[0] for a, f in zip(alone, fused)]
    assert saved == ([1, 0, 1, 0] if precision == "fp32" else [1, 1, 1, 1])
    for a, f in zip(alone, fused):
        assert np.isfinite(a[1]).all() and np.abs(a[1]).max() > 0 and _equal(a[1], f[1])


@pytest.mark.parametrize("first_channels", [3, 8])
@pytest.mark.parametrize("precision", ["fp32", "bf16"])
def test_a_batch_of_no_images(monkeypatch, capi, gpu_engine, precision, first_channels):
    """Between ordinary batches, through layers of all forms: an empty result in fp32, an error in bfloat16, and the next
    batch is what it was."""
    wl = pkg("workloads")
    b = wl.NetBuilder("empty")
    b.input([("data", (16, first_channels, 56, 56))])
    b.conv("conv1", "data", "conv1", first_channels, 64, 3, pad=1)
    b.relu("conv1_relu", "conv1")
    b.conv("conv2", "conv1", "conv2", 64, 64, 3, pad=1)
    b.pool("pool", "conv2", "pool", "MAX", k=2, stride=2)
    b.conv("left", "pool", "left", 64, 40, 1)
    b.conv("right", "pool", "right", 64, 24, 1)
    b.pool("last", "right", "last", "AVE", global_pooling=True)
    x = np.random.default_rng(68).standard_normal((16, first_channels, 56, 56)).astype(np.float32)
    monkeypatch.setenv("MINICAFFE_PRECISION", precision)
    net = capi.Net(gpu_engine, b.text(), None, from_buffer=True)
    net.set_params(wl.init_params(b.params, seed=68))
    net.mark_output("left")
    names = ("left", "last")
    net.forward(data=x)
    want = [net.blob(name).data.copy() for name in names]
    for _ in range(2):
        if precision == "bf16":
            with pytest.raises(capi.CaffeError):
                net.forward(data=x[:0])
        else:
            net.forward(data=x[:0])
            assert net.blob("left").shape == (0, 40, 28, 28) and net.blob("last").shape == (0, 24, 1, 1)
            assert net.blob("left").data.size == 0
        net.forward(data=x)
        for name, value in zip(names, want):
            assert np.isfinite(value).all() and _equal(net.blob(name).data, value), name


@pytest.mark.parametrize("columns,merged", [((256, 64), False), ((96, 384), True), ((256, 128), True), ((512, 128), True)], ids=str)
def test_short_sums_share_a_launch_where_that_pays(monkeypatch, capi, gpu_engine, columns, merged):
    """Some 17 million results of 64 channels: 256 and 64 columns stay two launches, and all give the same bits."""
    wl = pkg("workloads")
    side = 56
    batch = int(17.5e6 / (side * side * sum(columns)))
    b = wl.NetBuilder("short_sums")
    b.input([("data", (batch, 64, side, side))])
    b.conv("left", "data", "left", 64, columns[0], 1)
    b.relu("left_relu", "left")
    b.conv("right", "data", "right", 64, columns[1], 1)
    b.pool("pool", "left", "pool", "MAX", k=3, stride=2)
    b.conv("next", "pool", "next", columns[0], 16, 1, stride=4)
    b.pool("last", "right", "last", "AVE", global_pooling=True)
    weights = wl.init_params(b.params, seed=69)
    x = np.random.default_rng(69).standard_normal((batch, 64, side, side)).astype(np.float32)

    def run(siblings):
        monkeypatch.setenv("MCB200_SIBLINGS", siblings)
        net = capi.Net(gpu_engine, b.text(), None, from_buffer=True)
        net.set_params(weights)
        net.mark_output("next")
        net.forward(data=x)
        before = _launches(gpu_engine)
        net.forward(data=x)
        got = _launches(gpu_engine) - before, net.blob("next").data.copy(), net.blob("last").data.copy()
        net.close()
        return got

    alone, together = run("0"), run("1")
    assert alone[0] - together[0] == int(merged)
    for want, got in zip(alone[1:], together[1:]):
        assert np.isfinite(want).all() and np.abs(want).max() > 0 and _equal(want, got)


@pytest.mark.parametrize("parts", ["1", "3"])
@pytest.mark.parametrize("precision", ["fp32", "bf16"])
@pytest.mark.parametrize("batch,size", [(7, 56), (8, 61)])
def test_every_layer_on_its_own_gives_the_same_bits(monkeypatch, capi, gpu_engine, batch, size, precision, parts):
    """Neither merged layers nor the march nor a pooling in its store, against all of them, whole and in parts."""
    import test_sibling_layers_gpu as siblings
    wl = pkg("workloads")
    b = siblings._net(wl, batch, size)
    weights = wl.init_params(b.params, seed=70, bn_identity=False)
    rng = np.random.default_rng(70)
    images = [rng.standard_normal((batch, 3, size, size)).astype(np.float32) for _ in range(3)]
    marked = ("loc", "conf", "before", "other")
    monkeypatch.setenv("MINICAFFE_PRECISION", precision)

    def run(on, parts):
        monkeypatch.setenv("MCB200_SIBLINGS", on)
        monkeypatch.setenv("MCB200_MARCH", on)
        monkeypatch.setenv("MCB200_INPUT_PARTS", parts)
        net = capi.Net(gpu_engine, b.text(), None, from_buffer=True)
        net.set_params(weights)
        for name in marked:
            net.mark_output(name)
        got = []
        for x in images:
            net.forward(data=x)
            got.append([net.blob(name).data.copy() for name in marked + ("last",)])
        assert (["pool"] in net.schedule()) == (on == "0")
        net.close()
        return got

    for alone, together in zip(run("0", "1"), run("1", parts)):
        for want, got in zip(alone, together):
            assert np.isfinite(want).all() and np.abs(want).max() > 0 and _equal(want, got)
