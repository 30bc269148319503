"""A pass whose first layers run part by part behind the copies of a new input gives the bits of the pass
that copies first: every kernel's result for an image is independent of the images beside it."""
import numpy as np
import pytest

from conftest import pkg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu_engine(engine):
    engine.set_mode(True, 0)
    return engine


def _net(wl, batch, size):
    """Image -> row-mode convolution, pooling, a residual block, depthwise, PReLU, then a layer that ends the
    part-wise steps (12 output channels)."""
    b = wl.NetBuilder("parts")
    b.input([("data", (batch, 3, size, size))])
    b.conv("conv1", "data", "conv1", 3, 32, 5, stride=2, pad=2)
    b.relu("conv1_relu", "conv1")
    b.pool("pool1", "conv1", "pool1", "MAX", k=3, stride=2)
    b.conv_bn("wide", "pool1", "wide", 32, 64, 1, relu=False)
    b.conv_bn("a", "pool1", "a", 32, 32, 3, pad=1)
    b.conv_bn("z", "a", "z", 32, 64, 1, relu=False)
    b.eltwise_sum("sum", ["wide", "z"], "sum")
    b.relu("sum_relu", "sum")
    b.conv("dw", "sum", "dw", 64, 64, 3, stride=2, pad=1, group=64)
    b.raw("dw_prelu", "PReLU", ["dw"], ["dw"])
    b.params.append(("dw_prelu_0", (64,), "one", 0))
    b.conv("point", "dw", "point", 64, 40, 1)
    b.conv("odd", "point", "odd", 40, 12, 3, pad=1)
    b.pool("pool5", "odd", "pool5", "AVE", global_pooling=True)
    return b


@pytest.mark.parametrize("precision", ["fp32", "bf16"])
@pytest.mark.parametrize("batch,parts,size", [(2, 2, 33), (5, 3, 40), (8, 8, 64), (13, 4, 57)])
def test_parts_give_the_bits_of_the_whole(monkeypatch, capi, gpu_engine, batch, parts, size, precision):
    wl = pkg("workloads")
    b = _net(wl, batch, size)
    weights = wl.init_params(b.params, seed=batch, bn_identity=False)
    rng = np.random.default_rng(size)
    inputs = [rng.standard_normal((batch, 3, size, size)).astype(np.float32) for _ in range(2)]
    inputs.append(inputs[1].copy())
    inputs.append(inputs[0][:max(1, batch // 2)])          # the plan is made again for another batch
    monkeypatch.setenv("MINICAFFE_PRECISION", precision)

    def run(value):
        monkeypatch.setenv("MCB200_INPUT_PARTS", str(value))
        net = capi.Net(gpu_engine, b.text(), None, from_buffer=True)
        net.set_params(weights)
        net.mark_output("pool1")
        got = []
        for i, x in enumerate(inputs):
            if i == 2:                                      # new slopes reach the launch that follows them
                net.set_params({"dw_prelu_0": np.full(64, 0.25, np.float32)})
            net.forward(data=x)
            got += [net.blob("pool1").data.copy(), net.blob("pool5").data.copy()]
            net.forward()                                   # the same input once more
            got.append(net.blob("pool5").data.copy())
        net.close()
        return got

    whole, pieces = run(1), run(parts)
    for w, p in zip(whole, pieces):
        assert w.shape == p.shape and np.isfinite(w).all()
        assert (w == p).all()
    assert (whole[4] != whole[7]).any()                     # the slopes alone
    for i in range(0, len(whole), 3):
        assert (whole[i + 1] == whole[i + 2]).all()


@pytest.mark.parametrize("kind", ["proposal", "detection_output"])
def test_detection_layers_whose_buffers_grow(capi, gpu_engine, kind):
    """Input in parts into a buffer that is new in the same pass (the first pass, and each larger batch): its zero
    fill comes before the copies.  The pass that follows reads the same input from the device."""
    wl = pkg("workloads")
    if kind == "proposal":
        b, top = wl.proposal(), "rois"
        images = [wl.proposal_input(seed=i)[0] for i in range(40)]
        feeds = {k: np.concatenate([f[k] for f in images]) for k in images[0]}
    else:
        b, top = wl.detection_head(1, 8732, 21, 0.01, 0.45, 400, 200), "detection_out"
        feeds = wl.detection_head_input(40, 8732, 21, 0, peaked=True)
    net = capi.Net(gpu_engine, b.text(), None, from_buffer=True)
    for batch in (10, 22, 40):
        net.forward(**{k: v if k == "prior" else v[:batch] for k, v in feeds.items()})
        first = net.blob(top).data.copy()
        net.forward()
        again = net.blob(top).data.copy()
        assert first.shape == again.shape and np.array_equal(first.view(np.uint32), again.view(np.uint32))
        assert set(first.reshape(first.shape[0], -1)[:, 0]) == set(range(batch))
    net.close()


def test_input_is_released_after_a_refusal(capi, gpu_engine):
    """A head that the kernels refuse (its keys and boxes need more shared memory than an SM has) when its input is
    on the way already: the error comes back, the copies have ended, and the memory serves the next net."""
    wl = pkg("workloads")
    for _ in range(3):
        feed = wl.detection_head_input(12, 26000, 2, 1, peaked=True)
        net = capi.Net(gpu_engine, wl.detection_head(12, 26000, 2, 0.01, 0.45, 4000, 200).text(), None, from_buffer=True)
        with pytest.raises(capi.CaffeError):
            net.forward(**feed)
        net.close()
        feed = wl.detection_head_input(12, 26000, 2, 2, peaked=True)
        net = capi.Net(gpu_engine, wl.detection_head(12, 26000, 2, 0.01, 0.45, 400, 200).text(), None, from_buffer=True)
        net.forward(**feed)
        first = net.blob("detection_out").data.copy()
        net.forward()
        assert np.array_equal(first.view(np.uint32), net.blob("detection_out").data.view(np.uint32))
        net.close()


def test_parts_share_storage(monkeypatch, capi, gpu_engine):
    """A chain run part by part takes the storage of the same chain run whole, and at most one more of its largest
    blob: the one that collects the parts' results."""
    torch = pytest.importorskip("torch")
    wl = pkg("workloads")
    b = wl.mobilenet_v1(64)
    weights, feed = wl.init_params(b.params, 0), wl.normal_image_input(64, 224, 0)
    used = {}
    for parts in (1, 8):
        monkeypatch.setenv("MCB200_INPUT_PARTS", str(parts))
        gpu_engine.memory_pool_clear()
        before = torch.cuda.mem_get_info()[0]
        net = capi.Net(gpu_engine, b.text(), None, from_buffer=True)
        net.set_params(weights)
        net.forward(**feed)
        used[parts] = before - torch.cuda.mem_get_info()[0]
        largest = max(blob.count for _, blob in net.blobs()) * 4
        net.close()
    gpu_engine.memory_pool_clear()
    assert largest < used[1]
    assert used[8] <= used[1] + largest + (4 << 20), used


def test_nets_on_several_threads(monkeypatch, capi, gpu_engine):
    """Passes that meet on the device copy their input whole, one that is alone in parts: the same bits, whichever a
    pass happens to be."""
    import threading
    wl = pkg("workloads")
    b = _net(wl, 24, 48)
    weights = wl.init_params(b.params, seed=3, bn_identity=False)
    monkeypatch.setenv("MCB200_INPUT_PARTS", "4")
    d = wl.detection_head(24, 4000, 9, 0.01, 0.45, 200, 100)
    feeds = [{"data": np.random.default_rng(i).standard_normal((24, 3, 48, 48)).astype(np.float32)} for i in range(3)]
    heads = [wl.detection_head_input(24, 4000, 9, i, peaked=True) for i in range(3)]

    def passes(seed, rounds, out):
        gpu_engine.set_mode(True, 0)
        net, head = (capi.Net(gpu_engine, x.text(), None, from_buffer=True) for x in (b, d))
        net.set_params(weights)
        for i in range(rounds):
            k = (seed + i) % 3
            net.forward(**feeds[k])
            head.forward(**heads[k])
            out.append((k, net.blob("pool5").data.copy(), head.blob("detection_out").data.copy()))
        net.close()
        head.close()

    alone = []
    passes(0, 3, alone)
    want = {k: (p, q) for k, p, q in alone}
    results = [[] for _ in range(3)]
    threads = [threading.Thread(target=passes, args=(i, 12, results[i])) for i in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for got in results:
        assert len(got) == 12
        for k, p, q in got:
            assert np.array_equal(p.view(np.uint32), want[k][0].view(np.uint32))
            assert np.array_equal(q.view(np.uint32), want[k][1].view(np.uint32))
