"""Two layers of one input in one launch, and a pooling taken in a layer's store: the bits of every layer on its own."""
import numpy as np
import pytest

from conftest import pkg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu_engine(engine):
    engine.set_mode(True, 0)
    return engine


def _net(wl, batch, size):
    """An image in row mode, a marching layer with its pooling, a projection beside a reduction, two heads whose columns are
    no multiple of 32 or 8, a layer beside one of another geometry, and a layer that comes behind a rewrite of its input."""
    b = wl.NetBuilder("siblings")
    b.input([("data", (batch, 3, size, size))])
    b.conv("conv1", "data", "conv1", 3, 64, 3, pad=1)
    b.relu("conv1_relu", "conv1")
    b.conv("march", "conv1", "march", 64, 64, 3, pad=1)
    b.relu("march_relu", "march")
    b.pool("pool", "march", "pool", "MAX", k=2, stride=2)
    b.conv_bn("wide", "pool", "wide", 64, 136, 1, relu=False)
    b.conv_bn("narrow", "pool", "narrow", 64, 40, 1)
    b.conv("back", "narrow", "back", 40, 136, 3, pad=1)
    b.eltwise_sum("sum", ["wide", "back"], "sum")
    b.conv("loc", "sum", "loc", 136, 24, 3, stride=2, pad=1)
    b.conv("other", "sum", "other", 136, 32, 3, stride=1, pad=1)
    b.conv("conf", "sum", "conf", 136, 42, 3, stride=2, pad=1)
    b.relu("conf_relu", "conf")
    b.conv("before", "loc", "before", 24, 16, 1)
    b.relu("loc_relu", "loc")
    b.conv("after", "loc", "after", 24, 16, 1)
    b.pool("last", "after", "last", "AVE", global_pooling=True)
    return b


@pytest.mark.parametrize("precision", ["fp32", "bf16"])
@pytest.mark.parametrize("batch,size", [(1, 48), (3, 57), (8, 62)])
def test_one_launch_gives_the_bits_of_two(monkeypatch, capi, gpu_engine, batch, size, precision):
    wl = pkg("workloads")
    b = _net(wl, batch, size)
    weights = wl.init_params(b.params, seed=batch, bn_identity=False)
    rng = np.random.default_rng(size)
    images = [rng.standard_normal((batch, 3, size, size)).astype(np.float32) for _ in range(3)]
    monkeypatch.setenv("MINICAFFE_PRECISION", precision)
    marked = ("loc", "conf", "before", "other")

    def run(siblings, **env):
        monkeypatch.setenv("MCB200_SIBLINGS", siblings)
        net = capi.Net(gpu_engine, b.text(), None, from_buffer=True)
        net.set_params(weights)
        for name in marked:
            net.mark_output(name)
        got = []
        for i, x in enumerate(images):
            if i == 2:      # new weights of the layer that has no launch of its own
                net.set_params({"conf_0": weights["conf_0"] * 0.5, "narrow_1": weights["narrow_1"] + 0.25} if "narrow_1" in weights
                               else {"conf_0": weights["conf_0"] * 0.5})
            net.forward(data=x)
            got.append({name: net.blob(name).data.copy() for name in marked + ("last",)})
        net.close()
        return got

    for alone, together in zip(run("0"), run("1")):
        for name in alone:
            assert np.isfinite(alone[name]).all() and np.array_equal(alone[name].view(np.uint32), together[name].view(np.uint32)), name
