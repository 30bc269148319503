"""Deconvolution on the tensor cores in each of its forms (phase by phase, all phases side by side, over the
spread input), at the geometries where they meet their limits, against torch's transposed convolution in
double precision.  TF32 operands: a product is off by at most 2^-10 of itself, a sum of K of them by a random
walk's share of that; 2e-2 + 1e-2 |value| on results of order one leaves a factor of ten (the bound of the
other tensor-core tests).  BatchNorm on batch statistics behind it: fp32 sums of a few dozen values and double
above them, 1e-5 of the value."""
import numpy as np
import pytest

from conftest import pkg

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu_engine(engine):
    engine.set_mode(True, 0)
    return engine


@pytest.mark.parametrize("case", [
    # n, cin, h, w, cout, kernel, stride, pad, bias
    (2, 8, 5, 7, 68, 4, 2, 1, True),       # phases; a ragged N tile
    (3, 20, 1, 1, 72, 4, 1, 0, False),     # one input pixel: a phase per tap
    (2, 12, 6, 5, 100, 3, 2, 0, True),     # odd filter: phases of unequal taps, output cut short
    (1, 16, 4, 4, 66, 5, 3, 2, True),      # stride 3, rows that are not 16-byte aligned
    (2, 32, 9, 6, 64, 2, 4, 0, False),     # stride beyond the filter: phases without taps
    (2, 64, 8, 8, 3, 4, 2, 1, True),       # few channels: all phases in one N tile
    (1, 8, 3, 5, 5, 4, 2, 0, True),        # few channels, a grid no symmetric padding yields
    (1, 8, 4, 4, 6, 5, 5, 1, True),        # stride 5: the spread form
    (1, 6, 4, 3, 8, 4, 2, 1, True),        # a channel count that is no multiple of four: the spread form
], ids=lambda c: "x".join(str(int(v)) for v in c))
def test_deconvolution_forms(capi, gpu_engine, case):
    n, cin, h, w, cout, k, stride, pad, bias = case
    wl = pkg("workloads")
    rng = np.random.default_rng(sum(case))
    x = rng.standard_normal((n, cin, h, w)).astype(np.float32)
    weight = (rng.standard_normal((cin, cout, k, k)) / np.sqrt(cin)).astype(np.float32)
    b = wl.NetBuilder("deconv")
    b.input([("data", (n, cin, h, w))])
    b.raw("up", "Deconvolution", ["data"], ["up"], "convolution_param { num_output: %d kernel_size: %d stride: %d pad: %d bias_term: %s }"
          % (cout, k, stride, pad, "true" if bias else "false"))
    weights = {"up_0": weight}
    if bias:
        weights["up_1"] = rng.standard_normal(cout).astype(np.float32)
    net = capi.Net(gpu_engine, b.text(), None, from_buffer=True)
    net.set_params(weights)
    net.forward(data=x)
    got = net.blob("up").data.copy()
    net.close()
    want = torch.nn.functional.conv_transpose2d(torch.from_numpy(x).double(), torch.from_numpy(weight).double(),
                                                torch.from_numpy(weights["up_1"]).double() if bias else None, stride, pad).numpy()
    assert got.shape == want.shape
    assert (np.abs(got - want) <= 2e-2 + 1e-2 * np.abs(want)).all(), float(np.abs(got - want).max())


@pytest.mark.parametrize("shape", [(1, 4, 1, 1), (3, 68, 7, 5), (5, 1028, 3, 2), (64, 64, 32, 32), (2, 6, 5, 5)],
                         ids=lambda s: "x".join(map(str, s)))
def test_batch_statistics_with_scale_and_relu_behind(capi, gpu_engine, shape):
    wl = pkg("workloads")
    rng = np.random.default_rng(shape[1])
    x = (rng.standard_normal(shape) * 0.5 + 30.0).astype(np.float32)     # a mean of sixty standard deviations
    b = wl.NetBuilder("bn")
    b.input([("data", shape)])
    b.raw("pool", "Pooling", ["data"], ["x"], "pooling_param { pool: MAX kernel_size: 1 stride: 1 }")     # channels last from here
    b.raw("bn", "BatchNorm", ["x"], ["x"], "batch_norm_param { use_global_stats: false }")
    b.scale("sc", "x", shape[1])
    b.relu("relu", "x")
    gamma, beta = rng.uniform(0.5, 1.5, shape[1]).astype(np.float32), rng.standard_normal(shape[1]).astype(np.float32)
    net = capi.Net(gpu_engine, b.text(), None, from_buffer=True)
    net.set_params({"sc_0": gamma, "sc_1": beta})
    for _ in range(2):
        net.forward(data=x)
        got = net.blob("x").data.copy()
        d = x.astype(np.float64)
        mean, var = d.mean(axis=(0, 2, 3), keepdims=True), d.var(axis=(0, 2, 3), keepdims=True)
        # the layer's fp32 scale and shift: y = x * scale + shift with |x * scale| of sixty at 2^-24 each
        want = np.maximum((d - mean) / np.sqrt(var + 1e-5) * gamma.reshape(1, -1, 1, 1) + beta.reshape(1, -1, 1, 1), 0.0)
        scale = np.abs(mean) / np.sqrt(var + 1e-5) * gamma.reshape(1, -1, 1, 1) + 1.0
        assert (np.abs(got - want) <= 1e-5 * np.abs(want) + 4 * 2.0 ** -24 * scale).all(), float(np.abs(got - want).max())
    net.close()


@pytest.mark.parametrize("cout", [68, 3], ids=["phases", "window"])
@pytest.mark.parametrize("k,stride", [(4, 1), (3, 2), (4, 4), (2, 1)])
def test_one_net_from_a_pixel_to_a_map_and_back(capi, gpu_engine, cout, k, stride):
    """A single input pixel runs with a phase per tap, a larger input with one per step of the stride: the weights
    packed for the one do not serve the other.  Nor do they for two inputs of one layer."""
    wl = pkg("workloads")
    rng = np.random.default_rng(k)
    weight = (rng.standard_normal((12, cout, k, k)) / np.sqrt(12)).astype(np.float32)
    bias = rng.standard_normal(cout).astype(np.float32)
    b = wl.NetBuilder("deconv")
    b.input([("data", (2, 12, 1, 1)), ("more", (2, 12, 1, 1))])
    b.raw("up", "Deconvolution", ["data", "more"], ["up", "up_more"],
          "convolution_param { num_output: %d kernel_size: %d stride: %d }" % (cout, k, stride))
    net = capi.Net(gpu_engine, b.text(), None, from_buffer=True)
    net.set_params({"up_0": weight, "up_1": bias})
    for (h, w), (h2, w2) in (((1, 1), (1, 1)), ((2, 2), (2, 2)), ((1, 1), (1, 1)), ((1, 1), (3, 2)), ((3, 2), (1, 1))):
        feed = {"data": rng.standard_normal((2, 12, h, w)).astype(np.float32),
                "more": rng.standard_normal((2, 12, h2, w2)).astype(np.float32)}
        for _ in range(2):
            net.forward(**feed)
            for x, top in (("data", "up"), ("more", "up_more")):
                got = net.blob(top).data.copy()
                want = torch.nn.functional.conv_transpose2d(torch.from_numpy(feed[x]).double(), torch.from_numpy(weight).double(),
                                                            torch.from_numpy(bias).double(), stride).numpy()
                assert got.shape == want.shape
                assert (np.abs(got - want) <= 2e-2 + 1e-2 * np.abs(want)).all(), (h, w, h2, w2, top)
    net.close()


@pytest.mark.parametrize("shape,outlier,mean", [
    ((16, 8, 64, 64), 60.0, 0.0), ((16, 8, 64, 64), -200.0, 0.0), ((16, 8, 64, 64), 200.0, 1000.0),
    ((2, 1032, 9, 7), 50.0, -30.0), ((3, 260, 41, 40), 30.0, 0.0), ((9, 2048, 7, 7), 20.0, 3.0), ((64, 4096, 1, 1), 7.0, 0.0),
    ((2, 512, 1, 1), 1.0, 0.0), ((3, 4, 5, 5), 5.0, 0.0), ((1, 4, 1, 2), 1.0, 7.0), ((7, 12, 11, 13), 0.0, 4096.0),
], ids=str)
def test_batch_statistics_behind_a_first_pixel_far_from_the_mean(capi, gpu_engine, shape, outlier, mean):
    """Every channel's first value lies `outlier` standard deviations from the others' mean, as under a zero border.
    The bound is that of y = x * scale + shift alone, with exact statistics: four roundings in the layer's scale, six
    in its shift, one in the result, each 2^-24 of its value."""
    wl = pkg("workloads")
    rng = np.random.default_rng(shape[1])
    x = (rng.standard_normal(shape) + mean).astype(np.float32)
    x[0, :, 0, 0] = mean + outlier
    b = wl.NetBuilder("bn")
    b.input([("data", shape)])
    b.raw("pool", "Pooling", ["data"], ["x"], "pooling_param { pool: MAX kernel_size: 1 stride: 1 }")     # channels last from here
    b.raw("bn", "BatchNorm", ["x"], ["x"], "batch_norm_param { use_global_stats: false }")
    net = capi.Net(gpu_engine, b.text(), None, from_buffer=True)
    net.forward(data=x)
    got = net.blob("x").data.copy()
    net.close()
    d = x.astype(np.float64)
    centre, var = d.mean(axis=(0, 2, 3), keepdims=True), d.var(axis=(0, 2, 3), keepdims=True)
    std = np.sqrt(var + 1e-5)
    want = (d - centre) / std
    bound = 2.0 ** -24 * (4 * np.abs(d) / std + 6 * np.abs(centre) / std + np.abs(want) + 1)
    assert (np.abs(got - want) <= bound).all(), float((np.abs(got - want) / bound).max())


@pytest.mark.parametrize("c,hw,cout,k,pad", [(64, 18, 68, 3, 1), (64, 18, 8, 3, 1), (40, 14, 12, 4, 0), (12, 9, 72, 2, 1), (36, 17, 5, 5, 2)])
def test_stride_one_is_the_convolution(capi, gpu_engine, c, hw, cout, k, pad):
    """A deconvolution of stride 1 runs as the convolution with the reversed filter: the same bits."""
    wl = pkg("workloads")
    rng = np.random.default_rng(c)
    x = rng.standard_normal((2, c, hw, hw)).astype(np.float32)
    weight = (rng.standard_normal((c, cout, k, k)) / np.sqrt(c)).astype(np.float32)
    got = []
    for kind, w, p in (("Deconvolution", weight, pad), ("Convolution", weight.transpose(1, 0, 2, 3)[:, :, ::-1, ::-1], k - 1 - pad)):
        b = wl.NetBuilder("stride_one")
        b.input([("data", x.shape)])
        b.raw("up", kind, ["data"], ["up"], "convolution_param { num_output: %d kernel_size: %d pad: %d bias_term: false }" % (cout, k, p))
        net = capi.Net(gpu_engine, b.text(), None, from_buffer=True)
        net.set_params({"up_0": np.ascontiguousarray(w)})
        net.forward(data=x)
        got.append(net.blob("up").data.copy())
        net.close()
    assert got[0].shape == got[1].shape and np.array_equal(got[0].view(np.uint32), got[1].view(np.uint32))
