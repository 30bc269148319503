"""Layers that only rename axes (Permute to channels-last, Flatten, Reshape) do not run in front of a Concat
and share their bottom's storage elsewhere; prior boxes are computed on the device.  Copies are exact and
the boxes' operations correctly rounded, so every comparison is for equality."""
import numpy as np
import pytest

from conftest import pkg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu_engine(engine):
    engine.set_mode(True, 0)
    return engine


def _heads(wl, batch, channels, sizes):
    """Heads over pooled maps: Permute -> Flatten -> Concat -> Reshape -> Softmax -> Flatten."""
    b = wl.NetBuilder("views")
    b.input([("data", (batch, 8) + sizes[0])])
    flats = []
    prev = "data"
    for i, c in enumerate(channels):
        name = "head%d" % i
        b.conv(name, prev, name, 8, c, 1)
        b.raw(name + "_perm", "Permute", [name], [name + "_perm"],
              "permute_param { order: 0 order: 2 order: 3 order: 1 }")
        b.raw(name + "_flat", "Flatten", [name + "_perm"], [name + "_flat"], "flatten_param { axis: 1 }")
        flats.append(name + "_flat")
        if i + 1 < len(channels):
            b.pool("pool%d" % i, prev, "pool%d" % i, "MAX", k=2, stride=2)
            prev = "pool%d" % i
    b.raw("all", "Concat", flats, ["all"], "concat_param { axis: 1 }")
    b.raw("rows", "Reshape", ["all"], ["rows"], "reshape_param { shape { dim: 0 dim: -1 dim: 3 } }")
    b.softmax("soft", "rows", "soft", axis=2)
    b.raw("out", "Flatten", ["soft"], ["out"], "flatten_param { axis: 1 }")
    return b


@pytest.mark.parametrize("marked", [False, True])
@pytest.mark.parametrize("batch,channels,size", [(1, (12, 24), (6, 8)), (3, (6, 15, 3), (9, 5)), (2, (3,), (1, 1)),
                                                 (2, (12, 12, 12, 12, 12), (17, 17))])
def test_heads_in_front_of_concat(capi, gpu_engine, batch, channels, size, marked):
    wl = pkg("workloads")
    b = _heads(wl, batch, channels, [size])
    weights = wl.init_params(b.params, seed=3)
    rng = np.random.default_rng(batch)
    heads = ["head%d" % i for i in range(len(channels))]
    net = capi.Net(gpu_engine, b.text(), None, from_buffer=True)
    net.set_params(weights)
    for name in heads + ["all", "soft"] + (["rows", "head0_perm", "head0_flat"] if marked else []):
        net.mark_output(name)
    plain = capi.Net(gpu_engine, b.text(), None, from_buffer=True)
    plain.set_params(weights)
    for _ in range(2):
        x = rng.standard_normal((batch, 8) + size).astype(np.float32)
        net.forward(data=x)
        parts = [net.blob(h).data.copy() for h in heads]
        want = np.concatenate([p.transpose(0, 2, 3, 1).reshape(batch, -1) for p in parts], axis=1)
        assert (net.blob("all").data.reshape(want.shape) == want).all()
        if marked:
            assert (net.blob("rows").data.ravel() == want.ravel()).all()
            assert (net.blob("head0_perm").data == parts[0].transpose(0, 2, 3, 1)).all()
            assert (net.blob("head0_flat").data.ravel() == net.blob("head0_perm").data.ravel()).all()
        soft = net.blob("soft").data.copy()
        assert np.allclose(soft.reshape(batch, -1, 3).sum(2), 1, atol=1e-5)
        assert (net.blob("out").data.ravel() == soft.ravel()).all()
        plain.forward(data=x)                              # nothing marked: every view shares storage
        assert (plain.blob("out").data.ravel() == soft.ravel()).all()
    net.close()
    plain.close()


@pytest.mark.parametrize("axis,shapes", [
    (1, [(3, 5), (3, 7), (3, 1)]),                         # rows that are not 8-byte multiples
    (1, [(2, 6), (2, 10)]),
    (2, [(1, 2, 8), (1, 2, 4), (1, 2, 12)]),
    (0, [(2, 5), (1, 5)]),
    (1, [(2, 3, 4)] * 18),                                 # more sources than one launch takes
])
def test_concat_of_rows(capi, gpu_engine, axis, shapes):
    wl = pkg("workloads")
    b = wl.NetBuilder("concat")
    names = ["x%d" % i for i in range(len(shapes))]
    b.input(list(zip(names, shapes)))
    b.raw("y", "Concat", names, ["y"], "concat_param { axis: %d }" % axis)
    rng = np.random.default_rng(axis)
    xs = {n: rng.standard_normal(s).astype(np.float32) for n, s in zip(names, shapes)}
    net = capi.Net(gpu_engine, b.text(), None, from_buffer=True)
    net.forward(**xs)
    want = np.concatenate([xs[n] for n in names], axis=axis)
    got = net.blob("y").data
    assert got.size == want.size and (got.ravel() == want.ravel()).all()
    net.close()


def _priors(h, w, img_h, img_w, min_sizes, max_sizes, aspects, step, offset, clip, variance):
    """The layer's host expressions: float centres, double around them, one rounding per coordinate."""
    f = np.float32
    ars = [f(1)]
    for a in aspects:
        ars += [f(a), f(1.0 / np.float64(f(a)))]
    out = []
    sh, sw = (f(step), f(step)) if step else (f(img_h) / f(h), f(img_w) / f(w))
    for y in range(h):
        for x in range(w):
            cx, cy = np.float64((f(x) + f(offset)) * sw), np.float64((f(y) + f(offset)) * sh)
            for i, m in enumerate(min_sizes):
                sizes = [(f(m), f(m))]
                if max_sizes:
                    r = f(np.sqrt(np.float64(m * max_sizes[i])))
                    sizes.append((r, r))
                for a in ars[1:]:
                    sizes.append((f(m) * np.sqrt(a), f(m) / np.sqrt(a)))
                for bw, bh in sizes:
                    hw, hh = np.float64(bw) / 2, np.float64(bh) / 2
                    out += [f((cx - hw) / img_w), f((cy - hh) / img_h), f((cx + hw) / img_w), f((cy + hh) / img_h)]
    out = np.array(out, np.float32)
    if clip:
        out = np.minimum(np.maximum(out, f(0)), f(1))
    var = np.tile(np.array(variance, np.float32), out.size // len(variance))
    return np.stack([out, var])[None]


@pytest.mark.parametrize("h,w,img_h,img_w,min_sizes,max_sizes,aspects,step,clip,variance", [
    (3, 5, 300, 301, [30], [60], [2], 0, False, [0.1, 0.1, 0.2, 0.2]),
    (1, 1, 300, 300, [264], [315], [2, 3], 300, True, [0.1, 0.1, 0.2, 0.2]),
    (7, 4, 97, 55, [11, 23], [], [2], 13.5, True, [0.1]),
    (2, 3, 64, 64, list(range(5, 75)), [], [], 8, False, [0.1]),      # more boxes per cell than the kernel takes
])
def test_prior_boxes(capi, gpu_engine, h, w, img_h, img_w, min_sizes, max_sizes, aspects, step, clip, variance):
    wl = pkg("workloads")
    b = wl.NetBuilder("priors")
    b.input([("map", (2, 4, h, w)), ("img", (2, 3, img_h, img_w))])
    body = " ".join(["min_size: %g" % v for v in min_sizes] + ["max_size: %g" % v for v in max_sizes] +
                    ["aspect_ratio: %g" % v for v in aspects] + ["variance: %g" % v for v in variance] +
                    (["step: %g" % step] if step else []))
    b.raw("p", "PriorBox", ["map", "img"], ["p"],
          "prior_box_param { %s flip: true clip: %s offset: 0.5 }" % (body, "true" if clip else "false"))
    net = capi.Net(gpu_engine, b.text(), None, from_buffer=True)
    net.forward()
    got = net.blob("p").data.copy()
    net.close()
    want = _priors(h, w, img_h, img_w, min_sizes, max_sizes, aspects, step, 0.5, clip, variance)
    assert got.shape == want.shape
    assert (got == want).all(), np.abs(got - want).max()
