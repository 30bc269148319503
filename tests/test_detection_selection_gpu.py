"""DetectionOutput's selections where they can go wrong: ties that fill a bin, candidate lists around the sizes of
a warp, a block and a bit-matrix row, keep_top_k of nothing and of everything, and batches whose input arrives in parts.
Against the C restatement of the reference (oracle/), bit for bit."""
import importlib

import numpy as np
import pytest

from conftest import pkg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu_engine(engine):
    engine.set_mode(True, 0)
    return engine


@pytest.mark.parametrize("case", [
    # images, priors, classes, conf_thr, nms_thr, top_k, keep_top_k, score levels (0: distinct)
    (1, 31, 2, 0.01, 0.45, 400, 200, 0),
    (2, 33, 3, 0.0, 0.45, 32, 33, 0),
    (1, 3000, 3, 0.01, 0.45, 1023, 200, 0),      # a matrix of 32 words
    (1, 3000, 3, 0.01, 0.45, 1025, 300, 0),      # one candidate more: the warp's walk
    (1, 2500, 2, 0.01, 0.3, 400, -1, 0),
    (2, 500, 4, 0.99999, 0.45, 100, 50, 0),      # (nearly) nothing passes
    (1, 3000, 2, 0.01, 0.45, 400, 200, 2),       # ties beyond a bin's list: the radix walk, by prior index
    (9, 5000, 21, 0.01, 0.45, 400, 200, 0),      # input in parts
], ids=lambda c: "x".join(str(v) for v in c))
def test_selection_against_the_restatement(capi, gpu_engine, case):
    images, priors, classes, conf_thr, nms_thr, top_k, keep, levels = case
    wl, port = pkg("workloads"), importlib.import_module("oracle.port")
    b = wl.detection_head(batch=images, num_priors=priors, num_classes=classes, conf_thr=conf_thr, nms_thr=nms_thr, top_k=top_k,
                          keep_top_k=keep)
    feed = wl.detection_head_input(images, priors, classes, seed=priors, peaked=True)
    if levels:
        feed["conf"] = (np.round(feed["conf"] * levels) / levels * 0.8 + 0.1).astype(np.float32)
        keep = -1                                  # (across classes the reference's order of equals is unspecified)
        b = wl.detection_head(batch=images, num_priors=priors, num_classes=classes, conf_thr=conf_thr, nms_thr=nms_thr, top_k=top_k,
                              keep_top_k=keep)
    want = port.detection_output(feed["loc"], feed["conf"], feed["prior"], classes, confidence_threshold=conf_thr,
                                 nms_threshold=nms_thr, top_k=top_k, keep_top_k=keep)
    net = capi.Net(gpu_engine, b.text(), None, from_buffer=True)
    for again in range(2):      # the second pass finds its input on the device
        net.forward(**feed) if again == 0 else net.forward()
        got = net.blob("detection_out").data.copy().reshape(-1, 7)
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    net.close()


def _against_the_restatement(capi, gpu_engine, feed, images, priors, classes, conf_thr, top_k, keep, nms_thr=0.45):
    wl, port = pkg("workloads"), importlib.import_module("oracle.port")
    b = wl.detection_head(batch=images, num_priors=priors, num_classes=classes, conf_thr=conf_thr, nms_thr=nms_thr, top_k=top_k,
                          keep_top_k=keep)
    want = port.detection_output(feed["loc"], feed["conf"], feed["prior"], classes, confidence_threshold=conf_thr,
                                 nms_threshold=nms_thr, top_k=top_k, keep_top_k=keep)
    net = capi.Net(gpu_engine, b.text(), None, from_buffer=True)
    net.forward(**feed)
    got = net.blob("detection_out").data.copy().reshape(-1, 7)
    net.close()
    assert got.shape == want.shape and np.array_equal(got.view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("priors,top_k,passing", [
    (3000, 2000, 900),       # bits of 104 KB, a region of 12 KB of keys: the warp's walk
    (3000, 2000, 300),       # 12 000 bytes of bits in 12 000 bytes: the matrix, to the last byte
    (3000, 2000, 301),
    (1500, -1, 600),
    (4096, -1, 1024),
    (8732, 1100, 513),       # either side of the region of a full SSD head
    (8732, 1100, 514),
])
def test_short_lists_under_a_long_limit(capi, gpu_engine, priors, top_k, passing):
    """Beyond 1024 candidates per class no room for their overlap bits is set aside: a list that turns out short
    takes the bit matrix only where its bits fit into the keys' place."""
    feed = pkg("workloads").detection_head_input(1, priors, 2, seed=priors, peaked=True)
    rng = np.random.default_rng(passing)
    scores = 0.4 * rng.permutation(priors) / priors
    pick = rng.permutation(priors)[:passing]
    scores[pick] = 0.5 + 0.4 * np.arange(passing) / passing
    feed["conf"].reshape(priors, 2)[:, 1] = scores
    _against_the_restatement(capi, gpu_engine, feed, 1, priors, 2, 0.45, top_k, 200)


@pytest.mark.parametrize("images,priors,classes,top_k,keep", [(2, 40, 3, 1, 5), (1, 1, 2, 400, 200), (1, 1, 21, -1, -1), (3, 300, 2, 1, 1)])
def test_a_single_candidate_per_class(capi, gpu_engine, images, priors, classes, top_k, keep):
    """The smallest list: one key, behind which the boxes still start on 16 bytes."""
    feed = pkg("workloads").detection_head_input(images, priors, classes, seed=top_k + priors, peaked=True)
    _against_the_restatement(capi, gpu_engine, feed, images, priors, classes, 0.01, top_k, keep)


@pytest.mark.parametrize("images,top_k,keep", [(1, 0, 200), (3, 0, -1), (2, 0, 0), (2, 400, 0), (9, 1, 0)])
def test_limits_of_nothing(capi, gpu_engine, images, top_k, keep):
    """top_k 0 (no candidate of any class) and keep_top_k 0 (no detection of any image): a placeholder row per image."""
    feed = pkg("workloads").detection_head_input(images, 700, 4, seed=images, peaked=True)
    _against_the_restatement(capi, gpu_engine, feed, images, 700, 4, 0.01, top_k, keep)
