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
