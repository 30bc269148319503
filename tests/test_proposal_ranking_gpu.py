"""The proposal layer's ranking at the sizes where its selection can go wrong: fewer proposals than one
segment, several segments, the cut at pre_nms_topn inside one, scores that the sample misjudges (ties), a kept
list beyond shared memory, and more images than the wide clusters serve.  Against the C restatement of the
reference (oracle/), bit for bit."""
import importlib

import numpy as np
import pytest

from conftest import pkg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu_engine(engine):
    engine.set_mode(True, 0)
    return engine


def _ties(scores, levels):
    """Scores on `levels` values (the order among equals is by proposal index), and distinct scores in that order."""
    a = scores.shape[1] // 2
    tied = np.floor(scores * levels / 8).astype(np.float32)
    order = tied[0, a:].transpose(1, 2, 0).reshape(-1)             # proposal order: (y, x, anchor)
    rank = np.empty(order.size, dtype=np.float32)
    rank[np.argsort(-order, kind="stable")] = -np.arange(order.size, dtype=np.float32)
    distinct = scores.copy()
    distinct[0, a:] = rank.reshape(scores.shape[2], scores.shape[3], a).transpose(2, 0, 1)
    return tied, distinct


@pytest.mark.parametrize("case", [
    # anchors, H, W, pre, post, thresh, min_size, images, tie levels (0: distinct scores)
    (9, 10, 11, 6000, 300, 0.7, 16, 1, 0),      # 990 proposals: one segment
    (9, 31, 17, 3000, 2900, 0.9, 0, 2, 0),      # segments up to the cut at pre_nms_topn
    (15, 40, 33, 700, 600, 0.95, 0, 1, 0),      # the cut inside the first segment
    (9, 37, 29, 12000, 9000, 0.99, 0, 1, 0),    # a kept list too long for shared memory
    (9, 24, 25, 2500, 400, 0.6, 0, 1, 3),       # ties: exact selection by index
    (15, 24, 24, 6000, 50, 0.7, 16, 21, 0),     # clusters of four
    (3, 25, 27, 2000, 300, 0.0, 16, 1, 0),      # threshold 0: every quotient is divided out
], ids=lambda c: "x".join(str(v) for v in c))
def test_ranking_against_the_restatement(capi, gpu_engine, case):
    anchors, h, w, pre, post, thr, min_size, images, levels = case
    wl, port = pkg("workloads"), importlib.import_module("oracle.port")
    scales = {15: (2, 4, 8, 16, 32), 9: (8, 16, 32), 3: (8,)}[anchors]
    b = wl.NetBuilder("proposal_ranking")
    b.input([("rpn_cls_prob", (images, 2 * anchors, h, w)), ("rpn_bbox_pred", (images, 4 * anchors, h, w)), ("im_info", (images, 3))])
    b.raw("proposal", "Proposal", ["rpn_cls_prob", "rpn_bbox_pred", "im_info"], ["rois", "scores"],
          "proposal_param { feat_stride: 16 base_size: 16 min_size: %d pre_nms_topn: %d post_nms_topn: %d nms_thresh: %g "
          "ratio: 0.5 ratio: 1 ratio: 2 %s }" % (min_size, pre, post, thr, " ".join("scale: %d" % s for s in scales)))
    feeds = [wl.proposal_input(num_anchors=anchors, height=h, width=w, seed=300 + i, im_h=16.0 * h, im_w=16.0 * w)[0]
             for i in range(images)]
    want_rois, want_scores = [], []
    for i, f in enumerate(feeds):
        scores = f["rpn_cls_prob"]
        if levels:
            f["rpn_cls_prob"], scores = _ties(scores, levels)
        rois, kept = port.proposal(scores, f["rpn_bbox_pred"], f["im_info"], [0.5, 1.0, 2.0], scales, min_size=min_size,
                                   pre_nms_topn=pre, post_nms_topn=post, nms_thresh=thr)
        rois[:, 0] = i
        want_rois.append(rois)
        want_scores.append(kept)
    net = capi.Net(gpu_engine, b.text(), None, from_buffer=True)
    feed = {k: np.concatenate([f[k] for f in feeds]) for k in feeds[0]}
    for again in range(2):      # the second pass finds its input on the device
        net.forward(**feed) if again == 0 else net.forward()
        rois, kept = net.blob("rois").data.copy(), net.blob("scores").data.copy()
        assert np.array_equal(rois.view(np.uint32), np.concatenate(want_rois).view(np.uint32))
        if not levels:
            assert np.array_equal(kept.view(np.uint32), np.concatenate(want_scores).view(np.uint32))
    net.close()


@pytest.mark.parametrize("case", [
    (9, 6, 5, 6000, 5000, 0.7, 16, 3, 0),       # 270 proposals, room asked for 5000
    (9, 24, 25, 900, 16000, 0.9, 0, 2, 0),      # the cut at pre_nms_topn below it
], ids=lambda c: "x".join(str(v) for v in c))
def test_more_asked_for_than_there_is(capi, gpu_engine, case):
    test_ranking_against_the_restatement(capi, gpu_engine, case)
