"""Scratch of the proposal kernels: what they ask for follows what an image can keep, so that a large post_nms_topn over
a small map does not take a batch past the fixed scratch of the allocation-free entry."""
import ctypes

import pytest


class ProposalParams(ctypes.Structure):
    _fields_ = [(n, ctypes.c_int) for n in ("num_anchors", "height", "width", "feat_stride", "min_size", "pre_nms_topn",
                                            "post_nms_topn")] + [("nms_thresh", ctypes.c_float)]


@pytest.mark.parametrize("anchors,height,width,pre,post,batch", [
    (9, 4, 4, 6000, 5000, 64), (9, 1, 2, 6000, 300, 1500), (15, 63, 38, 6000, 300, 7), (9, 14, 14, 12000, 16000, 24),
    (15, 24, 24, 700, 9000, 20), (3, 8, 8, 100, 2000, 400)])
def test_workspace_follows_the_boxes(kernels, anchors, height, width, pre, post, batch):
    kernels.mcb200_proposal_workspace_bytes.restype = ctypes.c_size_t
    params = ProposalParams(anchors, height, width, 16, 16, pre, post, 0.7)
    n = anchors * height * width
    k = min(n, pre)
    # boxes, scores and 64-bit keys of all proposals, boxes and scores of the ranked ones, each array on 256 bytes
    bound = sum((size * batch + 255) // 256 * 256 for size in (16 * n, 4 * n, 8 * n, 16 * k, 4 * k))
    need = kernels.mcb200_proposal_workspace_bytes(ctypes.byref(params), batch)
    assert 0 < need <= bound
