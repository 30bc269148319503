"""The forward passes that users of this engine run, as measurable cases.

A case is one network at one size.  `prepare` does what a program does once: builds the Net, loads its
weights, shapes the input blobs and fills their (pinned) host memory, as a decoder that writes into the blob
does.  `run` is one pass through the C API's Python binding: the inputs' host pointers are asked for, which is how a
program says that it has written new data (the engine copies the input to the device again), the net is run,
and the outputs are read on the host.

The networks are the package's own generated configurations (ResNet-50, MobileNet-v1, SSD300 on VGG16, the WGAN
generator, the region-proposal layer, SSD's DetectionOutput, the R-FCN pooling head), with random weights.
"""
import importlib
import os

import numpy as np

capi = importlib.import_module("mini-caffe_b200.capi")
wl = importlib.import_module("mini-caffe_b200.workloads")

_engine = []


def engine():
    if not _engine:
        path = os.path.join(os.path.dirname(os.path.abspath(capi.__file__)), "lib", "libcaffe.so")
        library = capi.CaffeLibrary(path)
        library.set_mode(True, 0)
        _engine.append(library)
    return _engine[0]


# --------------------------------------------------------------------------- the cases

def listed():
    return [
        # One image through the region-proposal stage of a two-stage detector: video or camera, latency counts.
        dict(name="proposal_n1", net="proposal", batch=1, height=63, width=38, anchors=15),
        # The same stage over a batch of images, as an offline job runs it (the benchmark's stress size).
        dict(name="proposal_n32", net="proposal", batch=32, height=63, width=38, anchors=15),
        # SSD300's post-processing on a batch: 8732 priors, 21 classes, scores as a trained head gives them.
        dict(name="detection_output_n32", net="detection_output", batch=32, priors=8732, classes=21),
        # R-FCN's pooling head: 300 rois over 21 x 7 x 7 score maps of one image.
        dict(name="psroi_r300", net="psroi", rois=300, height=63, width=38, classes=21),
        # The light classifier on single images: the smallest network call, launches and latency count.
        dict(name="mobilenet_b1", net="mobilenet", batch=1, size=224, precision="fp32"),
        # The light classifier in a server's batches.
        dict(name="mobilenet_b64", net="mobilenet", batch=64, size=224, precision="fp32"),
        # The standard classifier on single images.
        dict(name="resnet50_b1", net="resnet50", batch=1, size=224, precision="fp32"),
        # A medium batch in the bfloat16 mode, as a latency-bounded server runs it.
        dict(name="resnet50_b16_bf16", net="resnet50", batch=16, size=224, precision="bf16"),
        # The headline configuration of the benchmark: ordinary throughput inference.
        dict(name="resnet50_b64", net="resnet50", batch=64, size=224, precision="fp32"),
        # The detector's trunk and heads on one frame; its maps (300, 150, 75, 38, 19, 10, 5, 3, 1) are ragged.
        dict(name="ssd300_b1_bf16", net="ssd300", batch=1, precision="bf16"),
        # The detector over a batch: the largest pass.
        dict(name="ssd300_b32", net="ssd300", batch=32, precision="fp32"),
        # A generator net: deconvolutions, BatchNorm on batch statistics, TanH.
        dict(name="wgan_b64", net="wgan", batch=64, precision="fp32"),
    ]


def _log_int(rng, low, high):
    return max(low, min(high, int(round(low * (high / low) ** rng.random()))))


def draw(rng):
    net = rng.choice(["proposal", "detection_output", "psroi", "mobilenet", "mobilenet", "resnet50", "resnet50", "resnet50",
                      "ssd300", "ssd300", "wgan"])
    precision = rng.choice(["fp32", "fp32", "bf16"])
    if net == "proposal":
        return dict(net=net, batch=_log_int(rng, 1, 32), height=rng.randint(24, 63), width=rng.randint(24, 63),
                    anchors=rng.choice([9, 15]))
    if net == "detection_output":
        return dict(net=net, batch=_log_int(rng, 1, 32), priors=rng.randint(1000, 8732), classes=rng.choice([2, 21, 21]))
    if net == "psroi":
        return dict(net=net, rois=rng.randint(50, 300), height=rng.randint(30, 63), width=rng.randint(30, 63),
                    classes=rng.choice([5, 21]))
    if net == "mobilenet":
        return dict(net=net, batch=_log_int(rng, 1, 64), size=rng.randint(128, 224), precision=precision)
    if net == "resnet50":
        return dict(net=net, batch=_log_int(rng, 1, 64), size=rng.randint(160, 256), precision=precision)
    if net == "ssd300":
        return dict(net=net, batch=_log_int(rng, 1, 32), precision=precision)
    return dict(net=net, batch=_log_int(rng, 1, 64), precision="fp32")


# --------------------------------------------------------------------------- networks

def _replace_dims(text, old, new):
    return text.replace(" ".join("dim: %d" % d for d in old), " ".join("dim: %d" % d for d in new))


def _builder(case):
    """(NetBuilder, prototxt, names of the outputs a program reads)."""
    net, batch = case["net"], case.get("batch", 1)
    if net == "proposal":
        a, h, w = case["anchors"], case["height"], case["width"]
        b = wl.proposal(num_anchors=a, height=h, width=w)
        text = b.text()
        for shape in ((1, 2 * a, h, w), (1, 4 * a, h, w), (1, 3)):
            text = _replace_dims(text, shape, (batch,) + shape[1:])
        return b, text, ["rois"]
    if net == "detection_output":
        b = wl.detection_head(batch=batch, num_priors=case["priors"], num_classes=case["classes"], conf_thr=0.01, nms_thr=0.45,
                              top_k=400, keep_top_k=200)
        return b, b.text(), ["detection_out"]
    if net == "psroi":
        b = wl.roi_pooling("PSROIPooling", batch=1, height=case["height"], width=case["width"], num_rois=case["rois"],
                           output_dim=case["classes"], group_size=7)
        return b, b.text(), ["pooled"]
    if net == "ssd300":
        # Trunk and heads; the post-processing of their outputs is the detection_output case.
        b = wl.ssd300_vgg16(batch, with_detection_output=False)
        return b, b.text(), ["mbox_loc", "mbox_conf_flatten", "mbox_priorbox"]
    if net == "wgan":
        b = wl.wgan_generator(batch)
        return b, b.text(), ["image"]
    b = wl.mobilenet_v1(batch) if net == "mobilenet" else wl.resnet50(batch)
    size = case["size"]
    return b, _replace_dims(b.text(), (batch, 3, 224, 224), (batch, 3, size, size)), ["prob"]


def _weights(case, builder, seed):
    """Random weights.  ResNet-50's BatchNorm variances are set to what the layers see, as training leaves them,
    so that activations stay of order one and the class scores are not one-hot."""
    weights = wl.init_params(builder.params, seed=seed)
    if case["net"] == "resnet50":
        pixel = 255.0 ** 2 / 12 + np.mean([(127.5 - m) ** 2 for m in wl.IMAGE_MEANS])
        for name, value in weights.items():
            if name == "bn_conv1_1":
                value[...] = 2 * pixel
            elif name.startswith("bn_res") and name.endswith(("branch2a_1", "branch1_1")):
                block = "abcdefgh".index(name[len("bn_res2")])
                value[...] = 2.0 * (1 + 0.7 * block)
    return weights


def _inputs(case, seed):
    net, batch = case["net"], case.get("batch", 1)
    if net == "proposal":
        rows = [wl.proposal_input(case["anchors"], case["height"], case["width"], seed=seed * 64 + i,
                                  im_h=16.0 * case["height"], im_w=16.0 * case["width"])[0] for i in range(batch)]
        return {k: np.concatenate([r[k] for r in rows]) for k in rows[0]}
    if net == "detection_output":
        return wl.detection_head_input(batch, case["priors"], case["classes"], seed, peaked=True)
    if net == "psroi":
        return wl.roi_pooling_input(1, case["classes"] * 49, case["height"], case["width"], case["rois"], seed=seed)
    if net == "ssd300":
        return wl.ssd_input(batch, seed)
    if net == "wgan":
        return wl.wgan_noise(batch, seed=seed)
    if net == "mobilenet":
        return wl.normal_image_input(batch, case["size"], seed)
    return wl.image_input(batch, case["size"], seed)


def _build(case):
    """(builder, Net, output names), in the precision that the case asks for."""
    builder, text, outputs = _builder(case)
    key, bf16 = "MINICAFFE_PRECISION", case.get("precision") == "bf16"
    before = os.environ.get(key)
    os.environ[key] = "bf16" if bf16 else "fp32"
    try:
        net = capi.Net(engine(), text, None, from_buffer=True)
    finally:
        if before is None:
            del os.environ[key]
        else:
            os.environ[key] = before
    for name in outputs:
        net.mark_output(name)
    return builder, net, outputs


def prepare(case, seed):
    builder, net, outputs = _build(case)
    if builder.params:
        net.set_params(_weights(case, builder, seed))
    blobs = []
    for name, value in _inputs(case, seed).items():
        blob = net.blob(name)
        blob.reshape(*value.shape)
        blob.data[...] = value
        blobs.append(blob)
    return {"net": net, "inputs": blobs, "outputs": {name: net.blob(name) for name in outputs}}


def run(state):
    for blob in state["inputs"]:
        blob.data                    # the program's images of this pass are written here
    state["net"].forward()
    return {name: blob.data for name, blob in state["outputs"].items()}


# --------------------------------------------------------------------------- what a pass needs

def work(case):
    """Bytes: inputs, weights and outputs once.  Operations: the multiply-adds of the dense layers; for the
    detection layers the decoding of each box and the overlaps that a greedy suppression cannot avoid."""
    net, batch = case["net"], case.get("batch", 1)
    if net == "proposal":
        n = case["anchors"] * case["height"] * case["width"]
        # the foreground half of the scores is what the layer reads
        return {"bytes": batch * 4.0 * (n + 4 * n + 3 + 300 * 5), "flops": batch * (40.0 * n + 12.0 * 300 * 300 / 2)}
    if net == "detection_output":
        p, c = case["priors"], case["classes"]
        return {"bytes": 4.0 * (batch * (4 * p + c * p + 200 * 7) + 8 * p),
                "flops": batch * (c - 1) * (1.0 * p + 400 * 30 + 12.0 * 200 * 200 / 2)}
    if net == "psroi":
        maps, out = case["classes"] * 49 * case["height"] * case["width"], case["rois"] * case["classes"] * 49
        # a bin of an ordinary box covers about a dozen cells
        return {"bytes": 4.0 * (maps + 5 * case["rois"] + out), "flops": 12.0 * out}
    builder, holder, outputs = _build(case)
    shapes = {name: blob.shape for name, blob in holder.blobs()}
    holder.close()
    first = "z" if net == "wgan" else "data"
    params = sum(int(np.prod(shape)) for _, shape, _, _ in builder.params)
    moved = int(np.prod(shapes[first])) + params + sum(int(np.prod(shapes[o])) for o in outputs)
    flops = float(wl.conv_work(builder, shapes)["flops"])
    if net == "wgan":
        # every input value of a deconvolution meets each weight of its channel
        bottoms = ["z", "deconv0", "deconv1", "deconv2", "deconv3"]
        weights = [shape for name, shape, _, _ in builder.params if len(shape) == 4]
        flops = sum(2.0 * np.prod(shapes[b]) * np.prod(w[1:]) for b, w in zip(bottoms, weights))
    return {"bytes": 4.0 * moved, "flops": float(flops)}


def tolerance(case):
    """Detection and pooling layers decide and average in fp32 in one defined order: the same bits.  The dense nets
    multiply in TF32 (or bfloat16): a product's rounding is 3e-4 (2e-3) of it, some fifty layers in a row add
    these up to 2e-3 (1.5e-2), and softmax passes an error on about twofold."""
    if case["net"] in ("proposal", "detection_output", "psroi"):
        return "exact"
    return {"rel": 2e-2} if case["precision"] == "bf16" else {"rel": 5e-3}
