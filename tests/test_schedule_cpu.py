"""The schedule a net is given (which layers are fused, which share a launch), which is decided without a device."""
import os

import pytest

from conftest import pkg


def _schedule(capi, engine, builder):
    net = capi.Net(engine, builder.text(), None, from_buffer=True)
    steps = net.schedule()
    net.close()
    return steps


def test_resnet50_stages_share_launches(capi, engine):
    """One image: every stage's projection runs with the reduction beside it.  64 images: not the first stage's, whose
    64 + 256 columns split tiles of 256."""
    wl = pkg("workloads")
    for batch, stages in ((1, "2345"), (64, "345")):
        steps = _schedule(capi, engine, wl.resnet50(batch))
        assert [s for s in steps if len(s) == 2] == [["res%sa_branch1" % i, "res%sa_branch2a" % i] for i in stages]
        names = [name for s in steps for name in s]
        assert len(names) == len(set(names))
        launched = [row[0] for row in wl.resnet50_conv_table() if row[0] not in names]
        assert launched == []


@pytest.mark.parametrize("batch,fused", [(5, False), (6, True), (32, True)])
def test_pooling_in_the_store_by_rows(capi, engine, batch, fused):
    wl = pkg("workloads")
    b = wl.NetBuilder("pooled")
    b.input([("data", (batch, 64, 56, 56))])
    b.conv("trunk", "data", "trunk", 64, 64, 1)
    b.conv("conv", "trunk", "conv", 64, 64, 3, pad=1)
    b.pool("pool", "conv", "pool", "MAX", k=2, stride=2)
    b.conv("last", "pool", "last", 64, 8, 1)
    assert (["pool"] not in _schedule(capi, engine, b)) == fused


@pytest.mark.parametrize("cout", [64, 128])
@pytest.mark.parametrize("batch", [6, 16, 32])
def test_a_layer_with_a_fused_pooling_keeps_its_launch(capi, engine, batch, cout):
    wl = pkg("workloads")
    b = wl.NetBuilder("pooled_sibling")
    b.input([("data", (batch, 64, 56, 56))])
    b.conv("trunk", "data", "trunk", 64, 64, 1)
    b.conv("plain", "trunk", "plain", 64, cout, 3, pad=1)
    b.conv("conv", "trunk", "conv", 64, 64, 3, pad=1)
    b.pool("pool", "conv", "pool", "MAX", k=2, stride=2)
    b.conv("last", "pool", "last", 64, 8, 1)
    steps = _schedule(capi, engine, b)
    assert ["plain"] in steps and ["conv"] in steps and ["pool"] not in steps


def test_without_merging_every_layer_has_a_step(capi, engine, monkeypatch):
    wl = pkg("workloads")
    monkeypatch.setenv("MCB200_SIBLINGS", "0")
    assert all(len(s) == 1 for s in _schedule(capi, engine, wl.ssd300_vgg16(1)))
    monkeypatch.setenv("MCB200_SIBLINGS", "1")
    heads = [s for s in _schedule(capi, engine, wl.ssd300_vgg16(1)) if len(s) == 2]
    assert len(heads) == 6 and all(s[0].endswith("mbox_loc") and s[1].endswith("mbox_conf") for s in heads)


def test_bench_rows_follow_the_schedule(capi, engine):
    import importlib.util
    from conftest import ROOT
    spec = importlib.util.spec_from_file_location("bench_rows", os.path.join(ROOT, "bench.py"))
    bench = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(bench)
    wl = pkg("workloads")
    table = wl.resnet50_conv_table()
    rows = bench.launch_rows(table, _schedule(capi, engine, wl.resnet50(64)))
    assert len(rows) == len(table) - 3
    assert sum(r[1] * r[2] * r[3] ** 2 * r[6] ** 2 for r in rows) == sum(r[1] * r[2] * r[3] ** 2 * r[6] ** 2 for r in table)
