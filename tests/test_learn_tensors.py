"""The optimiser works on the tensors that the network holds when it is called, on
the CPU: the calls into the library are recorded instead of made."""
import pytest
import torch

from sources_b200 import learn


@pytest.fixture
def net(monkeypatch):
    monkeypatch.setattr(learn.MPNet, "stream", property(lambda self: 0))
    net = learn.MPNet(device="cpu", seed=1)
    net.seen = []

    def record(fn, *args):
        if fn == "sphg_gnn_adam_all":
            lst = learn.AdamList.from_address(args[0])
            net.seen.append([tuple(getattr(lst.t[i], k) or 0 for k in ("w", "g", "m", "v", "wb", "wt")) for i in range(lst.count)])
    monkeypatch.setattr(net, "_k", record)
    return net


def pointers(net):
    return [tuple(learn._ptr(d.get(k)) for k in ("w", "g", "m", "v", "wb", "wt"))
            for d in list(net.W.values()) + list(net.B.values())]


def test_replaced_tensors_are_used(net):
    net.adam(1e-3)
    assert net.seen[-1] == pointers(net)
    for d, keys in ((net.W["dec.w1"], ("w", "m", "wb")), (net.B["p0.c1"], ("v",)), (net.W["p0.v1"], ("g",))):
        for k in keys:
            d[k] = d[k].clone()
    net.adam(1e-3)
    assert net.seen[-1] == pointers(net) != net.seen[0]


def test_replaced_gradients_are_cleared(net):
    net.W["p0.v1"]["g"] = torch.ones_like(net.W["p0.v1"]["g"])
    net.B["dec.b1"]["g"].fill_(2.0)
    net.zero_grad()
    assert all(not d["g"].any() for d in list(net.W.values()) + list(net.B.values()))
