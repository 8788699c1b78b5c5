"""Which buffers the network's library calls get (CPU, the calls recorded): the
whole ones while every tensor lies where the constructor put it, the tensors'
own as soon as a caller replaced one or gave it other storage."""
import pytest
import torch

from blade_b200 import _lib
from blade_b200 import mlp


@pytest.fixture
def net(monkeypatch):
    calls = []
    monkeypatch.setattr(_lib, "call", lambda name, *a: calls.append((name, [getattr(x, "value", x) for x in a])))
    monkeypatch.setattr(mlp.BF16MLP, "_s", lambda self: None)
    n = mlp.BF16MLP([24, 16, 8], max_batch=4, device="cpu")
    calls.clear()
    n.calls = calls
    return n


def _replace_data(n):
    n.W[0].data = torch.full_like(n.W[0], 0.5)
    return n.W[0]


def _replace_tensor(n):
    n.gW[1] = n.gW[1] * 0.5
    return n.gW[1]


def _replace_bias_data(n):
    n.b[1].data = torch.ones(8)
    return n.b[1]


def test_whole_buffers(net):
    net.adam_step()
    net._sync_bf16()
    assert [c[0] for c in net.calls] == ["bnb_mlp_adam", "bnb_to_bf16"]
    assert net.calls[0][1][1] == net._p.data_ptr() == net.W[0].data_ptr()
    net.W[0].copy_(torch.ones(16, 24))                    # in place: still the whole buffers
    net.calls.clear()
    net.adam_step(weight_decay=0.1)
    assert [c[1][0] for c in net.calls] == [net._nW, net._p.numel() - net._nW]


@pytest.mark.parametrize("replace", [_replace_data, _replace_tensor, _replace_bias_data])
def test_replaced_storage_is_the_one_used(net, replace):
    t = replace(net)
    net.adam_step()
    if t is net.W[0]:
        net._sync_bf16()
    names = [c[0] for c in net.calls]
    assert names.count("bnb_mlp_adam") == 4
    assert any(t.data_ptr() in c[1] for c in net.calls)
    assert net._p.data_ptr() not in [a for c in net.calls if t is net.W[0] for a in c[1]]
