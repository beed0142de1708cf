"""Mlp.adam takes one gradient per layer from each list, whatever else the lists
hold, and refuses a list that is too short before anything is launched."""
import ctypes as C
import types

import pytest


def _net(monkeypatch, calls):
    import torch
    from ps_claude_opt_b200 import screen

    def record(count, n, w, g, m, v, wb, *rest):
        calls.append([(w[i], g[i]) for i in range(min(count, len(g)))])
        return 0

    monkeypatch.setattr(screen, "_lib", lambda: types.SimpleNamespace(ps_adam_steps=record))
    net = object.__new__(screen.Mlp)
    net.W = [torch.zeros((4, 3)), torch.zeros((1, 4))]
    net.b = [torch.zeros(4), torch.zeros(1)]
    net.Wb = [torch.zeros_like(w, dtype=torch.bfloat16) for w in net.W]
    net.mW, net.vW = ([torch.zeros_like(w) for w in net.W] for _ in range(2))
    net.mb, net.vb = ([torch.zeros_like(b) for b in net.b] for _ in range(2))
    net.steps = 0
    net._stream = lambda: C.c_void_p(0)
    return net


@pytest.mark.parametrize("more", [0, 1])
def test_each_layer_gets_its_gradient(monkeypatch, more):
    import torch

    calls = []
    net = _net(monkeypatch, calls)
    gW = [torch.ones_like(w) for w in net.W] + [torch.ones(5)] * more
    gb = [torch.ones_like(b) for b in net.b] + [torch.ones(5)] * more
    net.adam(gW, gb)
    want = [(w.data_ptr(), g.data_ptr()) for w, g in zip(net.W + net.b, gW[:2] + gb[:2])]
    assert calls == [want]


@pytest.mark.parametrize("n_w,n_b", [(1, 2), (2, 1), (0, 0)])
def test_short_lists_are_refused(monkeypatch, n_w, n_b):
    import torch

    calls = []
    net = _net(monkeypatch, calls)
    gW = [torch.ones_like(w) for w in net.W][:n_w]
    gb = [torch.ones_like(b) for b in net.b][:n_b]
    with pytest.raises(IndexError):
        net.adam(gW, gb)
    assert calls == []
