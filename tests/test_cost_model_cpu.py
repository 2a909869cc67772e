"""The learned selector's host side, without a GPU: what its calls hand to the library."""
import pytest


class _Library:
    """Records the Adam call instead of launching it."""

    def ttcb_mlp_adam_multi(self, count, params, grads, m, v, n, *rest):
        self.call = (count, [list(x) for x in (params, grads, m, v)], list(n), rest)
        return 0


def _bare_net(monkeypatch):
    import torch
    from ttc_b200 import cost_model
    net = object.__new__(cost_model.MLP)
    shapes = [(3, 128), (128,), (128, 128), (128,), (128, 1), (1,)]
    net.params, net.m, net.v = ([torch.zeros(s) for s in shapes] for _ in range(3))
    net.t = 0
    lib = _Library()
    monkeypatch.setattr(cost_model, "_lib", lambda: lib)
    monkeypatch.setattr(cost_model, "_s", lambda: 0)
    return net, lib


@pytest.mark.parametrize("given", [6, 4, 1])
@pytest.mark.parametrize("lazy", [False, True])
def test_step_updates_as_many_tensors_as_gradients_are_given(monkeypatch, given, lazy):
    """MLP.step pairs parameters with gradients one by one: a shorter list, or any iterable, updates the
    leading parameters only, and no array that the library reads is shorter than its count."""
    import torch
    net, lib = _bare_net(monkeypatch)
    grads = [torch.zeros_like(p) for p in net.params[:given]]
    net.step((g for g in grads) if lazy else grads)
    count, arrays, n, _ = lib.call
    assert count == given and n == [p.numel() for p in net.params[:given]]
    for got, want in zip(arrays, (net.params, grads, net.m, net.v)):
        assert got == [t.data_ptr() for t in want[:given]]


def test_step_without_gradients_updates_nothing(monkeypatch):
    net, lib = _bare_net(monkeypatch)
    net.step([])
    assert net.t == 1 and not hasattr(lib, "call")
