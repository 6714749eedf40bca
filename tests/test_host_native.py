"""The native walk over a net's parameters (csrc/host.cpp)."""
import copy

import pytest
import torch
import torch.nn as nn
from torch._subclasses.fake_tensor import FakeTensorMode
from torch.nn.utils import parametrize, prune

import dlr_lock_b200 as D
from dlr_lock_b200.build import build_library


def test_any_change_of_a_parameter_is_seen():
    build_library()
    host = D._lib.host()
    net = D.DLRNet(32, 4, 3)
    dicts = net._param_dicts
    key = host.snapshot(dicts())
    assert len(key) == 16 * 12 and host.unchanged(key, dicts())
    with torch.no_grad():
        net.Us[2].mul_(2.0)                                    # in place
    assert not host.unchanged(key, dicts())
    key = host.snapshot(dicts())
    net.Vs[1].data = torch.zeros(4, 32)                        # another storage behind the same parameter
    assert not host.unchanged(key, dicts())
    key = host.snapshot(dicts())
    net.alphas[0] = nn.Parameter(torch.tensor(1.0))            # another parameter
    assert not host.unchanged(key, dicts())
    key = host.snapshot(dicts())
    net.rms_w.append(nn.Parameter(torch.ones(32)))             # one more
    assert not host.unchanged(key, dicts()) and host.unchanged(host.snapshot(dicts()), dicts())
    # parameters on the CPU are not for the fold kernel
    assert host.layers(dicts()) is None and host.state_layers(net.state_dict()) is None


class _Scaled(nn.Module):
    def forward(self, w):
        return 0.5 * w


def _pruned(net):
    prune.l1_unstructured(net.Vs, "0", 0.5)


def _prune_removed(net):                                       # a plain parameter again, but last in the list's own dict
    prune.l1_unstructured(net.Vs, "0", 0.5)
    prune.remove(net.Vs, "0")


def _parametrized_one(net):
    parametrize.register_parametrization(net.Vs, "0", _Scaled())


def _parametrized_all(net):
    for p in (net.Vs, net.Us, net.rms_w, net.alphas):
        parametrize.register_parametrization(p, "1", _Scaled())


@pytest.mark.parametrize("change", [None, _pruned, _prune_removed, _parametrized_one, _parametrized_all])
def test_layers_are_folded_as_the_lists_give_them(change, monkeypatch):
    build_library()
    monkeypatch.setattr(D.ops, "fold_weights", lambda V, U, w, a: (V * w[:, None, :], a[:, None, None] * U))
    torch.manual_seed(0)
    net = D.DLRNet(32, 4, 3, alpha_init=0.7)
    with torch.no_grad():
        for i in range(3):
            net.rms_w[i].normal_(1.0, 0.1)
    if change is not None:
        change(net)

    def check():
        Vp, Up = net.folded_weights()
        for i in range(3):
            assert torch.equal(Vp[i], net.Vs[i] * net.rms_w[i]) and torch.equal(Up[i], net.alphas[i] * net.Us[i]), i

    with torch.no_grad():
        check()
        if change in (None, _pruned, _prune_removed):
            assert net.folded_weights()[0] is net.folded_weights()[0]          # nothing changed: not folded again
        # an edit below a parametrization moves a tensor that is computed on each access
        getattr(net.Vs.parametrizations, "0").original.mul_(2.0) if change is _parametrized_one else net.Vs[0].mul_(2.0)
        check()
    if change in (None, _parametrized_one, _parametrized_all):
        net.folded_weights()                                   # with gradients on: the module can still be copied
        copy.deepcopy(net).folded_weights()


def test_tensors_without_memory_of_their_own_raise_or_are_left_to_torch():
    build_library()
    host = D._lib.host()
    one = lambda v: tuple({"0": t} for t in (v, v.detach().mT.contiguous(), torch.ones(32), torch.ones(())))

    def layer(v):                                              # a batch of layers, of which none has an address
        assert host.layers(one(v)) is None
        for call in (host.snapshot, lambda dicts: host.unchanged(b"", dicts)):
            with pytest.raises(RuntimeError):
                call(one(v))
        return v.sum()

    V = torch.randn(2, 4, 32)
    torch.vmap(layer)(V)
    torch.func.grad(layer)(V[0])
    with FakeTensorMode():
        fake = [torch.empty(s, device="cuda", dtype=torch.bfloat16) for s in ((4, 32), (32, 4), (32,), ())]
        assert host.layers(tuple({"0": t} for t in fake)) is None
        assert host.state_layers(dict(zip(("Vs.0", "Us.0", "rms_w.0", "alphas.0"), fake))) is None
        torch.vmap(lambda v: (host.layers(({"0": v},) + tuple({"0": t} for t in fake[1:])), v)[1])(torch.stack([fake[0]] * 2))


def test_parameters_whose_edits_are_not_counted_are_refused():
    build_library()
    with torch.inference_mode():
        net = D.DLRNet(32, 4, 3)
        with pytest.raises(RuntimeError, match="version counter"):
            net.folded_weights()
        key = b"\0" * (16 * 12)
        with pytest.raises(RuntimeError, match="version counter"):
            D._lib.host().unchanged(key, net._param_dicts())


def test_a_key_of_another_kind_counts_as_changed(monkeypatch):
    # a module that was saved whole, by a version whose key was a tuple
    build_library()
    monkeypatch.setattr(D.ops, "fold_weights", lambda V, U, w, a: (V * w[:, None, :], a[:, None, None] * U))
    net = D.DLRNet(32, 4, 3)
    net._folded = (tuple(range(24)), None, None)
    Vp, Up = net.folded_weights()
    assert torch.equal(Vp[2], net.Vs[2] * net.rms_w[2])


def test_a_helper_built_against_another_torch_is_not_loaded(monkeypatch):
    build_library()
    monkeypatch.setattr(D._lib, "_host_module", None)
    monkeypatch.setattr(torch, "__version__", "0.0")
    with pytest.raises(RuntimeError, match="build"):
        D._lib.host()
