"""Folding from unstacked tensors: the vector kernel and its scalar form, more layers than one launch takes, fp32 and bf16
parameters.  Bit-identical to the same arithmetic in torch on the CPU."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,r,L", [(2048, 64, 3), (8, 1, 2), (264, 40, 130), (1022, 3, 5), (16, 16, 257)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("round_alpha", [False, True])
def test_fold_layers(d, r, L, dtype, round_alpha):
    import dlr_lock_b200 as D
    g = torch.Generator().manual_seed(d + L)
    make = lambda *s: [torch.randn(s, generator=g).to(dtype) for _ in range(L)]
    V, U, w, a = make(r, d), make(d, r), make(d), make()
    groups = [[t.cuda() for t in x] for x in (V, U, w, a)]
    found = D._lib.host().layers(tuple({str(i): t for i, t in enumerate(x)} for x in groups))
    assert found is not None and found[:3] == (L, r, d)
    Vp, Up = D.ops.fold_layers(found, round_alpha)
    bf = lambda x: torch.stack(x).to(torch.bfloat16).float()
    alpha = torch.stack(a).float()
    if round_alpha:
        alpha = alpha.to(torch.bfloat16).float()
    assert torch.equal(Vp.cpu(), (bf(V) * bf(w)[:, None, :]).to(torch.bfloat16))
    assert torch.equal(Up.cpu(), (bf(U) * alpha[:, None, None]).to(torch.bfloat16))


def test_unaligned_and_unusual_parameters_take_the_general_way():
    import dlr_lock_b200 as D
    torch.manual_seed(0)
    net = D.DLRNet(64, 8, 3, alpha_init=0.5)
    sd = {k: v.to(torch.bfloat16).cuda() for k, v in net.state_dict().items()}
    want = D.pack_state_dict(sd, "cuda")
    flat = torch.empty(8 * 64 + 1, device="cuda", dtype=torch.bfloat16)
    off = flat[1:].view(8, 64).copy_(sd["Vs.1"])                        # two bytes off a 16-byte boundary
    got = D.pack_state_dict(dict(sd, **{"Vs.1": off}), "cuda")
    mixed = D.pack_state_dict(dict(sd, **{"Us.2": sd["Us.2"].t().contiguous().t()}), "cuda")     # not contiguous
    for p in (got, mixed):
        assert torch.equal(p.Vp, want.Vp) and torch.equal(p.Up, want.Up)


def test_what_is_not_a_net_is_refused():
    import dlr_lock_b200 as D
    torch.manual_seed(0)
    sd = {k: v.to(torch.bfloat16).cuda() for k, v in D.DLRNet(64, 8, 3).state_dict().items()}
    D.pack_state_dict(dict(sd, **{"Vs.extra": sd["Vs.0"]}), "cuda")             # (not a layer's name)
    for key in ("Vs.3", "Vs.70000", "_orig_mod.alphas.4"):
        with pytest.raises(ValueError):
            D.pack_state_dict(dict(sd, **{key: sd["Vs.0"]}), "cuda")
