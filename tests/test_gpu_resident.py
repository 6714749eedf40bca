"""The resident-cluster kernel (path 7) where its cuts can go wrong: partial row pairs and token tiles, one cluster and
several, more clusters than can be resident, one layer, and its bounded waits."""
import ctypes

import pytest
import torch

from oracle import dlrnet_oracle as O

pytestmark = pytest.mark.gpu

# Activations in fp32, operands rounded to bf16, as in the striped kernels: same gates.
TOL_TOTAL, TOL_UPDATE = 5e-3, 2e-2

CASES = [(1024, 32, 5, M) for M in (1, 2, 3, 8, 9, 63, 267, 530, 1100)]
CASES += [(2048, 64, 4, M) for M in (1, 5, 16, 31, 121, 249, 500)]
CASES += [(4096, 128, 3, M) for M in (1, 6, 17, 57, 115, 230)]
CASES += [(5120, 256, 2, M) for M in (1, 7, 57, 113, 226)]
CASES += [(1024, 32, 1, 4), (2048, 64, 1, 4), (4096, 128, 1, 20), (5120, 256, 1, 3)]


@pytest.mark.parametrize("d,r,L,M", CASES)
def test_resident_kernel(d, r, L, M, monkeypatch):
    import dlr_lock_b200 as D
    monkeypatch.setenv("DLRB200_FORCE_PATH", "7")
    dev = torch.device("cuda:0")
    p, x = O.seeded_case(d, r, L, M, seed=d + L + M, alpha=1.0, gain_jitter=0.1)
    plan = D.ops.query_call(M, d, r, L)
    assert plan.path == 7 and plan.rows_per_pass * (plan.grid // plan.cluster) >= M
    Vf, Uf = D.ops.fold_weights(p.V.to(dev), p.U.to(dev), p.w.to(dev), p.alpha.to(dev))
    buf = torch.full((M + 2, d), 7.0, device=dev, dtype=torch.bfloat16)          # rows around the output stay as they are
    y1 = D.ops.forward_folded(x.to(dev), Vf, Uf, p.eps, out=buf[1:M + 1])
    y2 = D.ops.forward_folded(x.to(dev), Vf, Uf, p.eps)
    torch.cuda.synchronize()
    D.ops.check_status()
    assert torch.equal(y1, y2)                                                   # sums in a fixed order
    assert bool((buf[0] == 7.0).all()) and bool((buf[M + 1] == 7.0).all())
    want = O.forward_fp32(x, p)
    assert O.rel_l2(y1.cpu(), want) <= TOL_TOTAL
    assert O.rel_l2_update_q(y1.cpu(), want, x) <= TOL_UPDATE


# Calls whose any-shape kernel works in fp32 throughout (one cluster per pair of rows): operands of three bf16 terms here.
# One row and two in the last cluster, one cluster and several, one layer.  The result is that of 64 bits rounded once, but
# for ties: an error e before the rounding moves at most 512 e of the values to their neighbour (a bf16 spacing is at least
# 2^-8 of a value), and e is about 1e-6 for fp32 sums of 256 products over the layers here.  Operands of 8 bits move 5 to 18 %.
@pytest.mark.parametrize("d,r,L,M", [(1024, 32, 1, 2), (1024, 32, 141, 2), (1024, 32, 4, 3), (1024, 32, 20, 8), (1024, 32, 7, 63), (1024, 32, 30, 64),
                                     (2048, 64, 1, 17), (2048, 64, 142, 17), (2048, 64, 20, 28), (2048, 64, 5, 27)])
def test_pair_of_rows_in_fp32(d, r, L, M):
    import dlr_lock_b200 as D
    dev = torch.device("cuda:0")
    p, x = O.seeded_case(d, r, L, M, seed=d + L + M, alpha=1.0, gain_jitter=0.1)
    Vf, Uf = D.ops.fold_weights(p.V.to(dev), p.U.to(dev), p.w.to(dev), p.alpha.to(dev))
    y = D.ops.forward_folded(x.to(dev), Vf, Uf, p.eps)
    again = D.ops.forward_folded(x.to(dev), Vf, Uf, p.eps)
    torch.cuda.synchronize()
    D.ops.check_status()
    assert torch.equal(y, again)
    h = x.to(dev).double()
    for V, U in zip(Vf.double(), Uf.double()):
        z = (h @ V.T) * torch.rsqrt(h.square().mean(-1, keepdim=True) + p.eps)
        h = h + torch.nn.functional.silu(z) @ U.T
    assert (y != h.to(torch.bfloat16)).double().mean() <= 1e-3
    assert O.rel_l2(y.double(), h) <= 1.01 * O.rel_l2(h.to(torch.bfloat16), h)


# every kernel of every shape, on stacks that may be asked for whole before anyone gives up: copies still land while the rest
# leaves
@pytest.mark.parametrize("L", [1, 2, 6])
@pytest.mark.parametrize("d,r,M", [(1024, 32, 1), (1024, 32, 8), (1024, 32, 267), (1024, 32, 530), (1024, 32, 1100), (2048, 64, 4), (2048, 64, 20),
                                   (2048, 64, 200), (2048, 64, 400), (4096, 128, 1), (4096, 128, 115), (4096, 128, 200), (5120, 256, 3),
                                   (5120, 256, 115), (5120, 256, 200)])
def test_resident_kernel_gives_up_while_the_status_word_is_set(d, r, L, M, monkeypatch):
    # the word an earlier kernel would have left behind, set by the host: the call returns, leaves its output and the word
    # alone, and the next call on a cleared word works
    import dlr_lock_b200 as D
    monkeypatch.setenv("DLRB200_FORCE_PATH", "7")
    dev = torch.device("cuda:0")
    p, x = O.seeded_case(d, r, L, M, seed=9, alpha=1.0, gain_jitter=0.1)
    Vf, Uf = D.ops.fold_weights(p.V.to(dev), p.U.to(dev), p.w.to(dev), p.alpha.to(dev))
    xd = x.to(dev)
    D.ops.forward_folded(xd, Vf, Uf)
    torch.cuda.synchronize()
    D.ops.check_status()
    ent = D.ops._workspaces[(0, torch.cuda.current_stream(dev).cuda_stream)]
    ent.status.fill_(0x307)
    torch.cuda.synchronize()
    out = torch.full_like(xd, 7.0)
    lib = D.ops._lib.load()
    vp = lambda t: ctypes.c_void_p(t.data_ptr())                    # (the tensor call would raise before it launches)
    st = ctypes.c_void_p(torch.cuda.current_stream(dev).cuda_stream)
    assert lib.dlrb200_forward(vp(xd), vp(out), vp(Vf), vp(Uf), M, d, r, L, 1e-6, vp(ent.ws), ent.ws.numel(), vp(ent.status), st) == 0
    torch.cuda.synchronize()
    assert bool((out == 7.0).all())
    with pytest.raises(D.ops._lib.DlrB200Error):                    # reported for this call too
        D.ops.forward_folded(xd, Vf, Uf)
    D.ops.check_status()                                            # and cleared
    y = D.ops.forward_folded(xd, Vf, Uf)
    torch.cuda.synchronize()
    D.ops.check_status()
    assert O.rel_l2(y.cpu(), O.forward_fp32(x, p)) <= TOL_TOTAL

