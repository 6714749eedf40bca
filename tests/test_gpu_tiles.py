"""Tensor-core kernels where their tiles can go wrong: partial tiles, one layer, several tiles per CTA."""
import pytest
import torch

from oracle import dlrnet_oracle as O

pytestmark = pytest.mark.gpu

# Activations in bf16 between layers, operands rounded to bf16: the gates of the other large-batch tests.
TOL_MODEL, TOL_TOTAL, TOL_UPDATE = 6e-3, 1e-2, 5e-2


def _check(d, r, L, M, path):
    import dlr_lock_b200 as D
    dev = torch.device("cuda:0")
    p, x = O.seeded_case(d, r, L, M, seed=d + r + L + M, alpha=1.0, gain_jitter=0.1)
    assert D.ops.query_call(M, d, r, L).path == path
    Vf, Uf = D.ops.fold_weights(p.V.to(dev), p.U.to(dev), p.w.to(dev), p.alpha.to(dev))
    buf = torch.full((M + 2, d), 7.0, device=dev, dtype=torch.bfloat16)          # rows around the output stay as they are
    y = D.ops.forward_folded(x.to(dev), Vf, Uf, p.eps, out=buf[1:M + 1])
    again = D.ops.forward_folded(x.to(dev), Vf, Uf, p.eps)
    torch.cuda.synchronize()
    D.ops.check_status()
    assert torch.equal(y, again)
    assert bool((buf[0] == 7.0).all()) and bool((buf[M + 1] == 7.0).all())
    model = O.forward_folded_fp32(x, Vf.cpu(), Uf.cpu(), p.eps, round_h=True)
    want = O.forward_fp32(x, p)
    assert O.rel_l2(y.cpu(), model) <= TOL_MODEL
    assert O.rel_l2(y.cpu(), want) <= TOL_TOTAL
    assert O.rel_l2_update(y.cpu(), want, x) <= TOL_UPDATE


# rank 256, two halves per chunk: four chunks (the fewest) and more, a split of 1, 2 and 4, several tiles per CTA
@pytest.mark.parametrize("d,L,M", [(512, 1, 65), (512, 2, 129), (640, 3, 128), (1024, 2, 66), (2048, 3, 257), (5120, 1, 130),
                                   (512, 2, 148 * 128 + 130)])
def test_streamed_rank_256(d, L, M, monkeypatch):
    monkeypatch.setenv("DLRB200_FORCE_PATH", "4")
    _check(d, 256, L, M, 4)


# the cluster kernel: both stripes, partial tiles, one layer, fewer and more tiles than clusters fit on the GPU at once
@pytest.mark.parametrize("stripe", [512, 256])
@pytest.mark.parametrize("d,r,L,M", [(512, 32, 3, 65), (512, 64, 2, 129), (512, 128, 1, 130), (1024, 32, 3, 257), (1024, 64, 1, 100),
                                     (1024, 128, 2, 384), (2048, 64, 2, 333), (2048, 128, 3, 128), (4096, 128, 2, 200),
                                     (512, 32, 2, 148 * 128 + 70), (1024, 32, 2, 74 * 128 + 1), (2048, 128, 2, 37 * 128 + 70)])
def test_cluster_kernel(d, r, L, M, stripe, monkeypatch):
    import dlr_lock_b200 as D
    monkeypatch.setenv("DLRB200_FORCE_PATH", "2")
    monkeypatch.setenv("DLRB200_CLUSTER_STRIPE", str(stripe))
    assert D.ops.query_call(M, d, r, L).stripe_cols == (512 if d > 2048 else stripe)
    _check(d, r, L, M, 2)


# the pair kernel: the fewest chunks a pair can have (eight), one, two and four pairs per cluster, one layer, several tiles
@pytest.mark.parametrize("d,r,L,M", [(512, 64, 1, 65), (512, 128, 3, 257), (640, 128, 2, 300), (1024, 64, 2, 130), (2048, 128, 2, 513),
                                     (4096, 128, 1, 300), (512, 64, 2, 74 * 256 + 1), (512, 128, 3, 150 * 256 + 70)])
def test_pair_kernel(d, r, L, M, monkeypatch):
    monkeypatch.setenv("DLRB200_FORCE_PATH", "5")
    _check(d, r, L, M, 5)


# the shortest waits on stacks that fit the rings whole: a call either says that it gave up or is right, and the next one works
@pytest.mark.parametrize("path,d,r,L,M", [(2, 1024, 32, 1, 200), (3, 1024, 64, 1, 5), (3, 512, 32, 2, 64), (4, 512, 64, 1, 65), (4, 512, 64, 2, 300), (4, 512, 256, 1, 129), (4, 1024, 128, 1, 200),
                                          (5, 512, 64, 1, 600)])
def test_a_call_that_gives_up_leaves_nothing_behind(path, d, r, L, M, monkeypatch):
    import dlr_lock_b200 as D
    monkeypatch.setenv("DLRB200_FORCE_PATH", str(path))
    dev = torch.device("cuda:0")
    p, x = O.seeded_case(d, r, L, M, seed=d + r + L, alpha=1.0, gain_jitter=0.1)
    Vf, Uf = D.ops.fold_weights(p.V.to(dev), p.U.to(dev), p.w.to(dev), p.alpha.to(dev))
    xd = x.to(dev)
    want = D.ops.forward_folded(xd, Vf, Uf, p.eps)
    torch.cuda.synchronize()
    D.ops.check_status()
    monkeypatch.setenv("DLRB200_SPIN_LIMIT", "1")
    y = D.ops.forward_folded(xd, Vf, Uf, p.eps)
    torch.cuda.synchronize()
    monkeypatch.delenv("DLRB200_SPIN_LIMIT")
    try:
        D.ops.check_status()
        assert torch.equal(y, want)
    except D.ops._lib.DlrB200Error:
        pass
    y = D.ops.forward_folded(xd, Vf, Uf, p.eps)
    torch.cuda.synchronize()
    D.ops.check_status()
    assert torch.equal(y, want)
