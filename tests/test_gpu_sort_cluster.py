"""The clustered label sort at the sizes where its split changes: token counts around whole groups of 32,
one to sixteen CTAs per head, cluster counts around the threads of a CTA."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("BH,N,K", [(1, 1, 1), (2, 31, 7), (1, 1023, 3), (3, 1024, 512), (2, 8191, 513), (1, 16385, 1024),
                                    (5, 40001, 100), (450, 97, 33)])
def test_sort_matches_stable_argsort(BH, N, K):
    from svoo_b200 import ops
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev).manual_seed(N)
    lab = torch.randint(0, K, (BH, N), generator=gen, device=dev, dtype=torch.int32)
    lab[:, : N // 3] = K // 2                                      # long stretches of one label
    idx, off = ops.sort_labels(lab, K)
    assert torch.equal(idx.long(), torch.argsort(lab, dim=1, stable=True))
    want = torch.zeros(BH, K + 1, dtype=torch.long, device=dev)
    want[:, 1:] = torch.stack([torch.bincount(r, minlength=K) for r in lab.long()]).cumsum(1)
    assert torch.equal(off.long(), want)


@pytest.mark.parametrize("J", [100, 129, 300, 600, 1024])
def test_sort_reduces_the_assignment_winners(J):
    """Labels that the co-clustering's sort reduces itself = those of the labels-only call, for every group count."""
    from svoo_b200 import ops
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev).manual_seed(J)
    x = torch.randn(2, 5003, 128, generator=gen, device=dev).to(torch.bfloat16)
    qi = torch.randint(0, 5003, (2, 64), generator=gen, device=dev)
    ki = torch.randint(0, 5003, (2, J), generator=gen, device=dev)
    c = ops.cocluster(x, x, qi, ki, 1)
    q0, k0 = (torch.gather(x, 1, i[..., None].expand(-1, -1, 128)) for i in (qi, ki))
    klab = ops.cocluster_assign(x, q0, k0)
    assert torch.equal(c.klabels, klab)
    assert torch.equal(c.k_sorted_idx.long(), torch.argsort(klab, dim=1, stable=True))
    assert torch.equal(c.ksizes.long(), torch.stack([torch.bincount(r, minlength=J) for r in klab.long()]))


@pytest.mark.parametrize("K", [1, 31, 33, 256, 257, 500, 511, 513, 1023])
def test_sort_of_sixteen_ctas_with_partial_warps(K):
    """Sixteen CTAs per head with cluster counts that end inside a warp: its lanes meet the cluster barriers from
    loops of different lengths."""
    from svoo_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(K)
    lab = torch.randint(0, K, (3, 40003), generator=gen, device="cuda", dtype=torch.int32)
    idx, off = ops.sort_labels(lab, K)
    assert torch.equal(idx.long(), torch.argsort(lab, dim=1, stable=True))
    assert torch.equal(off[:, 1:].long(), torch.stack([torch.bincount(r, minlength=K) for r in lab.long()]).cumsum(1))
