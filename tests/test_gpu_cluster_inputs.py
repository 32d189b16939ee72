"""Clustering inputs that are views: read in place where their rows allow it, copied otherwise."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["leading rows", "every other head", "different spacing", "transposed", "expanded", "offset"])
def test_views_cluster_like_copies(form):
    """Whatever the strides, the result is that of contiguous copies (bit for bit: the kernels are deterministic)."""
    from svoo_b200 import co_clustering as cc
    H, S, N = 3, 900, 777
    gen = torch.Generator(device="cuda").manual_seed(1)
    q, k = (torch.randn(2 * H, S, 128, generator=gen, device="cuda").to(torch.bfloat16) for _ in range(2))
    if form == "leading rows":
        q, k = q[:H, :N], k[:H, :N]
    elif form == "every other head":
        q, k = q[::2, :N], k[::2, :N]
    elif form == "different spacing":
        q, k = q[:H, :N], k[::2, :N]
    elif form == "transposed":
        q, k = (t.transpose(0, 1).contiguous().transpose(0, 1)[:H, :N] for t in (q, k))
    elif form == "expanded":
        q, k = (t[:1, :N].expand(H, N, 128) for t in (q, k))
    else:
        q, k = q[:H, 100:100 + N], k[:H, 100:100 + N]
    init = tuple(torch.randint(0, N, (H, c), generator=gen, device="cuda") for c in (20, 70))
    a = cc.co_cluster(q, k, 20, 70, 3, init_indices=init)
    b = cc.co_cluster(q.contiguous(), k.contiguous(), 20, 70, 3, init_indices=init)
    for x, y in zip(vars(a).values(), vars(b).values()):
        assert torch.equal(x, y)
