"""The attention kernels where their tilings can go wrong: query clusters around the 64 / 128 / 256-row tile
edges, key lists around the 64 / 128-key step edges, runs of single rows (more than 32 per tile), empty
clusters and empty rows of the map -- against a plain fp32 softmax.

Bound: every weight is rounded to bf16 (2^-9 relative, the weights sum to 1), the output once more
(2^-9); fp32 sums and ex2.approx are far below that: 2.5 * 2^-9 * max |v|.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _offsets(sizes, dev):
    off = torch.zeros(sizes.shape[0], sizes.shape[1] + 1, dtype=torch.int32)
    off[:, 1:] = sizes.cumsum(1)
    return off.to(dev)


def _reference(q, k, v, m, qs, ks, scale):
    out = torch.zeros_like(q, dtype=torch.float32)
    for h in range(q.shape[0]):
        rows = torch.repeat_interleave(torch.arange(qs.shape[1]), qs[h])
        cols = torch.repeat_interleave(torch.arange(ks.shape[1]), ks[h])
        keep = m[h].bool()[rows][:, cols].to(q.device)
        s = (q[h].float() @ k[h].float().T) * scale
        p = torch.softmax(s.masked_fill(~keep, float("-inf")), -1).nan_to_num(0.0)
        out[h] = p @ v[h].float()
    return out


CASES = {
    # query cluster sizes, key cluster sizes, every n-th key cluster selected (shifted by head and query cluster)
    "tile-edges": ([1, 64, 65, 128, 129, 192, 193, 256, 257, 385, 0, 2], [64, 1, 63, 128, 0, 65, 127, 900, 300, 24], 2),
    "single-row-runs": ([40, 0, 128, 33, 250, 500, 300, 6], [1] * 600 + [657], 2),
    "short-runs": ([31] * 30 + [97] * 9, [3, 5, 8, 1] * 106 + [1], 3),
    "long-runs": ([700, 900, 1, 650], [1100, 900, 251], 1),
    "large-clusters": ([700, 900, 651], [1100, 900, 251], 1),
    "large-clusters-short-runs": ([700, 900, 651], [7, 20, 1, 40] * 33 + [7], 2),
    "few-keys": ([130, 5, 70], [1, 0, 3, 201], 3),
}


@pytest.mark.parametrize("name", list(CASES))
@pytest.mark.parametrize("ear", [False, True])
def test_attention_tile_edges(name, ear):
    from svoo_b200 import ops
    dev = torch.device("cuda")
    qsz, ksz, nth = CASES[name]
    H, S = 3, sum(qsz)
    assert sum(ksz) == S, (sum(qsz), sum(ksz))
    gen = torch.Generator().manual_seed(11)
    qs = torch.stack([torch.tensor(qsz)[torch.randperm(len(qsz), generator=gen)] for _ in range(H)])
    ks = torch.stack([torch.tensor(ksz)[torch.randperm(len(ksz), generator=gen)] for _ in range(H)])
    q, k, v = ((3.0 if i < 2 else 1.0) * torch.randn(H, S, 128, generator=gen) for i in range(3))
    q, k, v = (t.to(dev, torch.bfloat16) for t in (q, k, v))
    QC, KC = len(qsz), len(ksz)
    sel = (torch.arange(KC)[None, None] + torch.arange(QC)[None, :, None] + torch.arange(H)[:, None, None]) % nth == 0
    if not ear and QC > 3:
        sel[0, 3] = False                                          # a query cluster without keys: zero rows
    m = sel.to(torch.uint8).to(dev)
    q_off, k_off = _offsets(qs, dev), _offsets(ks, dev)
    perm = torch.stack([torch.randperm(S, generator=gen) for _ in range(H)]).to(dev, torch.int32)
    scale = 128 ** -0.5
    if not ear:
        got = ops.sparse_attn(q, k, v, m, q_off, k_off, out_row_idx=perm)
        assert ops.attention_status(dev, H, S, QC, KC) == 0
        want = _reference(q, k, v, sel, qs, ks, scale)
        vmax = v.float().abs().max()
    else:
        # centroid j of a pruned cluster is a virtual key with bias log(size + 1e-6)
        kc, vc = (torch.randn(H, KC, 128, generator=gen).to(dev, torch.bfloat16) for _ in range(2))
        k_ext = torch.cat([k.reshape(-1, 128), kc.reshape(-1, 128)])
        v_ext = torch.cat([v.reshape(-1, 128), vc.reshape(-1, 128)])
        got = ops.sparse_attn_ear(q, k_ext, v_ext, m, q_off, k_off, out_row_idx=perm)
        assert ops.ear_attention_status(dev, H, S, QC, KC) == 0
        want = torch.zeros(H, S, 128, device=dev)
        for h in range(H):
            rows = torch.repeat_interleave(torch.arange(QC), qs[h])
            cols = torch.repeat_interleave(torch.arange(KC), ks[h])
            tok = sel[h][rows][:, cols].to(dev)
            s = (q[h].float() @ k[h].float().T * scale).masked_fill(~tok, float("-inf"))
            c = q[h].float() @ kc[h].float().T * scale + torch.log(ks[h].float() + 1e-6).to(dev)
            c = c.masked_fill(sel[h][rows].to(dev), float("-inf"))
            p = torch.softmax(torch.cat([s, c], 1), -1)
            want[h] = p @ torch.cat([v[h], vc[h]]).float()
        vmax = max(v.float().abs().max(), vc.float().abs().max())
    idx = perm.long()[..., None].expand(-1, -1, 128)
    err = (torch.gather(got.float(), 1, idx) - want).abs().max()
    assert err <= 2.5 * 2.0 ** -9 * vmax, float(err)
    again = ops.sparse_attn(q, k, v, m, q_off, k_off, out_row_idx=perm) if not ear else \
        ops.sparse_attn_ear(q, k_ext, v_ext, m, q_off, k_off, out_row_idx=perm)
    assert torch.equal(again, got)


@pytest.mark.parametrize("rows", [1, 64, 65, 128])
def test_query_clusters_without_keys(rows):
    """Most query clusters have no keys: their CTAs end at once and others start in their place.  Zero rows for them,
    the others undisturbed."""
    from svoo_b200 import ops
    dev = torch.device("cuda")
    H, QC, KC = 8, 160, 24
    gen = torch.Generator().manual_seed(rows)
    S = rows * QC
    qs = torch.full((H, QC), rows)
    ks = torch.full((H, KC), S // KC)
    ks[:, -1] += S - ks[0].sum()
    q, k, v = (torch.randn(H, S, 128, generator=gen).to(dev, torch.bfloat16) for _ in range(3))
    sel = torch.zeros(H, QC, KC, dtype=torch.bool)
    sel[:, ::5, 3] = True
    sel[:, 2::5, ::7] = True
    q_off, k_off = _offsets(qs, dev), _offsets(ks, dev)
    got = ops.sparse_attn(q, k, v, sel.to(torch.uint8).to(dev), q_off, k_off)
    assert ops.attention_status(dev, H, S, QC, KC) == 0
    dead = torch.repeat_interleave(~sel.any(-1), rows, dim=1).to(dev)
    assert (got[dead] == 0).all()
    want = _reference(q[:1], k[:1], v[:1], sel[:1], qs[:1], ks[:1], 128 ** -0.5)
    assert (got[:1].float() - want).abs().max() <= 2.5 * 2.0 ** -9 * v.float().abs().max()


@pytest.mark.parametrize("KC", [5, 33, 97, 1025])
def test_map_at_any_address(KC):
    """A map that starts and ends inside a 32-bit word gives the rows of an aligned one."""
    from svoo_b200 import ops
    dev = torch.device("cuda")
    H, QC, S = 3, 3, 2053
    gen = torch.Generator().manual_seed(KC)
    qs, ks = (torch.full((H, c), S // c) for c in (QC, KC))
    qs[:, 0] += S - qs[0].sum()
    ks[:, 0] += S - ks[0].sum()
    q, k, v = (torch.randn(H, S, 128, generator=gen).to(dev, torch.bfloat16) for _ in range(3))
    m = (torch.rand(H, QC, KC, generator=gen) < 0.5).to(torch.uint8).to(dev)
    want = ops.sparse_attn(q, k, v, m, _offsets(qs, dev), _offsets(ks, dev))
    for shift in (1, 2, 3):
        buf = torch.ones(m.numel() + 8, dtype=torch.uint8, device=dev)
        view = buf[shift:shift + m.numel()].view(H, QC, KC)
        view.copy_(m)
        assert torch.equal(ops.sparse_attn(q, k, v, view, _offsets(qs, dev), _offsets(ks, dev)), want)


@pytest.mark.parametrize("name", ["short", "long", "rising"] + list(CASES))
@pytest.mark.parametrize("ear", [False, True])
def test_single_tiles_are_the_same_in_either_kernel(name, ear):
    """Empty query clusters more and the single tiles go to their own kernel instead of the pair kernel: the same
    bits, output and log-sum-exp.  `rising`: row maxima that grow along the keys, so that O is rescaled, first in one
    half of a 128-key tile and then in the other."""
    from svoo_b200 import ops
    dev = torch.device("cuda")
    if name in CASES:
        qsz, ksz, _ = CASES[name]
    else:
        qsz = [100, 28, 64, 65, 1, 3712]                          # the last one leaves a remainder of 128 rows
        ksz = [3, 40, 1, 96, 5, 7] * 26 + [18] if name == "short" else [400, 1, 63, 64, 2, 130, 900, 2410]
    H, S, QC, KC = 2, sum(qsz), len(qsz), len(ksz)
    more = 40                                                     # split below 100 (error-aware) / 150 rows per query cluster
    assert sum(ksz) == S < 100 * (QC + more) and (name in CASES or S >= 150 * QC)
    gen = torch.Generator().manual_seed(KC)
    q, k, v = (torch.randn(H, S, 128, generator=gen) for _ in range(3))
    if name == "rising":
        k = k * torch.linspace(0.2, 6.0, S)[None, :, None]
    q, k, v = (t.to(dev, torch.bfloat16) for t in (q, k, v))
    kc, vc = (torch.randn(H * KC, 128, generator=gen).to(dev, torch.bfloat16) for _ in range(2))
    sel = (torch.rand(H, QC + more, KC, generator=gen) < 0.6).to(torch.uint8)
    sel[..., 0] = 1
    k_off = _offsets(torch.tensor([ksz] * H), dev)
    got = []
    for extra in (0, more):
        q_off = _offsets(torch.tensor([qsz + [0] * extra] * H), dev)
        m = sel[:, :QC + extra].contiguous().to(dev)
        if ear:
            got.append(ops.sparse_attn_ear(q, torch.cat([k.view(-1, 128), kc]), torch.cat([v.view(-1, 128), vc]), m, q_off,
                                           k_off, return_lse=True))
        else:
            got.append(ops.sparse_attn(q, k, v, m, q_off, k_off, return_lse=True))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])


def test_status_word_is_the_tensor_core_kernels_own():
    """The status word tells of the last tcgen05 call that used the workspace: that call clears it, the mma.sync
    cross-check leaves it alone."""
    import ctypes
    from svoo_b200 import ops
    from svoo_b200._lib import LIB
    dev = torch.device("cuda")
    H, S, QC, KC = 2, 300, 3, 4
    q, k, v = (torch.randn(H, S, 128, device=dev).to(torch.bfloat16) for _ in range(3))
    args = (torch.ones(H, QC, KC, dtype=torch.uint8, device=dev), _offsets(torch.tensor([[100] * QC] * H), dev),
            _offsets(torch.tensor([[75] * KC] * H), dev))
    off = ctypes.c_int64(0)
    assert LIB.svoo_b200_status_offset(H, S, QC, KC, ctypes.byref(off)) == 0
    ops.workspace(dev, H, S, QC, KC)[off.value:off.value + 4].view(torch.int32).fill_(1)       # as a kernel that gave up
    ops.sparse_attn(q, k, v, *args, kernel="simt")
    assert ops.attention_status(dev, H, S, QC, KC) == 1
    ops.sparse_attn(q, k, v, *args)
    assert ops.attention_status(dev, H, S, QC, KC) == 0
