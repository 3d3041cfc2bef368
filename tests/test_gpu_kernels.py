"""GPU numerics: every hand-written sm_100a kernel against a plain fp32 PyTorch reference."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from dcp_b200.ops import attention as A
from dcp_b200.ops import block_ops, model_ops


@pytest.fixture(scope="module")
def dev():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from dcp_b200.ops import _lib
    assert _lib.available(), "dcp_b200/_kernels.so must be built (python -m dcp_b200.csrc.build)"
    return torch.device("cuda", 0)


def _ranges(kind, nq, off=0):
    r = np.zeros((nq, 4), np.int32)
    i = np.arange(nq)
    if kind == "full":
        r[:, 1] = off
    elif kind == "causal":
        r[:, 1] = i + 1 + off
    elif kind == "two":   # sink + sliding window with a hole between them
        r[:, 1] = 40
        r[:, 2] = np.maximum(40, i + off - 120)
        r[:, 3] = i + 1 + off
    return r


CASES = [
    # nq, kv blocks (tokens per block), block size, hq, hkv, mask kind, key offset
    (128, [128], 128, 1, 1, "full", 128),
    (256, [256, 256, 256], 256, 4, 2, "causal", 512),
    (200, [256, 256, 180], 256, 4, 2, "two", 400),
    (1000, [1024, 1024], 1024, 8, 2, "causal", 1024),
    (77, [512], 512, 2, 1, "two", 300),
]


@pytest.mark.parametrize("case", CASES)
@pytest.mark.parametrize("variant", [0, 1, 2])   # one tile per CTA with P in TMEM / in smem; two tiles per CTA
def test_attention_forward(dev, case, variant):
    nq, kv_blocks, bs, hq, hkv, kind, off = case
    torch.manual_seed(0)
    nkv = len(kv_blocks) * bs
    q = torch.randn(nq + 128, hq, 128, device=dev).bfloat16()
    kv = torch.randn(nkv + 128, 2, hkv, 128, device=dev).bfloat16()
    out = torch.zeros_like(q)
    lse = torch.zeros(hq, nq + 128, device=dev)
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    rng = _ranges(kind, nq, off)
    row = A.AttnRow(0, nq, list(range(hq)), [(i * bs, n) for i, n in enumerate(kv_blocks)], rng)
    tabs = A.build_fwd_tables([row], bs, dev, tile_m=256 if variant == 2 else 128)
    A.attn_fwd(q, kv, tabs, [out], [lse], 128 ** -0.5, status, variant)
    torch.cuda.synchronize()
    assert status.item() == 0
    valid = torch.zeros(nkv, dtype=torch.bool)
    for i, n in enumerate(kv_blocks):
        valid[i * bs:i * bs + n] = True
    mask = A.ranges_to_dense(rng, nkv) & valid[None]
    ro, rl = A.attention_reference(q[:nq], kv[:nkv, 0], kv[:nkv, 1], mask, 128 ** -0.5)
    fin = torch.isfinite(rl)
    assert (out[:nq].float() - ro).abs().max() < 2e-2
    assert (lse[:, :nq][fin] - rl[fin]).abs().max() < 1e-3
    assert torch.isinf(lse[:, :nq][~fin]).all()


@pytest.mark.parametrize("case", CASES)
def test_attention_backward(dev, case):
    nq, kv_blocks, bs, hq, hkv, kind, off = case
    torch.manual_seed(1)
    nkv = len(kv_blocks) * bs
    q = torch.randn(nq + 128, hq, 128, device=dev).bfloat16()
    kv = torch.randn(nkv + 128, 2, hkv, 128, device=dev).bfloat16()
    dout = torch.randn(nq + 128, hq, 128, device=dev).bfloat16()
    out = torch.zeros_like(q)
    lse = torch.zeros(hq, nq + 128, device=dev)
    delta = torch.zeros_like(lse)
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    rng = _ranges(kind, nq, off)
    row = A.AttnRow(0, nq, list(range(hq)), [(i * bs, n) for i, n in enumerate(kv_blocks)], rng)
    scale = 128 ** -0.5
    A.attn_fwd(q, kv, A.build_fwd_tables([row], bs, dev), [out], [lse], scale, status, 0)
    A.attn_delta(out, dout, delta, 0, nq)
    bt = A.build_bwd_tables([row], bs, hq, hkv, dev)
    dq = torch.zeros(nq + 128, hq, 128, device=dev)
    dkv = torch.zeros(nkv + 128, 2, hkv, 128, device=dev)
    A.attn_bwd(q, dout, kv, lse, delta, bt, [dq], [dkv], scale, status)
    torch.cuda.synchronize()
    assert status.item() == 0
    valid = torch.zeros(nkv, dtype=torch.bool)
    for i, n in enumerate(kv_blocks):
        valid[i * bs:i * bs + n] = True
    mask = A.ranges_to_dense(rng, nkv) & valid[None]
    _, _, rdq, rdk, rdv = A.attention_reference_bwd(q[:nq], kv[:nkv, 0], kv[:nkv, 1], mask, scale, dout[:nq])
    rel = lambda a, b: ((a - b).abs().max() / (b.abs().max() + 1e-9)).item()
    assert rel(dq[:nq], rdq) < 2e-2 and rel(dkv[:nkv, 0], rdk) < 2e-2 and rel(dkv[:nkv, 1], rdv) < 2e-2
    assert dq[nq:].abs().max() == 0 and dkv[nkv:].abs().max() == 0     # nothing written past the valid rows


@pytest.mark.parametrize("nq,nkv,kind", [(1, 1, "full"), (130, 129, "window"), (256, 384, "window"), (300, 700, "climb")])
def test_attention_forward_masks_and_rescale(dev, nq, nkv, kind):
    """Mask words at the edges of 32 keys and of a tile, and a running maximum that moves in later tiles, fp64
    oracle.  P and V are bf16 (2^-9 of the largest value each, and P is cut, not rounded: 2^-8), the result is rounded
    to bf16 once more: 2^-6 of the largest value; the row sum is fp32 and unbiased to 1e-3 in the LSE."""
    g = torch.Generator().manual_seed(nq + nkv)
    q, kv = (torch.randn(n + 17, *s, generator=g).bfloat16().to(dev) for n, s in ((nq, (4, 128)), (nkv, (2, 2, 128))))
    i = np.arange(nq)
    rng = np.zeros((nq, 4), np.int32)
    rng[:, 1] = nkv
    if kind == "window":       # windows that start and end at every offset inside a word, disjoint, some rows empty
        rng[:, 1] = np.minimum(i % 67, nkv)
        rng[:, 2] = np.clip(i % 67 + i % 35, 0, nkv)
        rng[:, 3] = np.clip(i % 67 + i % 35 + i % 131, 0, nkv)
    if kind == "climb":        # later key tiles score far higher: O is rescaled
        q[:, :, 0] = 4.0
        kv[:nkv, 0, :, 0] = (torch.arange(nkv, device=dev) // 128 * 16.0)[:, None].bfloat16()
    row = A.AttnRow(0, nq, [0, 1, 2, 3], [(0, nkv)], rng)
    out, lse = torch.zeros_like(q), torch.zeros(4, nq + 17, device=dev)
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    A.attn_fwd(q, kv, A.build_fwd_tables([row], 1024, dev), [out], [lse], 128 ** -0.5, status)
    assert status.item() == 0
    k64, v64 = (kv[:nkv, j].double().repeat_interleave(2, 1).permute(1, 0, 2) for j in (0, 1))
    s = (q[:nq].double().permute(1, 0, 2) @ k64.transpose(1, 2) * 128 ** -0.5).masked_fill(~A.ranges_to_dense(rng, nkv).to(dev), float("-inf"))
    ref, rl = (s.softmax(-1).nan_to_num(0.0) @ v64).permute(1, 0, 2), torch.logsumexp(s, -1)
    empty = torch.isinf(rl)
    assert (out[:nq] - ref).abs().max() <= 2.0 ** -6 * ref.abs().max()
    assert torch.equal(torch.isinf(lse[:, :nq]), empty) and ((lse[:, :nq] - rl)[~empty].abs() < 1e-3).all()
    assert out[nq:].abs().max() == 0


@pytest.mark.parametrize("nkv", [128, 256, 300, 384, 512, 640, 1100])
@pytest.mark.parametrize("kind", ["plain", "late", "jump", "apart", "short", "many"])
def test_attention_forward_pairs_of_tiles(dev, nkv, kind):
    """Two query tiles that share a walk over the keys, every remainder of the three score buffers and two
    warpgroups, fp64 oracle.  late: rows whose first key lies in a later tile than their neighbours'; jump: scores that
    rise by 2^70 and more after the first tile (the second pass); apart: key tiles that only one of the query tiles
    sees, with values that are not finite where the other one does not look; short: the second query tile is empty; many:
    more tiles than pairs of CTAs, some of them with a second pass, some without any key.
    Bound as above: P and V are bf16, P is cut, the result is rounded once more, 2^-6 of the largest value."""
    nq, hq = {"short": (100, 4), "many": (2300, 16)}.get(kind, (256, 4))
    g = torch.Generator().manual_seed(nkv)
    q, kv = (torch.randn(n + 29, *s, generator=g).bfloat16().to(dev) for n, s in ((nq, (hq, 128)), (nkv, (2, 2, 128))))
    i = np.arange(nq)
    rng = np.zeros((nq, 4), np.int32)
    rng[:, 1] = nkv
    if kind == "late":
        rng[:, 0] = np.minimum(i * 5 % 700, nkv)          # the last ones see nothing at all
    if kind == "many":
        rng[512:800, 1] = 0
        q[1000:1300, 1, 0] = 16.0
    if kind in ("jump", "many"):
        q[:, 0, 0] = 16.0                                 # one head
        kv[128:nkv, 0, 0, 0] = (40.0 * (1 + torch.arange(nkv - 128, device=dev) // 128))[:].bfloat16()
    if kind == "apart":
        half = nkv // 256 * 128
        rng[:128, 1], rng[128:, 0] = half, half
        if half:
            kv[half:nkv, 1, 0, 5] = float("inf")          # first value head: only the second query tile sees these keys
            kv[:half, 1, 1, 7] = float("nan")             # second value head: only the first one does
    row = A.AttnRow(0, nq, list(range(hq)), [(0, nkv)], rng)
    out, lse = torch.zeros_like(q), torch.zeros(hq, nq + 29, device=dev)
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    A.attn_fwd(q, kv, A.build_fwd_tables([row], 2048, dev), [out], [lse], 128 ** -0.5, status)
    assert status.item() == 0
    k64, v64 = (kv[:nkv, j].double().repeat_interleave(hq // 2, 1).permute(1, 0, 2) for j in (0, 1))
    sees = A.ranges_to_dense(rng, nkv).to(dev)
    s = (q[:nq].double().permute(1, 0, 2) @ k64.transpose(1, 2) * 128 ** -0.5).masked_fill(~sees, float("-inf"))
    p, rl = s.softmax(-1).nan_to_num(0.0), torch.logsumexp(s, -1)
    got = out[:nq].double()
    if kind == "apart":
        fine = torch.ones(nq, 4, dtype=torch.bool, device=dev)
        if nkv >= 256:
            fine[128:, :2], fine[:128, 2:] = False, False
        assert torch.isfinite(got[fine]).all()
        v64, got = v64.nan_to_num(0.0, 0.0, 0.0), torch.where(fine[..., None], got, torch.zeros_like(got))
        ref = torch.where(fine[..., None], (p @ v64).permute(1, 0, 2), torch.zeros_like(got))
    else:
        ref = (p @ v64).permute(1, 0, 2)
    empty = torch.isinf(rl)
    assert (got - ref).abs().max() <= 2.0 ** -6 * ref.abs().max()
    assert torch.equal(torch.isinf(lse[:, :nq]), empty)
    assert ((lse[:, :nq] - rl)[~empty].abs() < 1e-3 + 2.0 ** -22 * rl[~empty].abs()).all()
    assert out[nq:].abs().max() == 0


@pytest.mark.parametrize("d", [64, 96, 128])
@pytest.mark.parametrize("rise,values", [(54, 0), (54, 90), (80, 0), (80, 90)])
def test_attention_forward_rising_scores_and_large_values(dev, d, rise, values):
    """Scores that rise by 2^rise behind the first key tile, with values of 2^values: the row sum, or only O, leaves what the first
    pass over a tile holds, and the result is representable all the same.  Bound as above, 2^-6 of the largest value."""
    nq, nkv, hq = 300, 384, 4
    g = torch.Generator().manual_seed(rise + values)
    q, kv = torch.zeros(nq, hq, 128), torch.zeros(nkv, 2, 2, 128)
    q[..., :d], kv[..., :d] = torch.randn(nq, hq, d, generator=g), torch.randn(nkv, 2, 2, d, generator=g)
    kv[:, 1] *= 2.0 ** values
    scale = d ** -0.5
    q[:, :2, 0] = 16.0                                                                     # the first KV head's queries
    kv[:, 0, 0, 0] = (torch.arange(nkv) >= 128) * (rise / (16.0 * scale * np.log2(np.e)))
    q, kv = q.bfloat16().to(dev), kv.bfloat16().to(dev)
    rng = np.zeros((nq, 4), np.int32)
    rng[:, 1] = nkv
    rng[7:11, 1] = 100                                                                     # rows that stay in the first key tile
    out, lse = torch.zeros_like(q), torch.zeros(hq, nq, device=dev)
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    A.attn_fwd(q, kv, A.build_fwd_tables([A.AttnRow(0, nq, list(range(hq)), [(0, nkv)], rng)], 512, dev), [out], [lse], scale, status, channels=d)
    assert status.item() == 0
    k64, v64 = (kv[:, j].double().repeat_interleave(2, 1).permute(1, 0, 2) for j in (0, 1))
    s = (q.double().permute(1, 0, 2) @ k64.transpose(1, 2) * scale).masked_fill(~A.ranges_to_dense(rng, nkv).to(dev), float("-inf"))
    ref, rl = (s.softmax(-1) @ v64).permute(1, 0, 2), torch.logsumexp(s, -1)
    assert ((out.double() - ref).abs() <= 2.0 ** -6 * ref.abs().max()).all()
    assert ((lse - rl).abs() < 1e-3 + 2.0 ** -22 * rl.abs()).all()


@pytest.mark.parametrize("nq,nkv", [(1, 1), (257, 300)])
def test_attention_forward_result_at_16_bytes(dev, nq, nkv):
    """A result whose rows begin 16 bytes off a sector: the same bits as at the start of one."""
    torch.manual_seed(0)
    q, kv = torch.randn(nq, 4, 128, device=dev).bfloat16(), torch.randn(nkv, 2, 2, 128, device=dev).bfloat16()
    rng = np.zeros((nq, 4), np.int32)
    rng[:, 1] = nkv
    tables = A.build_fwd_tables([A.AttnRow(0, nq, list(range(4)), [(0, nkv)], rng)], 512, dev)
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    flat = torch.zeros(2, q.numel() + 16, device=dev, dtype=torch.bfloat16)
    for buf, off in zip(flat, (0, 8)):
        A.attn_fwd(q, kv, tables, [buf[off:off + q.numel()].view_as(q)], [torch.zeros(4, nq, device=dev)], 128 ** -0.5, status)
    assert status.item() == 0 and flat[0, :q.numel()].abs().max() > 0
    assert torch.equal(flat[0, :q.numel()], flat[1, 8:8 + q.numel()]) and not flat[1, :8].any() and not flat[1, 8 + q.numel():].any()


@pytest.mark.parametrize("seeing", [0, 1, 700])
def test_attention_forward_many_tiles_without_keys(dev, seeing):
    """More tiles without any key per pair of CTAs than it holds records of, behind a tile that has some: zeros and -inf
    there, and the others as above (2^-6 of the largest value)."""
    nq, nkv, hq = 6400, 300, 16
    torch.manual_seed(seeing)
    q, kv = torch.randn(nq, hq, 128, device=dev).bfloat16(), torch.randn(nkv, 2, 4, 128, device=dev).bfloat16()
    rng = np.zeros((nq, 4), np.int32)
    rng[:seeing, 1] = nkv
    row = A.AttnRow(0, nq, list(range(hq)), [(0, nkv)], rng)
    out, lse = torch.full_like(q, 7), torch.zeros(hq, nq, device=dev)
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    A.attn_fwd(q, kv, A.build_fwd_tables([row], 2048, dev), [out], [lse], 128 ** -0.5, status)
    assert status.item() == 0
    assert out[seeing:].abs().max() == 0 and torch.isinf(lse[:, seeing:]).all()
    if seeing:
        k64, v64 = (kv[:, j].double().repeat_interleave(hq // 4, 1).permute(1, 0, 2) for j in (0, 1))
        s = q[:seeing].double().permute(1, 0, 2) @ k64.transpose(1, 2) * 128 ** -0.5
        ref = (s.softmax(-1) @ v64).permute(1, 0, 2)
        assert (out[:seeing].double() - ref).abs().max() <= 2.0 ** -6 * ref.abs().max()
        assert (lse[:, :seeing] - torch.logsumexp(s, -1)).abs().max() < 1e-3


@pytest.mark.parametrize("nq,nkv,kind,heads", [(1, 1, "causal", (4, 4)), (127, 129, "full", (4, 1)), (129, 127, "causal", (8, 2)),
                                                (256, 255, "two", (4, 2)), (64, 640, "full", (8, 1)), (700, 700, "two", (8, 2))])
def test_attention_backward_tile_edges(dev, nq, nkv, kind, heads):
    """Edges of the 128 x 128 items, items without and with masking, whole and split head groups, fp64 oracle.
    P, dS and the operands are bf16: 2^-8 relative each, four of them in a chain, so 2 % of the largest element."""
    hq, hkv = heads
    g = torch.Generator().manual_seed(nq * 1000 + nkv)
    new = lambda *shape: torch.randn(*shape, generator=g).bfloat16().to(dev)
    q, kv, dout = new(nq + 40, hq, 128), new(nkv + 40, 2, hkv, 128), new(nq + 40, hq, 128)
    i = np.arange(nq)
    rng = np.zeros((nq, 4), np.int32)
    off = max(nkv - nq, 0)
    if kind == "full":
        rng[:, 1] = nkv
    elif kind == "causal":
        rng[:, 1] = np.minimum(i + 1 + off, nkv)
    else:      # a sink and a window that ends mid-tile, some queries without any key
        rng[:, 1] = np.minimum(37, nkv)
        rng[:, 2] = np.clip(i - 70, 37, nkv)
        rng[:, 3] = np.clip(i + 5, 37, nkv)
        rng[i % 61 == 60] = 0
    row = A.AttnRow(0, nq, list(range(hq)), [(0, nkv)], rng)
    scale = 128 ** -0.5
    mask = A.ranges_to_dense(rng, nkv).to(dev)
    k64, v64 = (kv[:nkv, j].double().repeat_interleave(hq // hkv, 1).permute(1, 0, 2) for j in (0, 1))
    q64, do64 = q[:nq].double().permute(1, 0, 2), dout[:nq].double().permute(1, 0, 2)
    s = (q64 @ k64.transpose(1, 2) * scale).masked_fill(~mask, float("-inf"))
    p = s.softmax(-1).nan_to_num(0.0)
    out64 = p @ v64
    lse = torch.full((hq, nq + 40), 7.0, device=dev)
    lse[:, :nq] = torch.logsumexp(s, -1).float()
    delta = torch.full_like(lse, 7.0)
    delta[:, :nq] = (out64 * do64).sum(-1).float()
    ds = p * (do64 @ v64.transpose(1, 2) - (out64 * do64).sum(-1, keepdim=True)) * scale
    fold = lambda t: t.reshape(hkv, hq // hkv, nkv, 128).sum(1).permute(1, 0, 2)
    want = ((ds @ k64).permute(1, 0, 2), fold(ds.transpose(1, 2) @ q64), fold(p.transpose(1, 2) @ do64))
    tables = A.build_bwd_tables([row], 1024, hq, hkv, dev)
    assert tables.max_items > 0
    for max_items in (tables.max_items, 0):      # 0: head groups stay whole
        tables.max_items = max_items
        dq, dkv = torch.zeros(nq + 40, hq, 128, device=dev), torch.zeros(nkv + 40, 2, hkv, 128, device=dev)
        status = torch.zeros(1, dtype=torch.int32, device=dev)
        A.attn_bwd(q, dout, kv, lse, delta, tables, [dq], [dkv], scale, status)
        assert status.item() == 0
        for got, ref in zip((dq[:nq], dkv[:nkv, 0], dkv[:nkv, 1]), want):
            assert (got - ref).abs().max() <= 2e-2 * ref.abs().max() + 1e-6
        assert dq[nq:].abs().max() == 0 and dkv[nkv:].abs().max() == 0


@pytest.mark.parametrize("hq,hkv,parts", [(8, 2, 1), (8, 2, 2), (8, 2, 4), (16, 2, 4), (6, 2, 3), (12, 2, 2), (4, 1, 4), (16, 1, 8), (12, 1, 6)])
def test_attention_backward_split_head_groups(dev, hq, hkv, parts):
    """A head group over 1, some or all of its possible CTAs (at most 8), partial key and query tiles, fp64 oracle with the
    bound of ``test_attention_backward_tile_edges``; dK and dV are the same bits in every run."""
    n = 1500
    g = torch.Generator().manual_seed(hq * 10 + parts)
    new = lambda *shape: torch.randn(*shape, generator=g).bfloat16().to(dev)
    q, kv, dout = new(n, hq, 128), new(n, 2, hkv, 128), new(n, hq, 128)
    rng = np.zeros((n, 4), np.int32)
    rng[:, 1] = np.arange(n) + 1
    row = A.AttnRow(0, n, list(range(hq)), [(0, n)], rng)
    scale = 128 ** -0.5
    heads = lambda t: t.double().repeat_interleave(hq // t.shape[1], 1).permute(1, 0, 2)
    q64, k64, v64, do64 = heads(q), heads(kv[:, 0]), heads(kv[:, 1]), heads(dout)
    s = (q64 @ k64.transpose(1, 2) * scale).masked_fill(~A.ranges_to_dense(rng, n).to(dev), float("-inf"))
    p = s.softmax(-1)
    d64 = (p @ v64 * do64).sum(-1)
    ds = p * (do64 @ v64.transpose(1, 2) - d64[..., None]) * scale
    fold = lambda t: t.reshape(hkv, hq // hkv, n, 128).sum(1).permute(1, 0, 2)
    want = ((ds @ k64).permute(1, 0, 2), fold(ds.transpose(1, 2) @ q64), fold(p.transpose(1, 2) @ do64))
    lse, delta = torch.logsumexp(s, -1).float(), d64.float()
    tables = A.build_bwd_tables([row], 1024, hq, hkv, dev)
    # the group is split until the longest list x (heads of a CTA) x 148 SMs is within all visits
    tables.max_items = tables.n_items * hkv * parts // 148 if parts > 1 else 0
    first = None
    for _ in range(10):
        dq, dkv = torch.zeros(n, hq, 128, device=dev), torch.zeros(n, 2, hkv, 128, device=dev)
        status = torch.zeros(1, dtype=torch.int32, device=dev)
        A.attn_bwd(q, dout, kv, lse, delta, tables, [dq], [dkv], scale, status)
        assert status.item() == 0
        first = dkv if first is None else first
        assert torch.equal(dkv, first)
    for got, ref in zip((dq, dkv[:, 0], dkv[:, 1]), want):
        assert (got - ref).abs().max() <= 2e-2 * ref.abs().max()


def test_attention_backward_split_group_carries_copy_jobs(dev):
    """Head groups over several CTAs (clusters) in a launch whose first CTAs only copy rows and statistics from a peer's
    region (here a local one): the copies arrive, dK and dV are those of a launch without them."""
    from dcp_b200.planner.lowering import row_copy_jobs, stat_copy_jobs
    n, hq, hkv = 700, 8, 2
    g = torch.Generator().manual_seed(2)
    new = lambda *shape: torch.randn(*shape, generator=g).bfloat16().to(dev)
    q, kv, dout = new(n, hq, 128), new(n, 2, hkv, 128), new(n, hq, 128)
    rng = np.zeros((n, 4), np.int32)
    rng[:, 1] = np.arange(n) + 1
    row = A.AttnRow(0, n, list(range(hq)), [(0, n)], rng)
    out, lse = torch.zeros_like(q), torch.zeros(hq, n, device=dev)
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    A.attn_fwd(q, kv, A.build_fwd_tables([row], 1024, dev), [out], [lse], 128 ** -0.5, status)
    delta = torch.zeros_like(lse)
    A.attn_delta(out, dout, delta, 0, n)
    regions = {"q": q, "kv": kv, "dout": dout, "lse": lse, "delta": delta}
    staged = {k: torch.zeros_like(t) for k, t in regions.items()}
    ctx = A.CopyContext(lambda name: [regions[name].data_ptr(), staged[name].data_ptr()], 1, n)
    pulls = np.array([[0, 3, 10, 600]], np.int32)
    jobs = np.concatenate([row_copy_jobs(pulls, 0, hq * 16), row_copy_jobs(pulls, 1, 2 * hkv * 16), stat_copy_jobs(pulls, 3, hq)])
    tables = A.build_bwd_tables([row], 1024, hq, hkv, dev)
    runs = []
    for j in (None, torch.from_numpy(jobs).to(dev)):
        dq, dkv = torch.zeros(n, hq, 128, device=dev), torch.zeros(n, 2, hkv, 128, device=dev)
        A.attn_bwd(q, dout, kv, lse, delta, tables, [dq], [dkv], 128 ** -0.5, status, jobs=j, job_ctx=ctx)
        runs.append(dkv)
    assert status.item() == 0 and torch.equal(*runs)
    for name in ("q", "kv"):
        assert torch.equal(staged[name][10:610], regions[name][3:603]) and not staged[name][:10].any() and not staged[name][610:].any()
    assert torch.equal(staged["lse"][:, 10:610], lse[:, 3:603]) and not staged["delta"].any() and not staged["lse"][:, 610:].any()


def test_attention_backward_into_a_second_accumulator(dev):
    """Items that name another accumulator than the first (a peer's, here a second local one) add the rows the first
    would have got, and nothing beside them; items that want no dQ add none.  dQ is a sum of fp32 in changing order:
    1e-5 of the largest element."""
    n, hq, hkv = 700, 4, 2
    g = torch.Generator().manual_seed(1)
    new = lambda *shape: torch.randn(*shape, generator=g).bfloat16().to(dev)
    q, kv, dout = new(n, hq, 128), new(n, 2, hkv, 128), new(n, hq, 128)
    rng = np.zeros((n, 4), np.int32)
    rng[:, 1] = np.arange(n) + 1
    row = A.AttnRow(0, n, list(range(hq)), [(0, n)], rng)
    out, lse = torch.zeros_like(q), torch.zeros(hq, n, device=dev)
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    A.attn_fwd(q, kv, A.build_fwd_tables([row], 1024, dev), [out], [lse], 128 ** -0.5, status)
    delta = torch.zeros_like(lse)
    A.attn_delta(out, dout, delta, 0, n)
    runs = []
    for split in (False, True):
        tables = A.build_bwd_tables([row], 1024, hq, hkv, dev)
        tile = tables.items[:, 0] // 128           # query tile: 1 and 4 to the second accumulator, 2 to none
        if split:
            tables.items[:, 4] = ((tile == 1) | (tile >= 4)).int() - (tile == 2).int()
        dq = [torch.zeros(n, hq, 128, device=dev) for _ in range(2)]
        dkv = [torch.zeros(n, 2, hkv, 128, device=dev) for _ in range(2)]
        A.attn_bwd(q, dout, kv, lse, delta, tables, dq, dkv, 128 ** -0.5, status)
        assert status.item() == 0 and dkv[1].abs().max() == 0
        runs.append((dq, dkv[0]))
    (want, _), want_kv = runs[0]
    (first, second), got_kv = runs[1]
    assert torch.equal(got_kv, want_kv)
    tile = torch.arange(n, device=dev) // 128
    other = (tile == 1) | (tile >= 4)
    close = lambda a, b: (a - b).abs().max() <= 1e-5 * want.abs().max()
    assert close(first[(tile == 0) | (tile == 3)], want[(tile == 0) | (tile == 3)]) and close(second[other], want[other])
    assert first[other | (tile == 2)].abs().max() == 0 and second[~other].abs().max() == 0


@pytest.mark.parametrize("d", [64, 96, 128])
@pytest.mark.parametrize("nkv", [128, 256, 301])
def test_attention_backward_whole_and_part_key_tiles(dev, d, nkv):
    """Heads without a group, so that a CTA adds its dK and dV by itself: whole key tiles, and the part of one.  Added to what the
    accumulators hold, nothing beyond the keys or the channels; bound as for the other backward tests (2^-6 of the largest)."""
    nq, h = 200, 4
    torch.manual_seed(nkv)
    q, dout = torch.zeros(2, nq, h, 128, device=dev, dtype=torch.bfloat16)
    kv = torch.zeros(nkv + 40, 2, h, 128, device=dev, dtype=torch.bfloat16)
    for t in (q, dout, kv):
        t[..., :d] = torch.randn(*t.shape[:-1], d, device=dev).bfloat16()
    rng = np.zeros((nq, 4), np.int32)
    rng[:, 1] = np.minimum(np.arange(nq) + nkv - 150, nkv).clip(0)
    row = A.AttnRow(0, nq, list(range(h)), [(0, nkv)], rng)
    out, lse, delta = torch.zeros_like(q), torch.zeros(h, nq, device=dev), torch.zeros(h, nq, device=dev)
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    A.attn_fwd(q, kv, A.build_fwd_tables([row], 512, dev), [out], [lse], d ** -0.5, status, channels=d)
    A.attn_delta(out, dout, delta, 0, nq)
    dq, dkv = torch.zeros(nq, h, 128, device=dev), torch.ones(nkv + 40, 2, h, 128, device=dev)
    A.attn_bwd(q, dout, kv, lse, delta, A.build_bwd_tables([row], 512, h, h, dev), [dq], [dkv], d ** -0.5, status, channels=d)
    assert status.item() == 0
    assert (dkv[nkv:] == 1).all() and (dkv[..., d:] == 1).all()
    q64, o64, k64, v64 = (t.double().permute(1, 0, 2) for t in (q, dout, kv[:nkv, 0], kv[:nkv, 1]))
    s = (q64 @ k64.transpose(1, 2) * d ** -0.5).masked_fill(~A.ranges_to_dense(rng, nkv).to(dev), float("-inf"))
    p = s.softmax(-1).nan_to_num(0.0)
    ds = p * (o64 @ v64.transpose(1, 2) - ((p @ v64) * o64).sum(-1, keepdim=True)) * d ** -0.5
    for got, want in ((dkv[:nkv, 0] - 1, ds.transpose(1, 2) @ q64), (dkv[:nkv, 1] - 1, p.transpose(1, 2) @ o64), (dq, ds @ k64)):
        want = want.permute(1, 0, 2)
        assert (got.double() - want).abs().max() <= 2.0 ** -6 * want.abs().max()


@pytest.mark.parametrize("d", [8, 40, 64, 72, 96, 104])
@pytest.mark.parametrize("nq,nkv,heads", [(130, 300, (4, 2)), (600, 520, (16, 2))])   # head groups whole; split over clusters
def test_attention_over_fewer_channels(dev, d, nq, nkv, heads):
    """Products that leave the zeros of padded heads out, against products over all 128 channels of the same arenas: the
    terms left out are exact zeros, so S, P and the output agree to the bit; the gradients are sums of the same terms
    that the accumulators take in any order (float32, at most 600 of them: 600 x 2^-24 of the largest partial sum)."""
    hq, hkv = heads
    torch.manual_seed(0)
    q = torch.zeros(nq + 128, hq, 128, device=dev, dtype=torch.bfloat16)
    kv = torch.zeros(nkv + 128, 2, hkv, 128, device=dev, dtype=torch.bfloat16)
    dout = torch.zeros_like(q)
    q[:nq, :, :d], kv[:nkv, ..., :d], dout[:nq, :, :d] = (torch.randn(n, *h, d, device=dev).bfloat16() for n, h in
                                                          ((nq, (hq,)), (nkv, (2, hkv)), (nq, (hq,))))
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    rng = np.zeros((nq, 4), dtype=np.int32)
    rng[:, 1] = np.minimum(np.arange(nq) + 33, nkv)
    rng[5:9] = 0
    row = A.AttnRow(0, nq, list(range(hq)), [(0, nkv)], rng)
    ft, bt = A.build_fwd_tables([row], 1024, dev), A.build_bwd_tables([row], 1024, hq, hkv, dev)
    res = []
    for channels in (128, d):
        out, lse, delta = torch.full_like(q, 7), torch.zeros(hq, nq + 128, device=dev), torch.zeros(hq, nq + 128, device=dev)
        A.attn_fwd(q, kv, ft, [out], [lse], d ** -0.5, status, channels=channels)
        out = out[:nq]
        A.attn_delta(out, dout, delta, 0, nq)
        dq, dkv = torch.zeros(nq + 128, hq, 128, device=dev), torch.zeros(nkv + 128, 2, hkv, 128, device=dev)
        A.attn_bwd(q, dout, kv, lse, delta, bt, [dq], [dkv], d ** -0.5, status, channels=channels)
        torch.cuda.synchronize()
        assert status.item() == 0
        res.append((out, lse, dq, dkv))
    (out, lse, dq, dkv), (out_d, lse_d, dq_d, dkv_d) = res
    assert torch.equal(out, out_d) and torch.equal(lse, lse_d) and dq.abs().max() > 0.1 and dkv.abs().max() > 0.1
    assert (dq - dq_d).abs().max() <= 600 * 2.0 ** -24 * dq.abs().max()
    assert (dkv - dkv_d).abs().max() <= 600 * 2.0 ** -24 * dkv.abs().max()


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("d", [8, 96, 128])
def test_row_conversions(dev, dtype, d):
    """Padding and cutting rows of d channels round exactly as a torch conversion does, odd row counts, NaN and
    infinities included, and write nothing next to their rows."""
    g = torch.Generator().manual_seed(d)
    x = [(torch.randn(n, 3, d, generator=g) * 100).to(dtype).to(dev) for n in (1, 37)]
    x[1][5, 1, 0], x[1][6, 0, 1] = float("nan"), float("inf")
    dst = [torch.full((t.shape[0] + 1, 3, 128), 7.0, device=dev, dtype=torch.bfloat16) for t in x]
    A.pad_cast_rows([(t, y[:-1]) for t, y in zip(x, dst)])
    for t, y in zip(x, dst):
        want = torch.nn.functional.pad(t.to(torch.bfloat16), (0, 128 - d))
        assert torch.equal(y[:-1].nan_to_num(3.0), want.nan_to_num(3.0)) and (y[-1] == 7).all()
    for src_dtype in (torch.float32, torch.bfloat16):
        src = [torch.randn(n, 3, 128, generator=g).to(src_dtype).to(dev) for n in (37, 2)]
        src[0][5, 1, 0], src[0][6, 0, 1] = float("nan"), -float("inf")
        out = [torch.full((t.shape[0] + 1, 3, d), 7.0, device=dev, dtype=dtype) for t in src]
        A.cut_cast_rows([(t, y[:-1]) for t, y in zip(src, out)])
        for t, y in zip(src, out):
            assert torch.equal(y[:-1].nan_to_num(3.0), t[..., :d].to(dtype).nan_to_num(3.0)) and (y[-1] == 7).all()


@pytest.mark.parametrize("n,hq", [(1, 1), (33, 3), (257, 8), (2500, 32)])
def test_backward_preparation(dev, n, hq):
    """delta is an fp32 sum of 128 products (2^-24 each step of the tree, 1e-5 of the sum of magnitudes), rows beside the
    range stay, both accumulators are cleared as a whole."""
    o, do = torch.randn(n + 5, hq, 128, device=dev).bfloat16(), torch.randn(n + 5, hq, 128, device=dev).bfloat16()
    delta = torch.full((hq, n + 5), 7.0, device=dev)
    z = [torch.ones(k, 128, device=dev) for k in (n, 3)]
    A.attn_bwd_prep(o, do, delta, n, 2, zero=[t[:-1] for t in z])
    prod = o.double() * do.double()
    want, mag = prod.sum(-1).t()[:, 2:n + 2], prod.abs().sum(-1).t()[:, 2:n + 2]
    assert ((delta[:, 2:n + 2] - want).abs() <= 1e-5 * mag).all()
    assert (delta[:, :2] == 7).all() and (delta[:, n + 2:] == 7).all()
    assert all((t[:-1] == 0).all() and (t[-1] == 1).all() for t in z)


@pytest.mark.parametrize("n,t,h", [(1, 3, 1), (2, 17, 5), (3, 1, 4), (4, 100, 32), (5, 7, 3), (6, 33, 2), (7, 2, 8), (8, 64, 4), (11, 9, 3)])
def test_merge_of_stacked_partials(dev, n, t, h):
    """The stacked merge equals the table-driven one bit for bit: every count of sources with a kernel of its own and
    one without, ragged item counts, invalid (-inf, +inf, NaN) partials, strided and misaligned inputs."""
    g = torch.Generator().manual_seed(n * 100 + t)
    outs = torch.randn(n, t, h, 128, generator=g).bfloat16().to(dev)
    lses = (4 + 2 * torch.randn(n, t, h, generator=g)).to(dev)
    kind = torch.randint(0, 8, (n, t, h), generator=g).to(dev)
    for k, v in ((0, float("-inf")), (1, float("nan")), (2, float("inf"))):
        lses[kind == k] = v
    lses[:, 0, 0] = float("-inf")
    ops = torch.tensor([[0, t, 0, n]], dtype=torch.int32, device=dev)
    src = torch.arange(0, n * t, t, dtype=torch.int32, device=dev)
    want, want_lse = torch.empty(t, h, 128, device=dev, dtype=torch.bfloat16), torch.empty(h, t, device=dev)
    block_ops.merge_out_lse(ops, src, outs.view(n * t, h, 128), lses.permute(2, 0, 1).reshape(h, n * t).contiguous(), want, want_lse)
    shifted = torch.cat([outs.new_zeros(1), outs.flatten()])[1:].view(outs.shape)
    for o, l in ((outs, lses), (outs.transpose(1, 2).contiguous().transpose(1, 2), lses.transpose(1, 2).contiguous().transpose(1, 2)), (shifted, lses)):
        out, lse = block_ops.flash_attn_update_out_lse(o, l)
        assert torch.equal(out, want) and torch.equal(lse, want_lse.t())


@pytest.mark.parametrize("n", [8, 8 * 1023, 8 * 1025, 8 * (148 * 8 * 256 * 4 + 3)])
@pytest.mark.parametrize("scale", [1.0, 0.5])
def test_gradient_norm_and_clip_coefficient(dev, n, scale):
    """fp32 sums of at most a few hundred terms per thread, added in 64 bits: 1e-6 relative; a norm below
    the limit gives exactly 1, a NaN gradient a NaN coefficient."""
    from dcp_b200.parallel.dist_optimizer import FlatBuffers, ShardedAdamW
    bufs = FlatBuffers(n, dev)
    opt = ShardedAdamW(bufs, clip_grad=0.25)
    bufs.grads.normal_()
    norm = float(bufs.grads.double().norm()) * scale
    opt.step(scale)
    assert abs(opt.grad_norm() / norm - 1) < 1e-6 and abs(float(opt.clip_coef) / (0.25 / (norm + 1e-6)) - 1) < 1e-6
    bufs.grads.mul_(0.1 / norm)
    opt.step(scale)
    assert float(opt.clip_coef) == 1.0
    bufs.grads[n // 2] = float("nan")
    opt.step(scale)
    assert bool(torch.isnan(opt.clip_coef))


def test_rmsnorm(dev):
    torch.manual_seed(0)
    for hidden in (1024, 4096):
        x = torch.randn(300, hidden, device=dev).bfloat16().requires_grad_(True)
        w = (1 + 0.1 * torch.randn(hidden, device=dev)).bfloat16().requires_grad_(True)
        dy = torch.randn(300, hidden, device=dev).bfloat16()
        y = model_ops.rmsnorm(x, w, 1e-5)
        y.backward(dy)
        xr, wr = x.detach().float().requires_grad_(True), w.detach().float().requires_grad_(True)
        yr = xr * torch.rsqrt(xr.pow(2).mean(-1, keepdim=True) + 1e-5) * wr
        yr.backward(dy.float())
        assert (y.float() - yr).abs().max() < 3e-2
        assert (x.grad.float() - xr.grad).abs().max() < 5e-2
        assert ((w.grad.float() - wr.grad).abs() / (wr.grad.abs() + 1.0)).max() < 3e-2


def test_swiglu(dev):
    torch.manual_seed(0)
    gu = torch.randn(257, 2 * 1024, device=dev).bfloat16().requires_grad_(True)
    dy = torch.randn(257, 1024, device=dev).bfloat16()
    y = model_ops.swiglu(gu)
    y.backward(dy)
    gr = gu.detach().float().requires_grad_(True)
    g, u = gr.chunk(2, dim=-1)
    yr = torch.nn.functional.silu(g) * u
    yr.backward(dy.float())
    assert ((y.float() - yr).abs() / (yr.abs() + 1.0)).max() < 1e-2
    assert ((gu.grad.float() - gr.grad).abs() / (gr.grad.abs() + 1.0)).max() < 2e-2


@pytest.mark.parametrize("rows", [1, 7, 9, 300, 4000])
@pytest.mark.parametrize("hidden", [1024, 4096])
def test_rmsnorm_backward_with_residual(dev, rows, hidden):
    """One rounding to bf16 of the sum (2^-8 of it) plus 1e-5 for the fp32 row sums; dW is an fp32 sum over the rows
    (1e-5 of the magnitudes), whatever the number of CTAs."""
    g = torch.Generator().manual_seed(rows + hidden)
    x, dy, res = (torch.randn(rows, hidden, generator=g).bfloat16().to(dev) for _ in range(3))
    w = (1 + 0.1 * torch.randn(hidden, generator=g)).bfloat16().to(dev)
    _, rstd = model_ops.rmsnorm_fwd_raw(x, w, 1e-5)
    x64, r64 = x.double(), rstd.double()[:, None]
    gw = dy.double() * w.double()
    base = r64 * (gw - x64 * r64 * (gw * x64 * r64).mean(-1, keepdim=True))
    terms = dy.double() * x64 * r64
    for residual in (None, res):
        dx, dw = model_ops.rmsnorm_bwd_raw(x, w, rstd, dy, residual)
        want = base if residual is None else base + res.double()
        assert ((dx.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5 * (1 + base.abs())).all()
        assert ((dw.double() - terms.sum(0)).abs() <= 1e-5 * (terms.abs().sum(0) + 1)).all()


@pytest.mark.parametrize("how", ["strided", "shifted"])
def test_gradients_of_any_layout(dev, how):
    """The gradient that by-passes a norm and the one that reaches the embedding may be strided or start off a 16-byte
    boundary: the same result bit for bit."""
    change = {"strided": lambda t: torch.stack([t, t * 2], dim=-1)[..., 0],
              "shifted": lambda t: torch.cat([t.new_zeros(1), t.flatten()])[1:].view(t.shape)}[how]
    x, dy, res = (torch.randn(9, 1024, device=dev).bfloat16() for _ in range(3))
    w = torch.ones(1024, device=dev).bfloat16()
    _, rstd = model_ops.rmsnorm_fwd_raw(x, w, 1e-5)
    assert torch.equal(model_ops.rmsnorm_bwd_raw(x, w, rstd, dy, change(res))[0], model_ops.rmsnorm_bwd_raw(x, w, rstd, dy, res)[0])
    ids = torch.tensor([0, 3, 3, 1, 7, 7, 7, 2, 0], device=dev)
    a, b = torch.zeros(8, 1024, device=dev).bfloat16(), torch.zeros(8, 1024, device=dev).bfloat16()
    model_ops.embedding_grad(ids, dy, a)
    model_ops.embedding_grad(ids, change(dy), b)
    assert torch.equal(a, b)


@pytest.mark.parametrize("vocab", [8, 32760, 32768, 40008])
def test_cross_entropy_row_widths(dev, vocab):
    """Both CTA widths, fp64 oracle: the gradient is rounded to bf16 once (2^-8) and the fast exponentials are good to
    1e-5 of a probability; the loss is an fp32 logarithm of an fp32 sum."""
    g = torch.Generator().manual_seed(vocab)
    logits = (3 * torch.randn(5, vocab, generator=g)).bfloat16().to(dev)
    labels = torch.tensor([0, vocab - 1, vocab // 2, -100, 7], device=dev)
    l64 = logits.double()
    want = torch.nn.functional.cross_entropy(l64, labels.clamp(min=0), reduction="none") * (labels >= 0)
    grad = (l64.softmax(-1) - torch.nn.functional.one_hot(labels.clamp(min=0), vocab)) * (labels >= 0)[:, None] * 0.5
    loss = model_ops.cross_entropy_inplace(logits, labels, 0.5)
    assert ((loss - want).abs() < 1e-4).all()
    assert ((logits.double() - grad).abs() <= 2.0 ** -8 * grad.abs() + 1e-5 * l64.softmax(-1) + 1e-7).all()


@pytest.mark.parametrize("n,f", [(1, 8), (3, 2040), (2, 2048), (5, 8200), (300, 1024)])
def test_swiglu_row_lengths(dev, n, f):
    """Row lengths around a multiple of the CTA's stride, fp64 oracle: the result is rounded to bf16 once (2^-8), plus
    1e-5 for the fast exponential."""
    g = torch.Generator().manual_seed(f)
    gu, dy = (4 * torch.randn(n, 2 * f, generator=g)).bfloat16().to(dev), torch.randn(n, f, generator=g).bfloat16().to(dev)
    x = gu.double().requires_grad_(True)
    a, u = x.chunk(2, dim=-1)
    y = torch.nn.functional.silu(a) * u
    y.backward(dy.double())
    for got, want in ((model_ops.swiglu_fwd_raw(gu), y), (model_ops.swiglu_bwd_raw(gu, dy), x.grad)):
        assert ((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5 * (1 + want.abs())).all()


@pytest.mark.parametrize("rows,hidden", [(2, 2048), (43, 8192), (1000, 8192), (5000, 2048)])
def test_rmsnorm_backward_grid(dev, rows, hidden):
    """One, some and all of the CTAs the row count allows, with and without a residual, with the bounds of
    ``test_rmsnorm_backward_with_residual``."""
    test_rmsnorm_backward_with_residual(dev, rows, hidden)


@pytest.mark.parametrize("rows,vocab", [(1184, 32768), (1185, 32768), (3, 49144), (1185, 49144), (1185, 49152)])
def test_cross_entropy_dispatch(dev, rows, vocab):
    """Both sides of the rule that picks the CTA width, with the bounds of ``test_cross_entropy_row_widths``."""
    g = torch.Generator(device=dev).manual_seed(vocab)
    logits = (3 * torch.randn(rows, vocab, generator=g, device=dev)).bfloat16()
    labels = torch.randint(-1, vocab, (rows,), generator=g, device=dev)
    want = logits.clone()
    loss = model_ops.cross_entropy_inplace(logits, labels, 0.5)
    for lo in range(0, rows, 256):
        l64, lab, got = want[lo:lo + 256].double(), labels[lo:lo + 256], logits[lo:lo + 256].double()
        grad = l64.softmax(-1)
        tol = 1e-5 * grad + 1e-7
        grad[torch.arange(len(lab), device=dev), lab.clamp(min=0)] -= 1.0
        grad *= 0.5 * (lab >= 0)[:, None]
        assert ((got - grad).abs() <= 2.0 ** -8 * grad.abs() + tol).all()
        ref = torch.nn.functional.cross_entropy(l64, lab.clamp(min=0), reduction="none") * (lab >= 0)
        assert ((loss[lo:lo + 256] - ref).abs() < 1e-4).all()


@pytest.mark.parametrize("n,f", [(5, 72), (33, 320), (7, 1024), (2367, 1536), (2368, 1536), (2369, 1016), (2368, 1032), (3, 14336), (1300, 4104)])
def test_swiglu_dispatch(dev, n, f):
    """A CTA per row, several rows per CTA and several CTAs per row, with the bounds of ``test_swiglu_row_lengths``."""
    g = torch.Generator(device=dev).manual_seed(f)
    gu, dy = (4 * torch.randn(n, 2 * f, generator=g, device=dev)).bfloat16(), torch.randn(n, f, generator=g, device=dev).bfloat16()
    a, u = gu.double().chunk(2, dim=-1)
    sg = torch.sigmoid(a)
    want = (a * sg * u, torch.cat([dy.double() * u * (sg + a * sg * (1 - sg)), dy.double() * a * sg], -1))
    for got, ref in zip((model_ops.swiglu_fwd_raw(gu), model_ops.swiglu_bwd_raw(gu, dy)), want):
        assert ((got.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-5 * (1 + ref.abs())).all()


@pytest.mark.parametrize("n", [8, 8 * 257, 8 * (148 * 8 * 256 + 5)])
def test_scaled_gradients(dev, n):
    """The roundings are those of an fp32 product (the scalar is not rounded to bf16 first) and an accumulation of
    their own, bit for bit."""
    src, old = torch.randn(n, device=dev).bfloat16(), torch.randn(n, device=dev).bfloat16()
    src[0] = float("inf")
    for v in (1.0, 0.37):
        g = torch.tensor(v, device=dev)
        prod = (src.float() * g).bfloat16()
        assert torch.equal(model_ops.scale_rows(src, g), prod)
        dst = old.clone()
        model_ops.scale_rows(src, g, dst)
        assert torch.equal(dst, old + prod)


@pytest.mark.parametrize("runs", [[64], [65], [63, 2, 64, 1], [1, 63, 64, 128, 3], [5, 700, 59], [200, 1, 1, 1, 4500], [40000]])
def test_embedding_gradient_of_long_runs(dev, runs):
    """Runs of equal ids that end at, before and past the 64-place segments, with the bound of ``test_embedding_gradient``;
    the same bits in every run."""
    g = torch.Generator().manual_seed(len(runs))
    ids = torch.repeat_interleave(torch.arange(len(runs)) * 3 + 1, torch.tensor(runs))
    ids = ids[torch.randperm(ids.shape[0], generator=g)].to(dev)
    dy = torch.randn(ids.shape[0], 520, generator=g).bfloat16().to(dev)
    old = torch.randn(50, 520, generator=g).bfloat16().to(dev)
    add = torch.zeros(50, 520, dtype=torch.float64, device=dev).index_add_(0, ids, dy.double())
    mag = torch.zeros(50, 520, dtype=torch.float64, device=dev).index_add_(0, ids, dy.double().abs())
    want, first = old.double() + add, None
    for _ in range(3):
        grad = old.clone()
        model_ops.embedding_grad(ids, dy, grad)
        first = grad if first is None else first
        assert torch.equal(grad, first)
    assert ((first.double() - want).abs() <= 2.0 ** -8 * (add.abs() + want.abs()) + 1e-5 * mag + 1e-9).all()


@pytest.mark.parametrize("tokens", ["one", "same", "mixed"])
@pytest.mark.parametrize("hidden", [8, 520, 1024])
def test_embedding_gradient(dev, tokens, hidden):
    """fp32 sums (1e-5 of the magnitudes) rounded to bf16 before and after they are added to the old gradient (2^-8 of
    both); rows that no token names keep theirs."""
    g = torch.Generator().manual_seed(hidden)
    ids = {"one": torch.tensor([3]), "same": torch.full((1030,), 6), "mixed": torch.randint(0, 40, (700,), generator=g)}[tokens].to(dev)
    dy = torch.randn(ids.shape[0], hidden, generator=g).bfloat16().to(dev)
    grad = torch.randn(50, hidden, generator=g).bfloat16().to(dev)
    add = torch.zeros(50, hidden, dtype=torch.float64, device=dev).index_add_(0, ids, dy.double())
    mag = torch.zeros(50, hidden, dtype=torch.float64, device=dev).index_add_(0, ids, dy.double().abs())
    want, old = grad.double() + add, grad.clone()
    model_ops.embedding_grad(ids, dy, grad)
    assert ((grad.double() - want).abs() <= 2.0 ** -8 * (add.abs() + want.abs()) + 1e-5 * mag + 1e-9).all()
    rest = torch.ones(50, dtype=torch.bool, device=dev)
    rest[ids] = False
    assert torch.equal(grad[rest], old[rest])


def test_cross_entropy(dev):
    torch.manual_seed(0)
    logits = (3 * torch.randn(129, 4096, device=dev)).bfloat16()
    labels = torch.randint(0, 4096, (129,), device=dev)
    labels[5] = -100
    lr = logits.float().requires_grad_(True)
    ref = model_ops.cross_entropy_reference(lr, labels)
    (ref.sum() * 0.25).backward()
    loss = model_ops.cross_entropy_inplace(logits, labels, 0.25)
    assert (loss - ref.detach()).abs().max() < 2e-2
    assert (logits.float() - lr.grad).abs().max() < 2e-3
    assert loss[5] == 0 and logits[5].abs().max() == 0


def test_qkv_rope_split_and_pack(dev):
    torch.manual_seed(0)
    T, hq, hkv = 200, 8, 2
    qkv = torch.randn(T, (hq + 2 * hkv) * 128, device=dev).bfloat16()
    pos = torch.randint(0, 100000, (T,), device=dev)
    cos, sin = model_ops.rope_tables(pos, 500000.0, 128)
    q_arena = torch.zeros(T + 64, hq, 128, device=dev, dtype=torch.bfloat16)
    kv_arena = torch.zeros(T + 64, 2, hkv, 128, device=dev, dtype=torch.bfloat16)
    model_ops.qkv_rope_split(qkv, cos, sin, q_arena, kv_arena, hq, hkv, 32, 16)
    parts = qkv.view(T, hq + 2 * hkv, 128)
    assert (q_arena[32:32 + T].float() - model_ops.rope_reference(parts[:, :hq], cos, sin).float()).abs().max() < 3e-2
    assert (kv_arena[16:16 + T, 0].float() - model_ops.rope_reference(parts[:, hq:hq + hkv], cos, sin).float()).abs().max() < 3e-2
    assert torch.equal(kv_arena[16:16 + T, 1], parts[:, hq + hkv:])
    # the backward kernel applies the transposed rotation: <rope(x), g> == <x, rope^T(g)>
    dq = torch.randn(T + 64, hq, 128, device=dev)
    dkv = torch.randn(T + 64, 2, hkv, 128, device=dev)
    dqkv = model_ops.qkv_rope_pack_bwd(dq, dkv, cos, sin, T, hq, hkv, 32, 16).view(T, hq + 2 * hkv, 128).float()
    x = parts.float()
    lhs = (model_ops.rope_reference(x[:, :hq], cos, sin) * dq[32:32 + T]).sum() + \
          (model_ops.rope_reference(x[:, hq:hq + hkv], cos, sin) * dkv[16:16 + T, 0]).sum() + (x[:, hq + hkv:] * dkv[16:16 + T, 1]).sum()
    rhs = (x * dqkv).sum()
    assert abs(lhs - rhs) / abs(lhs) < 5e-3


def test_merge_out_lse_and_aliases(dev):
    torch.manual_seed(0)
    n, t, h = 3, 150, 4
    outs = torch.randn(n, t, h, 128, device=dev).bfloat16()
    lses = torch.randn(n, t, h, device=dev)
    lses[1, :10] = float("-inf")
    lses[:, 20] = float("-inf")
    o, l = block_ops.flash_attn_update_out_lse(outs, lses)
    ro, rl = block_ops.merge_out_lse_reference(outs, lses)
    fin = torch.isfinite(rl)
    assert (o.float() - ro)[fin].abs().max() < 2e-2
    assert (l - rl)[fin].abs().max() < 1e-4 and torch.isinf(l[~fin]).all()
    assert torch.allclose(block_ops.fused_blockwise_sum(outs).float(), outs.float().sum(0), atol=5e-2)
    block_ops.warmup_triton_ops()


def test_gather_push_cast(dev):
    torch.manual_seed(0)
    src = torch.randn(500, 4, 128, device=dev).bfloat16()
    dst = torch.zeros(300, 4, 128, device=dev, dtype=torch.bfloat16)
    ent = torch.tensor([[0, 10, 5, 100], [0, 400, 150, 77]], dtype=torch.int32, device=dev)
    block_ops.gather_rows(ent, [src], dst, 4 * 128 * 2)
    assert torch.equal(dst[5:105], src[10:110]) and torch.equal(dst[150:227], src[400:477]) and dst[105:150].abs().max() == 0
    stat = torch.randn(4, 500, device=dev)
    sdst = torch.zeros(4, 300, device=dev)
    block_ops.gather_stats(ent, [stat], sdst, 4, 500)
    assert torch.equal(sdst[:, 5:105], stat[:, 10:110])
    acc = torch.ones(300, 4, 128, device=dev)
    g = torch.randn(500, 4, 128, device=dev)
    block_ops.push_add_rows(ent, g, [acc], 4 * 128)     # (peer, src_row, dst_row, n)
    assert torch.allclose(acc[5:105], 1 + g[10:110]) and torch.allclose(acc[150:227], 1 + g[400:477])
    bf = torch.empty(300, 4, 128, device=dev, dtype=torch.bfloat16)
    block_ops.cast_f32_bf16(acc, bf)
    assert torch.equal(bf, acc.bfloat16())


def test_corrupt_tables_are_reported_not_executed(dev):
    """A table entry that points outside its arena makes the kernel set the bad-arguments status
    and skip the work; nothing is stored out of range and the context stays usable."""
    torch.manual_seed(0)
    nq, bs, hq, hkv = 256, 256, 4, 2
    q = torch.randn(nq + 128, hq, 128, device=dev).bfloat16()
    kv = torch.randn(bs + 128, 2, hkv, 128, device=dev).bfloat16()
    dout = torch.randn_like(q)
    out = torch.zeros_like(q)
    lse = torch.zeros(hq, nq + 128, device=dev)
    delta = torch.zeros_like(lse)
    rng = _ranges("causal", nq, 0)
    row = A.AttnRow(0, nq, list(range(hq)), [(0, bs)], rng)
    tabs = A.build_fwd_tables([row], bs, dev)
    tabs.tiles[0, 7] = 1 << 28                       # out_row far past the destination
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    A.attn_fwd(q, kv, tabs, [out], [lse], 128 ** -0.5, status, 0)
    torch.cuda.synchronize()
    assert status.item() == 3
    bt = A.build_bwd_tables([row], bs, hq, hkv, dev)
    bt.items[0, 5] = 1 << 28                         # dq_row far past the accumulator
    status.zero_()
    dq = torch.zeros(nq + 128, hq, 128, device=dev)
    dkv = torch.zeros(bs + 128, 2, hkv, 128, device=dev)
    A.attn_bwd(q, dout, kv, lse, delta, bt, [dq], [dkv], 128 ** -0.5, status)
    torch.cuda.synchronize()
    assert status.item() == 3
    assert torch.isfinite(dq).all() and torch.isfinite(dkv).all()
    assert torch.ones(4, device=dev).sum().item() == 4


def test_barrier_wait_is_bounded(dev):
    """A peer flag nobody sets: the barrier kernel gives up after its deadline and reports it."""
    flags = torch.zeros(64, dtype=torch.int32, device=dev)
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    # both "ranks" point at local memory; rank 1 never runs, so flags[1] of rank 0's row stays 0
    block_ops.signal_barrier([flags.data_ptr(), flags[32:].data_ptr()], 0, 2, 1, status, timeout_s=0.2)
    torch.cuda.synchronize()
    assert status.item() == 2
    assert flags[32].item() == 1          # our own arrival was published to the peer's row
    # the context is still usable
    assert torch.ones(4, device=dev).sum().item() == 4


def test_adamw_and_reduce_scatter_single_rank(dev):
    from dcp_b200.parallel.dist_optimizer import FlatBuffers, ShardedAdamW
    torch.manual_seed(0)
    n = 4096
    bufs = FlatBuffers(n, dev)
    bufs.params.copy_(torch.randn(n, device=dev).bfloat16())
    p0 = bufs.params.float().clone()
    opt = ShardedAdamW(bufs, lr=1e-2, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.1, clip_grad=None)
    ref_p = p0.clone().requires_grad_(True)
    ref = torch.optim.AdamW([ref_p], lr=1e-2, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.1)
    for _ in range(3):
        g = torch.randn(n, device=dev).bfloat16()
        bufs.grads.copy_(g)
        opt.step(1.0)
        ref_p.grad = g.float()
        ref.step()
    assert (opt.master - ref_p.detach()).abs().max() < 1e-5
    assert torch.equal(bufs.params, opt.master.bfloat16())


@pytest.mark.parametrize("d,heads", [(128, (8, 2)), (128, (5, 1)), (64, (8, 2)), (64, (6, 6)), (96, (4, 1))])
@pytest.mark.parametrize("kind", ["full", "causal", "two"])
def test_attention_backward_levels_of_dq(dev, d, heads, kind):
    """dQ through a buffer per 256 keys: the same bits in every run where it was cleared, also where all key tiles begin at the same
    query; elsewhere added to what dQ holds; within rounding of additions to one buffer (8 of 2^-24 of the largest partial sum,
    and 2^-20 of the largest element, which is at least 1 here).  Rows without keys keep what they hold, and so do channels beyond the
    heads'."""
    import dataclasses
    (hq, hkv), nq, nkv = heads, 520, 1100
    torch.manual_seed(d + hq)
    q, dout = torch.zeros(2, nq, hq, 128, device=dev, dtype=torch.bfloat16)
    kv = torch.zeros(nkv, 2, hkv, 128, device=dev, dtype=torch.bfloat16)
    for t in (q, dout, kv):
        t[..., :d] = torch.randn(*t.shape[:-1], d, device=dev).bfloat16()
    rng = np.zeros((nq, 4), np.int32)
    rng[:, 1] = nkv if kind == "full" else np.arange(nq) + 581
    if kind == "two":
        rng[:, 1], rng[:, 2], rng[:, 3] = 200, 600, np.arange(nq) + 581
        rng[100:140] = 0
    row = A.AttnRow(0, nq, list(range(hq)), [(0, nkv)], rng)
    out, lse, delta = torch.zeros_like(q), torch.zeros(hq, nq, device=dev), torch.zeros(hq, nq, device=dev)
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    A.attn_fwd(q, kv, A.build_fwd_tables([row], 1152, dev), [out], [lse], d ** -0.5, status, channels=d)
    A.attn_delta(out, dout, delta, 0, nq)
    levels = A.build_bwd_tables([row], 1152, hq, hkv, dev)
    assert levels.dq_levels == 5
    first = None
    for tables in [levels] * 12 + [dataclasses.replace(levels, dq_levels=0)]:
        junk = torch.full((5 * nq * hq * 128,), float("nan"), device=dev)
        del junk                                            # the buffers' memory
        dq, dkv = torch.zeros(nq, hq, 128, device=dev), torch.zeros(nkv, 2, hkv, 128, device=dev)
        dq[:, :, 3] = 1.0
        dq[..., d:] = 5.0
        A.attn_bwd(q, dout, kv, lse, delta, tables, [dq], [dkv], d ** -0.5, status, channels=d)
        first = first or (dq, dkv)
        assert torch.equal(dkv, first[1])
        if tables is levels:
            assert torch.equal(dq[..., :3], first[0][..., :3]) and torch.equal(dq[..., 4:], first[0][..., 4:])
            assert (dq[..., 3] - first[0][..., 3]).abs().max() <= 2.0 ** -20 * dq[..., :d].abs().max()
    assert status.item() == 0 and (first[0][..., d:] == 5.0).all()
    assert (dq - first[0]).abs().max() <= 2.0 ** -20 * dq[..., :d].abs().max()
    if kind == "two":
        assert (first[0][100:140, :, 3] == 1.0).all() and not first[0][100:140, :, :3].any()


def test_levels_of_dq_need_whole_key_tiles():
    """Key tiles that begin anywhere may share 256 positions with two others: no levels then."""
    rng = np.zeros((200, 4), np.int32)
    rng[:, 1] = 400
    rows = lambda bs: [A.AttnRow(0, 200, [0], [(0, min(bs, 400)), (400, 100)], rng)]
    assert A.build_bwd_tables(rows(200), 200, 1, 1, "cpu").dq_levels == 0
    assert A.build_bwd_tables(rows(256), 256, 1, 1, "cpu").dq_levels == 2
    assert A.build_bwd_tables([], 256, 1, 1, "cpu").dq_levels == 0
