"""The retrieval chain over the shapes its launch rule tells apart (clusters of 1 .. 16 blocks per head, and the launches
over all SMs beyond), and attention at the group sizes where its form changes."""
import math

import pytest
import torch

from conftest import srht_signs, synth_keys, synth_queries

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# (batch, heads, keys, candidates, K): one key; fewer keys than a cluster has blocks; odd slices; many heads (one block per
# head); candidates crowded into one slice; every key a candidate; equal keys only (flat counts and scores); a long zone
@pytest.mark.parametrize("bs,H,N,C,K,kind", [
    (1, 1, 1, 1, 1, "plain"), (1, 3, 9, 5, 2, "plain"), (1, 8, 8191, 820, 100, "plain"), (2, 4, 20011, 4003, 2048, "plain"),
    (5, 8, 3001, 700, 256, "plain"), (20, 8, 1500, 300, 64, "plain"), (1, 2, 30000, 9000, 1000, "crowded"),
    (1, 2, 5000, 5000, 3000, "plain"), (1, 2, 9000, 4000, 1500, "equal"), (1, 1, 700001, 70001, 2048, "plain")])
def test_retrieve_matches_oracle(oracle, bs, H, N, C, K, kind):
    from pariskv_b200 import ops
    g = torch.Generator().manual_seed(N + bs)
    keys = synth_keys(g, bs, H, N)
    if kind == "equal":
        keys = keys[:, :, :1].expand(bs, H, N, 128).contiguous()
    q = synth_queries(g, keys, 4)
    if kind == "crowded":                    # a third of the zone points with the query: most candidates come from there
        m = q.view(bs, 4 * H, 128).view(bs, H, 4, 128).float().mean(2, keepdim=True)
        keys[:, :, 3000:13000] = (keys[:, :, 3000:13000].float() * 0.2 + m / m.norm(dim=-1, keepdim=True) * 8.0).to(torch.bfloat16)
    signs = srht_signs()
    _, cen = oracle.constants()
    counts = torch.zeros(bs, H, 16, 256, dtype=torch.int32, device=DEV)
    cb, w, pk = ops.encode_keys(keys.to(DEV), signs.to(DEV), cluster_counts=counts)
    cb_o, w_o, pk_o = oracle.encode(keys, signs)
    assert torch.equal(cb.cpu(), cb_o)
    ref = oracle.retrieve(q, signs, cb_o, w_o, pk_o, oracle.cluster_counts(cb_o), cen, 0.25, C, K)
    tiers = oracle.tier_counts(N, 0.25)
    fin, ex = ops.retrieve(q.to(DEV), signs.to(DEV), cen.to(DEV), cb, w, pk, counts, tiers, C, K, want=("cand", "scores_f32"))
    assert torch.equal(ex["cand"].cpu(), ref["cand"])
    assert torch.equal(ex["scores_f32"].cpu(), ref["score32"])
    assert torch.equal(fin.cpu(), ref["final"])
    fin2, _ = ops.retrieve(q.to(DEV), signs.to(DEV), cen.to(DEV), cb, w, pk, counts, tiers, C, K)   # nothing but the result
    assert torch.equal(fin2, fin)
    _, ex2 = ops.retrieve(q.to(DEV), signs.to(DEV), cen.to(DEV), cb, w, pk, counts, tiers, C, 0, want=("cand", "scores_f32"))
    assert torch.equal(ex2["cand"].cpu(), ref["cand"]) and torch.equal(ex2["scores_f32"].cpu(), ref["score32"])


def _records(bs, H, N, size, first=0):
    """Views of the 4-bit codes and the weights in records of `size` bytes, the first `first` records not used."""
    rec = torch.zeros(bs, H, N + first, size, dtype=torch.uint8, device=DEV)[:, :, first:]
    return rec.view(torch.bfloat16)[..., 32:48].permute(0, 1, 3, 2), rec[..., :64].unflatten(-1, (16, 4)).permute(0, 1, 3, 2, 4)


# lists of less than, exactly and one more than the 32 candidates of a warp's round; odd rounds; one block and clusters; the
# form in several launches
@pytest.mark.parametrize("layout", ["arrays", "96", "112", "128", "128 from the fourth", "planes"])
@pytest.mark.parametrize("bs,H,N,C", [(1, 1, 31, 31), (1, 1, 40, 32), (1, 2, 33, 33), (1, 2, 3001, 1029), (20, 8, 700, 130), (1, 1, 700001, 3001)])
def test_rerank_of_any_record_layout(oracle, bs, H, N, C, layout):
    from pariskv_b200 import ops
    g = torch.Generator().manual_seed(N + C)
    keys = synth_keys(g, bs, H, N)
    q = synth_queries(g, keys, 4)
    signs = srht_signs()
    _, cen = oracle.constants()
    counts = torch.zeros(bs, H, 16, 256, dtype=torch.int32, device=DEV)
    cb = torch.zeros(bs, H, N, 16, dtype=torch.uint8, device=DEV).permute(0, 1, 3, 2)
    if layout == "planes":
        cb = cb.contiguous()
        w, pk = torch.zeros(bs, H, 16, N, dtype=torch.bfloat16, device=DEV), torch.zeros(bs, H, 16, N, 4, dtype=torch.uint8, device=DEV)
    elif layout == "arrays":
        w = torch.zeros(bs, H, N, 16, dtype=torch.bfloat16, device=DEV).permute(0, 1, 3, 2)
        pk = torch.zeros(bs, H, N, 16, 4, dtype=torch.uint8, device=DEV).permute(0, 1, 3, 2, 4)
    else:
        w, pk = _records(bs, H, N, int(layout.split()[0]), 4 if "from" in layout else 0)
    ops.encode_keys(keys.to(DEV), signs.to(DEV), cb, w, pk, cluster_counts=counts)
    cb_o, w_o, pk_o = oracle.encode(keys, signs)
    assert torch.equal(cb.cpu(), cb_o) and torch.equal(w.cpu().float(), w_o.float()) and torch.equal(pk.cpu(), pk_o)
    K = (C + 1) // 2
    ref = oracle.retrieve(q, signs, cb_o, w_o, pk_o, oracle.cluster_counts(cb_o), cen, 0.25, C, K)
    fin, ex = ops.retrieve(q.to(DEV), signs.to(DEV), cen.to(DEV), cb, w, pk, counts, oracle.tier_counts(N, 0.25), C, K,
                           want=("cand", "scores_f32"))
    assert torch.equal(ex["cand"].cpu(), ref["cand"])
    assert torch.equal(ex["scores_f32"].cpu(), ref["score32"])
    assert torch.equal(fin.cpu(), ref["final"])


# The bins of the final selection lie between the extremes of every warp's first 32 candidates: with norms that rise along the
# zone all that is selected lies beyond them, with falling ones nothing; one block per head and clusters
@pytest.mark.parametrize("bs,H,N,K", [(20, 8, 1500, 300), (1, 8, 6000, 700), (1, 1, 9000, 1), (1, 2, 9000, 8999)])
@pytest.mark.parametrize("step", [3.0, -3.0])
def test_final_selection_beyond_the_first_rounds(oracle, bs, H, N, K, step):
    from pariskv_b200 import ops
    g = torch.Generator().manual_seed(N + K)
    norm = torch.exp(torch.linspace(-step / 2, step / 2, N)).view(1, 1, N, 1)
    keys = (synth_keys(g, bs, H, N).float() * norm).to(torch.bfloat16)
    q = synth_queries(g, keys, 4)
    signs = srht_signs()
    _, cen = oracle.constants()
    counts = torch.zeros(bs, H, 16, 256, dtype=torch.int32, device=DEV)
    cb, w, pk = ops.encode_keys(keys.to(DEV), signs.to(DEV), cluster_counts=counts)
    ref = oracle.retrieve(q, signs, cb.cpu(), w.cpu(), pk.cpu(), counts.cpu(), cen, 0.25, N, K)
    fin, _ = ops.retrieve(q.to(DEV), signs.to(DEV), cen.to(DEV), cb, w, pk, counts, oracle.tier_counts(N, 0.25), N, K)
    assert torch.equal(fin.cpu(), ref["final"])


# Scores that are not numbers or infinite (positions of the zone): a NaN ranks above infinity.  Positions from 512 on lie behind the
# first round of every warp (of the first block of a cluster), whose extremes the bins lie between; with weights that are 64 times as
# large there, most of what is selected lies above that range, as the NaN does.  The weights as arrays of planes: the form in several
# launches
@pytest.mark.parametrize("bs,H,N", [(20, 8, 1500), (1, 8, 6000), (1, 1, 9000)])
@pytest.mark.parametrize("nan,inf,rise", [((3,), (), False), ((3, 40), (5,), False), ((), (3, 5), False), ((550,), (), False),
                                          ((3, 550), (560,), False), ((550, 555), (560,), False), ((550,), (), True)])
def test_final_selection_with_scores_that_are_no_numbers(oracle, bs, H, N, nan, inf, rise):
    from pariskv_b200 import ops
    g = torch.Generator().manual_seed(N)
    keys = synth_keys(g, bs, H, N)
    q = synth_queries(g, keys, 4)
    signs = srht_signs()
    _, cen = oracle.constants()
    counts = torch.zeros(bs, H, 16, 256, dtype=torch.int32, device=DEV)
    cb, w, pk = ops.encode_keys(keys.to(DEV), signs.to(DEV), cluster_counts=counts)
    if rise:
        w[..., 512:] *= 64
    for n in nan:
        w[:, :, 7, n] = float("nan")
    for n in inf:
        w[:, :, 7, n] = float("inf")   # of either sign in the score, as the key's code has it
    args = (counts, oracle.tier_counts(N, 0.25), N)
    forms = [(cb, w, pk), (cb.contiguous(), w.contiguous(), pk.contiguous())]
    for K in (2, 300):
        for form in forms:
            fin, ex = ops.retrieve(q.to(DEV), signs.to(DEV), cen.to(DEV), *form, *args, K, want=("cand", "scores_f32"))
            assert torch.equal(ex["scores_f32"].isnan().sum(-1).cpu(), torch.full((bs, H), len(nan)))
            assert torch.equal(ex["cand"], torch.arange(N, device=DEV).expand(bs, H, N))
            at = torch.sort(ex["scores_f32"], dim=-1, descending=True, stable=True).indices[..., :K].sort(dim=-1).values
            assert torch.equal(fin, at)


# more entries per block than it lists in shared memory (4096), and just as many
@pytest.mark.parametrize("rows,L,K", [(1, 300000, 290000), (3, 100000, 65536), (200, 9000, 4097), (200, 9000, 4096)])
def test_final_topk_of_long_lists(oracle, rows, L, K):
    from pariskv_b200 import ops
    g = torch.Generator().manual_seed(L + K)
    scores = torch.randn(1, rows, L, generator=g)
    cand = torch.randint(0, 1 << 40, (1, rows, L), generator=g)
    at = torch.sort(torch.sort(scores, dim=-1, descending=True, stable=True).indices[..., :K], dim=-1).values
    assert torch.equal(ops.final_topk(scores.to(DEV), cand.to(DEV), K).cpu(), torch.gather(cand, 2, at))


@pytest.mark.parametrize("group", [5, 8, 9])
@pytest.mark.parametrize("n_window,K", [(1, 0), (63, 1), (64, 64), (70, 1000)])
def test_attention_group_sizes(oracle, group, n_window, K):
    from pariskv_b200 import ops
    g = torch.Generator().manual_seed(group * 1000 + K)
    bs, H, N = 2, 3, 1500
    kv = torch.randn(bs, H, N, 2, 128, generator=g).to(torch.bfloat16)
    q = (torch.randn(bs, 1, H * group, 128, generator=g) * 3).to(torch.bfloat16)
    wk = torch.randn(bs, H, 256, 128, generator=g).to(torch.bfloat16)
    wv = torch.randn(bs, H, 256, 128, generator=g).to(torch.bfloat16)
    rk, rv, args = [wk[:, :, :n_window]], [wv[:, :, :n_window]], ()
    if K:
        sel = torch.stack([torch.stack([torch.randperm(N, generator=g)[:K].sort().values for _ in range(H)]) for _ in range(bs)])
        dkv = kv.to(DEV)
        args = (dkv[:, :, :, 0], dkv[:, :, :, 1], sel.to(DEV))
        rk.append(oracle.gather(kv[:, :, :, 0].contiguous(), sel))
        rv.append(oracle.gather(kv[:, :, :, 1].contiguous(), sel))
    out = ops.sparse_attention(q.to(DEV), wk.to(DEV), wv.to(DEV), n_window, *args)
    ref = oracle.attention(q, torch.cat(rk, 2), torch.cat(rv, 2))
    assert (out.float().cpu() - ref).abs().max().item() <= 2e-2


# (heads, window, selected rows): clusters of 16 blocks with a tile each, of 9 with two, of 13 with three, of 6 with three; a
# head over more blocks than a cluster has; last tiles of a row, and heads without any
@pytest.mark.parametrize("H,n_window,K", [(1, 1, 2047), (8, 196, 2048), (4, 1, 4900), (16, 100, 2048), (2, 100, 6100), (8, 5, 2044), (3, 0, 900)])
@pytest.mark.parametrize("group,offset", [(4, 0), (8, 0), (5, 2)])
def test_attention_in_a_cluster(oracle, H, n_window, K, group, offset):
    from pariskv_b200 import ops
    g = torch.Generator().manual_seed(K + group)
    kv = torch.randn(1, H, K + 50, 2, 128, generator=g).to(torch.bfloat16)
    q = (torch.randn(1, 1, H * group, 128, generator=g) * 3).to(torch.bfloat16)
    wk, wv = (torch.randn(1, H, max(n_window, 1), 128, generator=g).to(torch.bfloat16) for _ in range(2))
    sel = torch.stack([torch.randperm(K + 50, generator=g)[:K] for _ in range(H)])[None]
    n_sel = torch.randint(0, K + 1, (1, H), generator=g, dtype=torch.int32)
    n_sel[0, 0], n_sel[0, -1] = K, 0 if H > 1 else K
    dkv = kv.to(DEV)
    buf = torch.zeros(H * group * 128 + offset, dtype=torch.bfloat16, device=DEV)   # an output that is not 8-byte aligned
    out = buf[offset:].view(1, 1, H * group, 128)
    lse = torch.empty(1, H * group, dtype=torch.float32, device=DEV)
    ops.sparse_attention(q.to(DEV), wk.to(DEV) if n_window else None, wv.to(DEV) if n_window else None, n_window, dkv[:, :, :, 0], dkv[:, :, :, 1],
                         sel.to(DEV), n_sel=n_sel.to(DEV), out=out, lse=lse)
    for h in range(H):
        n = int(n_sel[0, h])
        k = torch.cat([kv[:, h:h + 1, sel[0, h, :n], 0], wk[:, h:h + 1, :n_window]], 2)
        v = torch.cat([kv[:, h:h + 1, sel[0, h, :n], 1], wv[:, h:h + 1, :n_window]], 2)
        mine = slice(h * group, (h + 1) * group)
        if k.shape[2] == 0:
            assert (out[:, :, mine] == 0).all() and (lse[:, mine] == -float("inf")).all()
            continue
        ref = oracle.attention(q[:, :, mine].contiguous(), k.contiguous(), v.contiguous())
        assert (out[:, :, mine].float().cpu() - ref).abs().max().item() <= 2e-2
        logits = torch.einsum("gd,nd->gn", q[0, 0, mine].double(), k[0, 0].double()) / 128 ** 0.5
        want = torch.logsumexp(logits, 1) / math.log(2.0)
        assert (lse[0, mine].double().cpu() - want).abs().max().item() <= 1e-4   # 32-bit sums of some thousand terms


@pytest.mark.parametrize("bs,H,n_window,K", [(1, 1, 127, 0), (1, 1, 128, 1), (1, 2, 1, 127), (2, 37, 100, 156), (2, 37, 100, 157)])
def test_attention_tile_edges(oracle, bs, H, n_window, K):
    """One tile of 128 rows per block up to a block per SM (2 x 37 heads of 256 rows on 148 SMs), tiles of 64 beyond."""
    from pariskv_b200 import ops
    g = torch.Generator().manual_seed(n_window + K)
    k, v = (torch.randn(bs, H, 300, 128, generator=g).to(torch.bfloat16) for _ in range(2))
    q = (torch.randn(bs, 1, 4 * H, 128, generator=g) * 3).to(torch.bfloat16)
    wk, wv = (torch.randn(bs, H, n_window, 128, generator=g).to(torch.bfloat16) for _ in range(2))
    sel = torch.stack([torch.stack([torch.randperm(300, generator=g)[:K] for _ in range(H)]) for _ in range(bs)])
    args = (k.to(DEV), v.to(DEV), sel.to(DEV)) if K else ()
    out = ops.sparse_attention(q.to(DEV), wk.to(DEV), wv.to(DEV), n_window, *args)
    rk, rv = ([torch.cat([oracle.gather(k, sel), wk], 2), torch.cat([oracle.gather(v, sel), wv], 2)] if K else (wk, wv))
    assert (out.float().cpu() - oracle.attention(q, rk, rv)).abs().max().item() <= 2e-2


def test_attention_shared_scratch_serves_any_batch():
    """Calls without their own scratch, few heads first and then many: the arrival counters of the second lie where the
    partial records of the first may have been."""
    from pariskv_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(3)
    assert ops.attention_scratch_bytes(7, 9, 64) - (7 * 9 + 64) // 64 * 256 == 7 * 9 * 132 * 4   # the header's length
    for bs, H in ((1, 1), (10, 8), (1, 4), (3, 30), (40, 8), (1, 1), (1100, 8), (2, 3), (1024, 8), (1100, 8), (1, 1)):
        k, v = (torch.randn(bs, H, 150, 128, generator=g, device=DEV).to(torch.bfloat16) for _ in range(2))
        q = torch.randn(bs, 1, 2 * H, 128, generator=g, device=DEV).to(torch.bfloat16)
        s = torch.einsum("bhgd,bhnd->bhgn", q.view(bs, H, 2, 128).double(), k.double()) / 128 ** 0.5
        ref = torch.einsum("bhgn,bhnd->bhgd", torch.softmax(s, -1), v.double()).reshape(q.shape)
        assert (ops.sparse_attention(q, k, v, 150).double() - ref).abs().max().item() <= 2e-2, (bs, H)


@pytest.mark.filterwarnings("ignore")
def test_mirror_ops_under_transforms_and_tracing():
    """The mirror modules call the library themselves on plain eager tensors only: function transforms, graph capture by
    tracing and tensors that need gradients go through the dispatcher, which batches, records or refuses them."""
    from pariskv_b200 import torch_ops
    from pariskv_b200.cache_hub.topk import bucket_topk
    x = torch.randint(0, 90, (3, 2, 500), dtype=torch.int32, device=DEV, generator=torch.Generator(DEV).manual_seed(1))
    want = torch.stack([bucket_topk(r, 7) for r in x])

    def f(r):
        return bucket_topk(r, 7)
    assert torch.equal(torch.vmap(f)(x), want)
    assert torch.equal(torch.func.functionalize(f)(x[0]), want[0])
    traced = torch.jit.trace(f, (x[0],), check_trace=False)
    assert torch.equal(traced(x[1]), want[1])
    assert torch_ops.direct(x) and not torch_ops.direct(x, torch.zeros(2, device=DEV, requires_grad=True))
    assert not torch_ops.direct(x.as_subclass(type("Sub", (torch.Tensor,), {})))
    neg = torch._neg_view(torch.randn(2, 500, device=DEV))
    assert not torch_ops.direct(neg) and torch.equal(bucket_topk(neg, 7), bucket_topk(neg.clone(), 7))
    with torch.device("cpu"):
        assert not torch_ops.direct(x)


# Heads of which clusters of 10, 6, 5, 4, 3 and 2 blocks are taken (on B200): from four blocks on, the sixteen tier tables are made
# by the blocks in turn and exchanged, unevenly with 5, 6 and 10; the counting's last round is one of 3 keys, or a whole one.
@pytest.mark.parametrize("bs,H,N", [(1, 8, 12003), (2, 8, 12003), (1, 20, 12003), (11, 2, 12160), (3, 8, 12003), (13, 2, 12003), (7, 4, 12160), (5, 6, 12003),
                                    (4, 8, 12003), (33, 1, 12160), (6, 6, 12003), (5, 8, 12003), (9, 6, 12003), (9, 8, 12003)])
def test_retrieve_on_clusters_of_every_size(oracle, bs, H, N):
    from pariskv_b200 import ops
    g = torch.Generator().manual_seed(N + bs * H)
    keys = synth_keys(g, bs, H, N)
    q, signs, C, K = synth_queries(g, keys, 2), srht_signs(), 2000, 700
    _, cen = oracle.constants()
    counts = torch.zeros(bs, H, 16, 256, dtype=torch.int32, device=DEV)
    cb, w, pk = ops.encode_keys(keys.to(DEV), signs.to(DEV), cluster_counts=counts)
    ref = oracle.retrieve(q, signs, cb.cpu(), w.cpu(), pk.cpu(), counts.cpu(), cen, 0.25, C, K)
    fin, ex = ops.retrieve(q.to(DEV), signs.to(DEV), cen.to(DEV), cb, w, pk, counts, oracle.tier_counts(N, 0.25), C, K,
                           want=("cand", "scores_f32"))
    assert torch.equal(ex["cand"].cpu(), ref["cand"])
    assert torch.equal(ex["scores_f32"].cpu(), ref["score32"])
    assert torch.equal(fin.cpu(), ref["final"])
