"""GPU parity tests: every CUDA op, called through the C ABI, against the CPU oracle on the same
seeded inputs.  Integer / index results must be bit-exact; rerank scores within 1e-3 relative."""
import math

import numpy as np
import pytest
import torch

from conftest import bf16_from_bits, bits_of, srht_signs, synth_keys, synth_queries

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


@pytest.fixture(scope="module")
def ops():
    from pariskv_b200 import ops as _ops
    return _ops


def _encode_oracle_vs_gpu(ops, oracle, keys, signs, layout):
    bs, H, L, _ = keys.shape
    cb_o, w_o, pk_o = oracle.encode(keys, signs)
    kg, sg = keys.to(DEV), signs.to(DEV)
    counts = torch.zeros(bs, H, 16, 256, dtype=torch.int32, device=DEV)
    if layout == "key_major":
        cb, w, pk = ops.encode_keys(kg, sg, cluster_counts=counts)
    else:  # the reference's plane-major tensors, written through a view that starts at column 4
        cbf = torch.zeros(bs, H, 16, L + 8, dtype=torch.uint8, device=DEV)
        wf = torch.zeros(bs, H, 16, L + 8, dtype=torch.bfloat16, device=DEV)
        pkf = torch.zeros(bs, H, 16, L + 8, 4, dtype=torch.uint8, device=DEV)
        cb, w, pk = cbf[..., 4:4 + L], wf[..., 4:4 + L], pkf[..., 4:4 + L, :]
        ops.encode_keys(kg, sg, cb, w, pk, cluster_counts=counts)
    assert torch.equal(cb.cpu(), cb_o), "sign codes differ"
    assert torch.equal(pk.cpu(), pk_o), "4-bit codes differ"
    assert torch.equal(bits_of(w), bits_of(w_o)), "block weights differ"
    assert torch.equal(counts.cpu(), oracle.cluster_counts(cb_o))
    assert torch.equal(ops.count_clusters(cb).cpu(), oracle.cluster_counts(cb_o))
    return cb, w, pk, counts


@pytest.mark.parametrize("layout", ["key_major", "plane_major"])
@pytest.mark.parametrize("L", [1, 15, 16, 17, 127, 1000])
def test_encode_bit_exact(ops, oracle, layout, L):
    g = torch.Generator().manual_seed(L)
    keys = synth_keys(g, 2, 3, L)
    if L > 3:
        keys[0, 0, 0] = 0
        keys[0, 0, 1] = 0
        keys[0, 0, 1, 9] = 2.0
    _encode_oracle_vs_gpu(ops, oracle, keys, srht_signs(), layout)


def test_encode_golden(ops, golden):
    e = golden("encode")
    keys, signs = bf16_from_bits(e["keys"]), bf16_from_bits(e["signs"])
    cb, w, pk = ops.encode_keys(keys.to(DEV), signs.to(DEV))
    assert torch.equal(cb.cpu(), torch.from_numpy(e["codebook"]))
    assert torch.equal(pk.cpu(), torch.from_numpy(e["packed_4bit"]))
    assert torch.equal(bits_of(w), bits_of(bf16_from_bits(e["block_weight"])))


def test_encode_empty(ops):
    keys = torch.empty(1, 2, 0, 128, dtype=torch.bfloat16, device=DEV)
    cb, w, pk = ops.encode_keys(keys, srht_signs().to(DEV))
    assert cb.shape == (1, 2, 16, 0)


@pytest.mark.parametrize("group", [1, 4, 7])
def test_query_prep_and_rank(ops, oracle, group):
    g = torch.Generator().manual_seed(3 + group)
    keys = synth_keys(g, 2, 2, 64)
    q = synth_queries(g, keys, group)
    signs = srht_signs()
    qb_o, qn_o = oracle.query_prep(q, 2, signs)
    qb, qn, qa = ops.query_prep(q.to(DEV), 2, signs.to(DEV), want_avg=True)
    assert torch.equal(bits_of(qb), bits_of(qb_o))
    assert torch.equal(bits_of(qn), bits_of(qn_o))
    ids = ops.rank_clusters(qb)
    assert torch.equal(ids.cpu(), oracle.cluster_rank(qb_o))


def test_query_prep_golden(ops, golden):
    q = golden("query_collision")
    qb, qn = ops.query_prep(bf16_from_bits(q["queries"]).to(DEV), 2, bf16_from_bits(q["signs"]).to(DEV))
    assert torch.equal(bits_of(qb), bits_of(bf16_from_bits(q["q_blocks"])))
    assert torch.equal(bits_of(qn), bits_of(bf16_from_bits(q["q_norm"])))


def _rand_collision_inputs(gen, bs, H, B, NC, N):
    ids = torch.stack([torch.stack([torch.stack([torch.randperm(NC, generator=gen) for _ in range(B)])
                                    for _ in range(H)]) for _ in range(bs)])
    ckc = torch.randint(1, max(2, N // 4), (bs, H, B, NC), generator=gen, dtype=torch.int32)
    cb = torch.randint(0, NC, (bs, H, B, N), generator=gen, dtype=torch.int32).to(torch.uint8)
    return ids, ckc, cb


@pytest.mark.parametrize("N", [1, 31, 32, 33, 1023, 1025, 5000])
@pytest.mark.parametrize("layout", ["plane", "plane_offset4", "plane_offset3", "key_major", "generic"])
def test_collision_fused_bit_exact(ops, oracle, N, layout):
    g = torch.Generator().manual_seed(N)
    bs, H, B, NC = 2, 3, 16, 256
    ids, ckc, cb = _rand_collision_inputs(g, bs, H, B, NC, N)
    tiers = oracle.tier_counts(N * 40, 0.2)
    ref = oracle.collision(ids, ckc, cb, tiers)
    if layout == "plane":
        cbg = cb.to(DEV)
    elif layout.startswith("plane_offset"):
        off = int(layout[-1])
        full = torch.zeros(bs, H, B, N + 32, dtype=torch.uint8, device=DEV)
        full[..., off:off + N] = cb.to(DEV)
        cbg = full[..., off:off + N]
    elif layout == "key_major":
        cbg = cb.to(DEV).permute(0, 1, 3, 2).contiguous().permute(0, 1, 3, 2)
    else:  # odd strides: falls to the byte-wise kernel
        full = torch.zeros(bs, H, B, N + 5, dtype=torch.uint8, device=DEV)
        full[..., :N] = cb.to(DEV)
        cbg = full[..., :N]
    out = ops.collision_fused(ids.to(DEV), ckc.to(DEV), cbg, tiers)
    assert torch.equal(out.cpu(), ref)
    out32 = ops.collision_fused(ids.to(torch.int32).to(DEV), ckc.to(DEV), cbg, tiers[-1:])
    assert torch.equal(out32.cpu(), oracle.collision(ids, ckc, cb, tiers[-1:]))


def test_collision_golden(ops, golden):
    c = golden("collision")
    for tag in ("n2048", "n1000"):
        out = ops.collision_fused(torch.from_numpy(c[tag + "_sorted_ids"].astype(np.int64)).to(DEV),
                                  torch.from_numpy(c[tag + "_cluster_counts"]).to(DEV),
                                  torch.from_numpy(c[tag + "_codebook"]).to(DEV), c[tag + "_tier_counts"].tolist())
        assert torch.equal(out.cpu(), torch.from_numpy(c[tag + "_cache_cnt"]))
    cb = torch.from_numpy(c["single_codebook"]).to(DEV).transpose(-1, -2).contiguous()
    out = torch.empty(1, 2, 777, dtype=torch.int32, device=DEV)
    ops.collision(torch.from_numpy(c["single_sorted_ids"]).to(DEV), torch.from_numpy(c["single_topk_cluster_cnt"]).to(DEV),
                  cb, out)
    assert torch.equal(out.cpu(), torch.from_numpy(c["single_cache_cnt"]))


@pytest.mark.parametrize("L,k", [(1, 1), (31, 31), (33, 1), (1000, 100), (4097, 4096), (20000, 2000), (300000, 30000)])
@pytest.mark.parametrize("kind", ["counts", "float_counts", "float", "ties"])
def test_topk_exact(ops, oracle, L, k, kind):
    g = torch.Generator().manual_seed(L + k)
    rows = 3
    if kind == "counts":
        x = torch.randint(0, 97, (rows, L), generator=g, dtype=torch.int32)
    elif kind == "float_counts":
        x = torch.randint(0, 97, (rows, L), generator=g).to(torch.float32)
    elif kind == "float":
        x = torch.randn(rows, L, generator=g) * 50
    else:
        x = torch.randint(-2, 3, (rows, L), generator=g, dtype=torch.int32)
    out = ops.topk(x.to(DEV), k)
    assert torch.equal(out.cpu(), oracle.topk(x, k))
    if k <= 4096:
        out = ops.topk(x.to(DEV), k, order=1)
        assert torch.equal(out.cpu(), oracle.topk(x, k, sorted_by_value=True))


@pytest.mark.parametrize("case", ["all_equal", "two_values", "dense_ties_float", "negatives", "tiny_spread", "signed_zero"])
@pytest.mark.parametrize("L,k", [(1500, 1), (5000, 2048), (13101, 2048), (16384, 16000), (16384, 16384)])
def test_topk_short_rows_tie_paths(ops, oracle, L, k, case):
    """The selection's levels: values that agree in the top 12 / 24 bits, the threshold bin above and below its ranking
    capacity, and equal keys at the last bit."""
    g = torch.Generator().manual_seed(L * 7 + k)
    rows = 2
    if case == "all_equal":
        x = torch.full((rows, L), 3.25)
    elif case == "two_values":
        x = torch.randint(0, 2, (rows, L), generator=g).to(torch.float32) * 0.5 + 1.0
    elif case == "dense_ties_float":
        x = torch.randint(0, 40, (rows, L), generator=g).to(torch.float32) / 7.0
    elif case == "negatives":
        x = -torch.rand(rows, L, generator=g) * 1e-3
    elif case == "tiny_spread":   # all values share the top 24 key bits
        x = (1.0 + torch.randint(0, 200, (rows, L), generator=g).to(torch.float32) * 2.0 ** -23)
    else:
        x = torch.zeros(rows, L)
        x[:, ::3] = -0.0
        x[:, 1::5] = 1e-30
    out = ops.topk(x.to(DEV), k)
    assert torch.equal(out.cpu(), oracle.topk(x, k))


@pytest.mark.parametrize("L,k", [(3, 2), (100, 30), (5000, 1100), (40000, 4000)])
@pytest.mark.parametrize("low", [0, (1 << 24) - 2, (1 << 25) + 1, -(1 << 25) - 7, -(1 << 31), (1 << 31) - 100000])
def test_topk_whole_numbers_at_any_size(ops, oracle, L, k, low):
    """int32 rows that 32-bit floats cannot hold, on both sides of 256 distinct values (a bin per value below), and rows from
    end to end of the type."""
    g = torch.Generator().manual_seed(L + k)
    for span in (3, 256, 257, 100000, (1 << 32) - 1):
        lo, hi = (low, min(low + span, 1 << 31)) if span < 1 << 31 else (-(1 << 31), 1 << 31)
        x = torch.randint(lo, hi, (2, L), generator=g, dtype=torch.int64).to(torch.int32)
        x[0, 0], x[0, -1] = hi - 1, lo
        assert torch.equal(ops.topk(x.to(DEV), k).cpu(), oracle.topk(x, k)), span


@pytest.mark.parametrize("k", [1, 2, 300, 3000])
@pytest.mark.parametrize("kind", ["whole", "huge", "inf"])
def test_topk_at_the_upper_end_of_the_type(ops, oracle, k, kind):
    """Threshold bins that are cut further (over 1024 elements) and whose last part holds the highest values of the type: its
    bounds do not wrap around."""
    g = torch.Generator().manual_seed(k)
    if kind == "whole":
        x = torch.randint((1 << 31) - 3000, 1 << 31, (16, 5000), generator=g, dtype=torch.int64).to(torch.int32)
        x[:, 0], x[:, 77] = -(1 << 31), (1 << 31) - 1
    else:
        x = torch.randn(16, 5000, generator=g)
        x[:, 100:100 + min(k + 1, 2900)] = torch.finfo(torch.float32).max if kind == "huge" else float("inf")
        x[:, -1] = -x[:, 100]
    assert torch.equal(ops.topk(x.to(DEV), k).cpu(), oracle.topk(x, k))


def test_topk_3d_strided_rows(ops, oracle):
    g = torch.Generator().manual_seed(5)
    x = torch.randint(0, 97, (2, 4, 3000), generator=g, dtype=torch.int32)
    out = ops.topk(x.to(DEV)[:, :, :2500], 300)
    assert torch.equal(out.cpu(), oracle.topk(x[:, :, :2500].contiguous(), 300))


def test_topk_rejects_bad_k(ops):
    x = torch.zeros(2, 10, dtype=torch.int32, device=DEV)
    with pytest.raises(RuntimeError):
        ops.topk(x, 11)
    with pytest.raises(RuntimeError):
        ops.topk(x, 0)


def _rerank_inputs(gen, bs, H, N):
    sign = torch.randint(0, 2, (bs, H, 16, N, 8), generator=gen)
    mag = torch.randint(0, 8, (bs, H, 16, N, 8), generator=gen)
    v4 = (sign << 3) | mag
    k4 = ((v4[..., 1::2] << 4) | v4[..., 0::2]).to(torch.uint8)
    w = torch.randn(bs, H, 16, N, generator=gen).abs().to(torch.bfloat16)
    qb = torch.randn(bs, H, 16, 8, generator=gen).to(torch.bfloat16)
    qn = (torch.randn(bs, H, 1, generator=gen).abs() + 0.1).to(torch.bfloat16)
    return k4, w, qb, qn


@pytest.mark.parametrize("layout", ["key_major", "plane_major"])
@pytest.mark.parametrize("C", [1, 127, 129, 1500])
def test_rerank_matches_oracle(ops, oracle, layout, C):
    g = torch.Generator().manual_seed(C)
    bs, H, N = 2, 2, 3000
    k4, w, qb, qn = _rerank_inputs(g, bs, H, N)
    _, cen = oracle.constants()
    cand = torch.stack([torch.stack([torch.randperm(N, generator=g)[:C].sort().values for _ in range(H)])
                        for _ in range(bs)])
    s32_o, sbf_o = oracle.rerank(cand, k4, w, qb, qn, cen)
    if layout == "key_major":
        k4g = k4.to(DEV).permute(0, 1, 3, 2, 4).contiguous().permute(0, 1, 3, 2, 4)
        wg = w.to(DEV).permute(0, 1, 3, 2).contiguous().permute(0, 1, 3, 2)
    else:
        k4g, wg = k4.to(DEV), w.to(DEV)
    v4b = torch.zeros(bs, H, 16, C, 8, dtype=torch.bfloat16, device=DEV)
    sbf, s32 = ops.rerank(cand.to(DEV), k4g, wg, qb.to(DEV), qn.to(DEV), cen.to(DEV), v4b=v4b, want_f32=True)
    assert torch.equal(s32.cpu(), s32_o), "fp32 scores must be bit-identical to the oracle's pinned order"
    assert torch.equal(bits_of(sbf), bits_of(sbf_o))
    # the optional unpacked-level output equals +-center[level]
    nib = torch.stack([k4 & 0xF, k4 >> 4], -1).view(bs, H, 16, N, 8).long()
    lev = torch.where((nib & 8) > 0, cen.float()[nib & 7], -cen.float()[nib & 7])
    idx = cand.view(bs, H, 1, C, 1).expand(bs, H, 16, C, 8)
    assert torch.equal(v4b.float().cpu(), torch.gather(lev, 3, idx))


def test_rerank_golden_within_tolerance(ops, golden):
    r = golden("rerank")
    N = r["key_4bit"].shape[3]
    cand = torch.arange(N).view(1, 1, N).expand(1, 2, N).contiguous()
    _, s32 = ops.rerank(cand.to(DEV), torch.from_numpy(r["key_4bit"]).to(DEV), bf16_from_bits(r["key_block_weight"]).to(DEV),
                        bf16_from_bits(r["q_blocks"]).to(DEV), bf16_from_bits(r["q_norm"]).to(DEV),
                        bf16_from_bits(r["mag_centers"]).to(DEV), want_f32=True)
    ref = torch.from_numpy(r["scores_fp32"])
    rel = ((s32.cpu() - ref).abs() / ref.abs().clamp(min=1e-3 * ref.abs().max())).max().item()
    assert rel <= 1e-3, rel  # tolerance stated by the task: 1e-3 relative, fp32 accumulate
    fin = ops.final_topk(s32, cand.to(DEV), int(r["final_topk"]))
    for h in range(2):
        assert set(fin[0, h].tolist()) == set(r["final_fp32"][0, h].tolist())


def test_final_topk(ops, oracle):
    g = torch.Generator().manual_seed(11)
    s = torch.randn(2, 3, 5000, generator=g)
    s[0, 0, :100] = 1.5  # ties at the top
    cand = torch.stack([torch.stack([torch.randperm(40000, generator=g)[:5000].sort().values for _ in range(3)])
                        for _ in range(2)])
    out = ops.final_topk(s.to(DEV), cand.to(DEV), 256)
    assert torch.equal(out.cpu(), oracle.final_topk(s, cand, 256))


def test_adaptive_topk_golden_configs(ops, oracle, golden):
    a = golden("adaptive_topk")
    for i in range(4):
        cs = bf16_from_bits(a[f"c{i}_cand_scores"])
        scale = float(a[f"c{i}_attn_scale"])
        sl = torch.from_numpy(a[f"c{i}_sl_logits"])
        slv = torch.from_numpy(a[f"c{i}_sl_vnorm"])
        cv = torch.from_numpy(a[f"c{i}_cand_vnorm"])
        ci = torch.from_numpy(a[f"c{i}_cand_indices"].astype(np.int64))
        thr = float(a[f"c{i}_threshold"])
        K_out = min(int(a[f"c{i}_topk_cap"]), cs.shape[-1])
        k_ref = torch.from_numpy(a[f"c{i}_adaptive_k"])
        idx_ref = torch.from_numpy(a[f"c{i}_topk_indices"].astype(np.int64))
        # v2 form: bf16 scores scaled in the kernel
        k, idx = ops.adaptive_topk(sl.to(DEV), cs.to(DEV), scale, slv.to(DEV), ci.to(DEV), cv.to(DEV), thr, K_out)
        assert torch.equal(k.cpu(), k_ref), f"config {i}: adaptive_k differs from the reference"
        for b in range(k.shape[0]):
            for h in range(k.shape[1]):
                kk = int(k_ref[b, h])
                assert set(idx[b, h, :kk].tolist()) == set(idx_ref[b, h, :kk].tolist())
        # against the oracle everything is bit-exact, order included
        cl = torch.from_numpy((cs.float().numpy() * np.float32(scale)).astype(np.float32))
        k_o, idx_o = oracle.adaptive_topk(sl, slv, cl, cv, ci, thr, K_out)
        assert torch.equal(k.cpu(), k_o)
        assert torch.equal(idx.cpu(), idx_o)
        # v1 form: fp32 logits, scale 1; gathered value norms
        vn = torch.zeros(ci.shape[0], ci.shape[1], int(ci.max()) + 5)
        vn.scatter_(2, ci + 4, cv)
        k1, idx1 = ops.adaptive_topk(sl.to(DEV), cl.to(DEV), 1.0, slv.to(DEV), ci.to(DEV), None, thr, K_out,
                                     value_norm=vn.to(DEV), sink_size=4)
        assert torch.equal(k1.cpu(), k_o) and torch.equal(idx1.cpu(), idx_o)
        kc, _ = ops.adaptive_topk(sl.to(DEV), cs.to(DEV), scale, slv.to(DEV), ci.to(DEV), cv.to(DEV), thr, K_out,
                                  min_k=300, max_k=500)
        assert torch.equal(kc.cpu(), k_o.clamp(300, 500))


def test_h2d_gather_matches_indexing(ops, oracle):
    # the reference's own self-check shape: bs 2, 8 heads, N 32768, k 100 (cache_hub/gather_trans/trans_h2d.py:108-147)
    g = torch.Generator().manual_seed(0)
    bs, H, N, K = 2, 8, 32768, 100
    sk = torch.randn(bs, H, N, 128, generator=g).to(torch.bfloat16).pin_memory()
    sv = torch.randn(bs, H, N, 128, generator=g).to(torch.bfloat16).pin_memory()
    idx = torch.randint(0, N, (bs, H, K), generator=g)
    dk = torch.zeros(bs, H, 160, 128, dtype=torch.bfloat16, device=DEV)
    dv = torch.zeros_like(dk)
    ops.h2d_gather_kv(sk, sv, idx.to(DEV), dk, dv)
    assert torch.equal(dk[:, :, :K].cpu(), oracle.gather(sk, idx))
    assert torch.equal(dv[:, :, :K].cpu(), oracle.gather(sv, idx))
    assert dk[:, :, K:].abs().sum().item() == 0
    # host-side gather op
    out = torch.empty(bs, H, K, 128, dtype=torch.bfloat16)
    ops.gather_kv_out_cpu(sk, idx, out)
    assert torch.equal(out, oracle.gather(sk, idx))
    with pytest.raises(RuntimeError):
        bad = idx.clone()
        bad[0, 0, 0] = N
        ops.gather_kv_out_cpu(sk, bad, out)


def test_h2d_gather_packed(ops):
    g = torch.Generator().manual_seed(1)
    bs, H, N = 1, 4, 4096
    sk = torch.randn(bs, H, N, 128, generator=g).to(torch.bfloat16).pin_memory()
    sv = torch.randn(bs, H, N, 128, generator=g).to(torch.bfloat16).pin_memory()
    ks = [5, 0, 300, 77]
    sl_end = 10
    cu_topk = torch.tensor([0] + list(np.cumsum(ks)), dtype=torch.int32)
    cu_k = torch.tensor([0] + list(np.cumsum([k + sl_end for k in ks])), dtype=torch.int32)
    idx = torch.cat([torch.randperm(N, generator=g)[:k] for k in ks])
    kp = torch.zeros(int(cu_k[-1]), 128, dtype=torch.bfloat16, device=DEV)
    vp = torch.zeros_like(kp)
    ops.h2d_gather_kv_packed(sk, sv, kp, vp, idx.to(DEV), cu_topk.to(DEV), cu_k.to(DEV), sl_end, max(ks))
    for vh in range(4):
        sel = idx[cu_topk[vh]:cu_topk[vh + 1]]
        o = int(cu_k[vh]) + sl_end
        assert torch.equal(kp[o:o + ks[vh]].cpu(), sk[0, vh, sel])
        assert torch.equal(vp[o:o + ks[vh]].cpu(), sv[0, vh, sel])
        assert kp[int(cu_k[vh]):o].abs().sum().item() == 0


@pytest.mark.parametrize("store", ["pinned_host", "device"])
@pytest.mark.parametrize("n_window,K,group", [(0, 64, 4), (68, 0, 4), (196, 256, 4), (70, 1000, 7), (5, 33, 1)])
def test_sparse_attention(ops, oracle, store, n_window, K, group):
    g = torch.Generator().manual_seed(n_window + K)
    bs, H, N = 2, 2, 5000
    keys = synth_keys(g, bs, H, N)
    vals = torch.randn(bs, H, N, 128, generator=g).to(torch.bfloat16)
    q = synth_queries(g, keys, group) * 3
    wk = torch.randn(bs, H, 256, 128, generator=g).to(torch.bfloat16)
    wv = torch.randn(bs, H, 256, 128, generator=g).to(torch.bfloat16)
    sel = torch.stack([torch.stack([torch.randperm(N - 4, generator=g)[:K].sort().values for _ in range(H)])
                       for _ in range(bs)]) if K else None
    off = 4
    ks = keys.pin_memory() if store == "pinned_host" else keys.to(DEV)
    vs = vals.pin_memory() if store == "pinned_host" else vals.to(DEV)
    out = ops.sparse_attention(q.to(DEV), wk.to(DEV), wv.to(DEV), n_window, ks if K else None, vs if K else None,
                               sel.to(DEV) if K else None, index_offset=off)
    rows_k = [wk[:, :, :n_window]]
    rows_v = [wv[:, :, :n_window]]
    if K:
        rows_k.append(oracle.gather(keys, sel + off))
        rows_v.append(oracle.gather(vals, sel + off))
    ref = oracle.attention(q, torch.cat(rows_k, 2), torch.cat(rows_v, 2))
    err = (out.float().cpu() - ref).abs().max().item()
    assert err <= 2e-2, err  # bf16 output: max abs 2e-2


def test_sparse_attention_per_head_counts(ops, oracle):
    g = torch.Generator().manual_seed(9)
    bs, H, N, K = 1, 4, 2000, 300
    keys = synth_keys(g, bs, H, N)
    vals = torch.randn(bs, H, N, 128, generator=g).to(torch.bfloat16)
    q = synth_queries(g, keys, 4) * 3
    wk = torch.randn(bs, H, 80, 128, generator=g).to(torch.bfloat16)
    wv = torch.randn(bs, H, 80, 128, generator=g).to(torch.bfloat16)
    sel = torch.stack([torch.stack([torch.randperm(N, generator=g)[:K] for _ in range(H)]) for _ in range(bs)])
    n_sel = torch.tensor([[300, 0, 17, 129]], dtype=torch.int32)
    out = ops.sparse_attention(q.to(DEV), wk.to(DEV), wv.to(DEV), 80, keys.to(DEV), vals.to(DEV), sel.to(DEV),
                               n_sel=n_sel.to(DEV))
    for h in range(H):
        n = int(n_sel[0, h])
        kk = torch.cat([wk[:, h:h + 1], oracle.gather(keys[:, h:h + 1], sel[:, h:h + 1, :n])], 2)
        vv = torch.cat([wv[:, h:h + 1], oracle.gather(vals[:, h:h + 1], sel[:, h:h + 1, :n])], 2)
        ref = oracle.attention(q[:, :, 4 * h:4 * h + 4], kk, vv)
        assert (out[:, :, 4 * h:4 * h + 4].float().cpu() - ref).abs().max().item() <= 2e-2


@pytest.mark.parametrize("where", ["pinned_host", "device"])
def test_sparse_attention_interleaved_store(ops, where):
    """K and V rows as the two strided halves of one [bs,H,N,2,128] buffer give the same bits as separate stores."""
    g = torch.Generator().manual_seed(21)
    bs, H, N, K = 2, 2, 3000, 200
    keys = synth_keys(g, bs, H, N)
    vals = torch.randn(bs, H, N, 128, generator=g).to(torch.bfloat16)
    q = (synth_queries(g, keys, 4) * 3).to(DEV)
    wk = torch.randn(bs, H, 16, 128, generator=g).to(torch.bfloat16).to(DEV)
    wv = torch.randn(bs, H, 16, 128, generator=g).to(torch.bfloat16).to(DEV)
    sel = torch.stack([torch.stack([torch.randperm(N, generator=g)[:K].sort().values for _ in range(H)])
                       for _ in range(bs)]).to(DEV)
    kv = torch.stack((keys, vals), dim=3)
    kv = kv.pin_memory() if where == "pinned_host" else kv.to(DEV)
    a = ops.sparse_attention(q, wk, wv, 16, kv[:, :, :, 0], kv[:, :, :, 1], sel)
    b = ops.sparse_attention(q, wk, wv, 16, keys.to(DEV), vals.to(DEV), sel)
    assert torch.equal(a, b)
    with pytest.raises(RuntimeError):   # K and V must share strides
        ops.sparse_attention(q, wk, wv, 16, kv[:, :, :, 0], vals.to(DEV), sel)


@pytest.mark.parametrize("bs,H", [(1, 4), (10, 8)])   # a tile of 128 rows per block; several tiles of 64 in a row
@pytest.mark.parametrize("group", [1, 4, 5, 8, 9])
def test_sparse_attention_keeps_32_bits(ops, group, bs, H):
    """Probabilities and sums are held in 32 bits for every group size: hardly an output differs from the 64-bit result
    rounded to bf16.  An error e of the result before its rounding changes the rounding of a share of 2 |e| / ulp of the
    outputs.  Sums in 32 bits: |e| below 2^-18 of the absolute products' sum, which is some three times the result over rows
    of random sign, so 2 * 3 * 2^-18 / 2^-8 = 0.6 % at the very most (measured: below 0.1 %).  Probabilities rounded to
    bf16 change 7.8 % of these outputs."""
    g = torch.Generator(device=DEV).manual_seed(group * 100 + bs)
    n = 90
    k = torch.randn(bs, H, n, 128, generator=g, device=DEV).to(torch.bfloat16)
    v = torch.randn(bs, H, n, 128, generator=g, device=DEV).to(torch.bfloat16)
    q = torch.randn(bs, 1, H * group, 128, generator=g, device=DEV).to(torch.bfloat16)
    out = ops.sparse_attention(q, k, v, n)
    s = torch.einsum("bhgd,bhnd->bhgn", q.view(bs, H, group, 128).double(), k.double()) / math.sqrt(128.0)
    ref = torch.einsum("bhgn,bhnd->bhgd", torch.softmax(s, -1), v.double()).reshape(out.shape)
    assert (out != ref.to(torch.bfloat16)).double().mean().item() <= 0.006
    # an infinite value stays one: no product of the split probabilities turns it into something that is not a number
    v[0, 0, 17, 5] = float("inf")
    out = ops.sparse_attention(q, k, v, n)
    hit = torch.zeros_like(out, dtype=torch.bool)
    hit[0, 0, :group, 5] = True
    assert torch.equal(torch.isposinf(out), hit) and not torch.isnan(out).any()


@pytest.mark.parametrize("bs,H", [(1, 2), (20, 8)])   # blocks of a head in a cluster; two tiles of 64 in a row
@pytest.mark.parametrize("group", [1, 4, 8, 9])       # (9: the scalar form)
def test_sparse_attention_merges_partials_of_tiny_weight(ops, group, bs, H):
    """Rows 2^-130.6 of the others' weight hold an infinite value, in the block of the others and in one of their own: the factor
    that their partials are merged with is a subnormal number, not zero, so the output is infinite as in 64 bits."""
    g = torch.Generator(device=DEV).manual_seed(group)
    n = 256
    k = torch.zeros(bs, H, n, 128, dtype=torch.bfloat16, device=DEV)
    k[:, :, 16:, 0] = -32.0                                # q k / sqrt(128) = -90.5
    q = torch.zeros(bs, 1, H * group, 128, dtype=torch.bfloat16, device=DEV)
    q[..., 0] = 32.0
    v = torch.randn(bs, H, n, 128, generator=g, device=DEV).to(torch.bfloat16)
    v[:, :, 20, 5], v[:, :, 200, 6] = float("inf"), float("-inf")
    out = ops.sparse_attention(q, k, v, n).view(bs, H, group, 128)
    s = torch.einsum("bhgd,bhnd->bhgn", q.view(bs, H, group, 128).double(), k.double()) / math.sqrt(128.0)
    ref = torch.einsum("bhgn,bhnd->bhgd", torch.softmax(s, -1), v.double())
    assert torch.isposinf(ref[..., 5]).all() and torch.isneginf(ref[..., 6]).all()
    assert torch.equal(torch.isposinf(out), torch.isposinf(ref)) and torch.equal(torch.isneginf(out), torch.isneginf(ref))
    rest = torch.isfinite(ref)
    assert (out.double()[rest] - ref[rest]).abs().max().item() <= 2e-2


# ---- glue kernels of the sequence-sharded form (against the torch formulation used by the gloo tests) ----
def test_shard_pack_unpack_owned_merge(ops):
    from pariskv_b200 import dist as pkd
    g = torch.Generator().manual_seed(11)
    bs, H, C, Kl, world, start = 2, 3, 5000, 257, 3, 70000
    cand = torch.stack([torch.randperm(40000, generator=g)[:C].sort().values for _ in range(bs * H)]).view(bs, H, C)
    scores = torch.randn(bs, H, C, generator=g)
    pos = torch.stack([torch.randperm(C, generator=g)[:Kl].sort().values for _ in range(bs * H)]).view(bs, H, Kl)
    fin = torch.gather(cand, 2, pos)
    packed = ops.shard_pack_topk(cand.cuda(), scores.cuda(), fin.cuda(), start).cpu()
    assert torch.equal(packed[..., 1], fin + start)
    assert torch.equal(packed[..., 0].to(torch.int32).view(torch.float32), torch.gather(scores, 2, pos))

    gathered = torch.randint(-2 ** 31, 2 ** 31 - 1, (world, bs, H, Kl, 2), generator=g, dtype=torch.int64)
    sc, idx = ops.shard_unpack_topk(gathered.cuda())
    want = gathered.permute(1, 2, 0, 3, 4).reshape(bs, H, world * Kl, 2)
    assert torch.equal(idx.cpu(), want[..., 1])
    assert torch.equal(sc.cpu().view(torch.int32), want[..., 0].to(torch.int32))

    final = torch.stack([torch.randperm(100000, generator=g)[:Kl].sort().values for _ in range(bs * H)]).view(bs, H, Kl)
    for (s, e) in ((0, 100000), (30000, 60000), (99999, 100000), (50, 50)):
        local, n = ops.shard_owned_rows(final.cuda(), s, e)
        wl, wn = pkd.owned_rows(final, s, e)
        assert torch.equal(n.cpu(), wn)
        for b in range(bs):
            for h in range(H):
                k = int(wn[b, h])
                assert torch.equal(local.cpu()[b, h, :k], wl[b, h, :k])
                assert int(local.cpu()[b, h, k:].abs().sum()) == 0

    Hq = 8
    parts = torch.randn(world, bs, Hq, 129, generator=g)
    parts[..., 128] *= 6
    parts[1, :, 2, 128] = float("-inf")                 # a rank without rows for some heads
    parts[:, 1, 5, 128] = float("-inf")                 # nobody has rows: result 0
    parts[..., :128] = parts[..., :128].to(torch.bfloat16).float()
    got = ops.shard_merge_partial(parts.cuda()).float().cpu()
    want = pkd.merge_gathered_partials(parts)
    want[1, 0, 5] = 0
    assert (got - want).abs().max().item() <= 1e-2
    out = parts[0, :, :, :128].to(torch.bfloat16).unsqueeze(1).contiguous()
    pp = ops.shard_pack_partial(out.cuda(), parts[0, :, :, 128].contiguous().cuda()).cpu()
    assert torch.equal(pp[..., :128], out[:, 0].float()) and torch.equal(pp[..., 128], parts[0, :, :, 128])


def test_peer_exchange_wait_runs_out_and_reports():
    """The flag wait of the peer-memory exchange is bounded: with a flag word that no rank ever publishes the
    collecting kernel gives up after about a second, raises the status word of the control block and returns —
    the context stays usable and the host can tell."""
    import ctypes
    import time
    from pariskv_b200 import _lib as L
    world, bs, H, Kl = 2, 1, 2, 64
    gather_off, flags_off = 0, world * bs * H * Kl * 16
    buf = torch.zeros(flags_off + 256, dtype=torch.uint8, device=DEV)        # gather area and flags of "this rank"
    ctl = torch.zeros(8, dtype=torch.int32, device=DEV)
    ctl[0] = 1                                                              # exchange 1 was started locally ...
    buf[flags_off:flags_off + 4] = torch.tensor([1, 0, 0, 0], dtype=torch.uint8, device=DEV)   # ... rank 0 published,
    scores = torch.empty(bs, H, world * Kl, dtype=torch.float32, device=DEV)                    # rank 1 never does
    indices = torch.empty(bs, H, world * Kl, dtype=torch.int64, device=DEV)
    ds, di = L.desc(scores), L.desc(indices)
    torch.cuda.synchronize()
    t0 = time.time()
    rc = L.load().pk_shard_collect_topk(buf.data_ptr(), gather_off, flags_off, ctl.data_ptr(), world, Kl,
                                        L.ref(ds), L.ref(di), L.stream_ptr(torch.device(DEV)))
    assert rc == 0
    torch.cuda.synchronize()
    waited = time.time() - t0
    assert int(ctl[2]) == 1, "the expired wait was not reported"
    assert 0.05 < waited < 20.0, waited
    # the context is intact: the same call with both flags published returns at once and leaves the status alone
    ctl[2] = 0
    buf[flags_off + 4:flags_off + 8] = torch.tensor([1, 0, 0, 0], dtype=torch.uint8, device=DEV)
    rc = L.load().pk_shard_collect_topk(buf.data_ptr(), gather_off, flags_off, ctl.data_ptr(), world, Kl,
                                        L.ref(ds), L.ref(di), L.stream_ptr(torch.device(DEV)))
    torch.cuda.synchronize()
    assert rc == 0 and int(ctl[2]) == 0
    assert int(indices.abs().sum()) == 0 and float(scores.abs().sum()) == 0.0   # the zeroed gather area, unpacked


def test_tp_reduce_wait_runs_out_and_reports():
    """The one-launch reduction over peer memory with a peer that never sends: two local buffers stand for the two
    ranks' gather areas, this "rank 0" stores into both and then waits for rank 1's slots, which nobody fills.  The
    wait is bounded: the launch ends after about a second with the status word raised, the context stays usable, and
    the same exchange with rank 1's slots filled in by hand returns the right sum at once."""
    import time
    from pariskv_b200 import _lib as L
    world, n = 2, 512
    area = world * n * 4
    mine = torch.zeros(2 * area, dtype=torch.uint8, device=DEV)       # rank 0's two gather areas
    other = torch.zeros(2 * area, dtype=torch.uint8, device=DEV)      # rank 1's (only written to)
    ctl = torch.zeros(4, dtype=torch.int32, device=DEV)
    part = torch.randn(1, n).to(torch.bfloat16).to(DEV)
    res = torch.randn(1, n).to(torch.bfloat16).to(DEV)
    out = torch.empty_like(part)
    bases = L.u64_array([mine.data_ptr(), other.data_ptr()])
    d = [L.desc(part), L.desc(res), L.desc(out)]

    def call():
        rc = L.load().pk_tp_allreduce(L.ref(d[0]), L.ref(d[1]), L.ref(d[2]), bases, world, 0, 0, area, 0, ctl.data_ptr(),
                                      None, None, 1e-6, L.stream_ptr(torch.device(DEV)))
        assert rc == 0
        torch.cuda.synchronize()

    t0 = time.time()
    call()                                                            # exchange 1 -> area 1
    waited = time.time() - t0
    assert int(ctl[2]) == 1, "the expired wait was not reported"
    assert 0.05 < waited < 20.0, waited
    # exchange 2 -> area 0: fill rank 1's slots {two bf16, exchange number} by hand, then the launch returns at once
    ctl[2] = 0
    theirs = torch.randn(1, n).to(torch.bfloat16).to(DEV)
    slots = mine.view(torch.int32).view(2, world, n // 2, 2)          # [area][source rank][word]{data, number}
    slots[0, 1, :, 0] = theirs.view(torch.int32).view(-1)
    slots[0, 1, :, 1] = 2
    t0 = time.time()
    call()
    assert time.time() - t0 < 0.5 and int(ctl[2]) == 0
    want = (res.float() + part.float() + theirs.float()).to(torch.bfloat16)
    assert torch.equal(out, want)


def test_mirror_rerank_v4b_is_optional_and_correct(ops, oracle):
    """Documented difference from the reference wrapper (cache_hub/rerank/rerank.py:214-263): the debug tensor v4b
    is produced only on request.  Without want_v4b the second return value is None; with it the tensor holds the
    signed magnitude levels of every candidate, the values the reference writes."""
    from pariskv_b200.cache_hub.rerank.rerank import partial_rerank_cuda
    g = torch.Generator().manual_seed(3)
    pk, w, qb, qn = (t.to(DEV) for t in _rerank_inputs(g, 1, 2, 900))
    cen = oracle.constants()[1].to(DEV)
    cand = torch.stack([torch.randperm(900, generator=g)[:130].sort().values for _ in range(2)]).view(1, 2, 130).to(DEV)
    s0, none = partial_rerank_cuda(cand, pk, w, qb, qn, cen, 16, 8)
    assert none is None
    s1, v4b = partial_rerank_cuda(cand, pk, w, qb, qn, cen, 16, 8, want_v4b=True)
    assert torch.equal(s0, s1) and v4b.shape == (1, 2, 16, 130, 8)
    codes = torch.gather(pk.cpu(), 3, cand.cpu()[:, :, None, :, None].expand(1, 2, 16, 130, 4)).to(torch.int32)
    nib = torch.stack([codes & 0xF, codes >> 4], -1).view(1, 2, 16, 130, 8)
    lev = cen.cpu().float()[(nib & 7).long()] * torch.where((nib & 8) != 0, 1.0, -1.0)
    assert torch.equal(v4b.float().cpu(), lev)


def test_mirror_rerank_fused_returns_ascending_indices(ops, oracle):
    """Documented difference from cache_hub/rerank/rerank.py:266-294: rerank_rabitq_fused returns the final indices in
    ascending key order (the reference returns them ordered by score); the SET is the top-K by fp32 score."""
    from pariskv_b200.cache_hub.rerank.rerank import rerank_rabitq_fused
    g = torch.Generator().manual_seed(4)
    pk, w, qb, qn = (t.to(DEV) for t in _rerank_inputs(g, 1, 2, 3000))
    cen = oracle.constants()[1].to(DEV)
    cnt = torch.randint(0, 97, (1, 2, 3000), generator=g, dtype=torch.int32).to(DEV)
    fin, sbf, _ = rerank_rabitq_fused(cnt, pk, w, qb, qn, cen, 0.2, 100, 16, 8)
    assert fin.shape == (1, 2, 100) and bool((fin[..., 1:] > fin[..., :-1]).all())
    cand = ops.topk(cnt, 600)
    _, s32 = ops.rerank(cand, pk, w, qb, qn, cen, want_f32=True)
    for h in range(2):
        order = sorted(range(600), key=lambda i: (-float(s32[0, h, i]), i))[:100]
        assert sorted(int(cand[0, h, i]) for i in order) == fin[0, h].tolist()


def test_torch_custom_ops_run_the_same_kernels(ops, oracle):
    """torch.ops.pariskv.* (the registered custom ops the mirror modules call) give the bits of the direct calls."""
    from pariskv_b200 import torch_ops  # noqa: F401
    g = torch.Generator().manual_seed(8)
    ids, counts, codes = _rand_collision_inputs(g, 1, 2, 16, 256, 3000)
    tiers = [30, 90, 180, 300, 450, 600]
    a = torch.ops.pariskv.collision_fused(ids.to(DEV), counts.to(DEV), codes.to(DEV), list(tiers))
    assert torch.equal(a, ops.collision_fused(ids.to(DEV), counts.to(DEV), codes.to(DEV), tiers))
    cand = torch.ops.pariskv.topk(a, 300)
    assert torch.equal(cand, ops.topk(a, 300))
    pk, w, qb, qn = (t.to(DEV) for t in _rerank_inputs(g, 1, 2, 3000))
    cen = oracle.constants()[1].to(DEV)
    s = torch.ops.pariskv.rerank(cand, pk, w, qb, qn, cen)
    assert torch.equal(s, ops.rerank(cand, pk, w, qb, qn, cen)[0])
    src_k = torch.randn(1, 2, 3000, 128, generator=g).to(torch.bfloat16).pin_memory()
    src_v = torch.randn(1, 2, 3000, 128, generator=g).to(torch.bfloat16).pin_memory()
    dk = torch.zeros(1, 2, 300, 128, dtype=torch.bfloat16, device=DEV)
    dv = torch.zeros_like(dk)
    torch.ops.pariskv.gather_trans(src_k, src_v, cand, dk, dv)
    idx = cand.cpu()[..., None].expand(1, 2, 300, 128)
    assert torch.equal(dk.cpu(), torch.gather(src_k, 2, idx)) and torch.equal(dv.cpu(), torch.gather(src_v, 2, idx))


# ---- decode glue: the elementwise steps of a decoder layer ---------------------------------------------------------
@pytest.mark.parametrize("B,Hq,Hk", [(1, 32, 8), (3, 4, 1), (16, 32, 8)])
def test_qk_norm_rope_against_fp32(ops, B, Hq, Hk):
    """y = x * rsqrt(mean(x^2) + eps) * w per head, then rotate-half RoPE; fp32 torch reference, bf16 tolerance."""
    g = torch.Generator().manual_seed(B * 100 + Hq)
    heads = Hq + Hk
    qkv = torch.randn(B, (heads + Hk) * 128, generator=g).to(torch.bfloat16)
    w = (1.0 + 0.2 * torch.randn(heads, 128, generator=g)).to(torch.bfloat16)
    ang = torch.rand(B, 64, generator=g) * 6.28
    cos = torch.cos(ang).repeat(1, 2).to(torch.bfloat16)
    sin = torch.cat([-torch.sin(ang), torch.sin(ang)], -1).to(torch.bfloat16)
    for cs in ((cos, sin), (cos[:1].contiguous(), sin[:1].contiguous())):
        out = ops.qk_norm_rope(qkv.to(DEV), w.to(DEV), cs[0].to(DEV), cs[1].to(DEV), 1e-6)
        x = qkv[:, :heads * 128].float().view(B, heads, 128)
        y = (x * torch.rsqrt((x * x).mean(-1, keepdim=True) + 1e-6) * w.float()).to(torch.bfloat16).float()
        ref = y * cs[0].float().view(-1, 1, 128) + torch.roll(y, 64, -1) * cs[1].float().view(-1, 1, 128)
        assert out.shape == (B, heads, 128)
        assert (out.float().cpu() - ref).abs().max().item() <= 3e-2


@pytest.mark.parametrize("B,n", [(1, 4096), (5, 1024), (2, 8192), (1, 40)])
def test_add_rmsnorm_and_silu_mul_against_fp32(ops, B, n):
    g = torch.Generator().manual_seed(n + B)
    a = torch.randn(B, n, generator=g).to(torch.bfloat16)
    r = torch.randn(B, n, generator=g).to(torch.bfloat16)
    w = (1.0 + 0.2 * torch.randn(n, generator=g)).to(torch.bfloat16)
    for res in (r, None):
        h, x = ops.add_rmsnorm(a.to(DEV), None if res is None else res.to(DEV), w.to(DEV), 1e-6)
        hr = (a.float() + (0 if res is None else res.float())).to(torch.bfloat16)
        assert torch.equal(h.cpu(), hr)          # one bf16 rounding of an exact fp32 sum
        xr = hr.float() * torch.rsqrt((hr.float() ** 2).mean(-1, keepdim=True) + 1e-6) * w.float()
        assert (x.float().cpu() - xr).abs().max().item() <= 2e-2 * max(1.0, xr.abs().max().item())
    gu = torch.randn(B, 2 * n, generator=g).to(torch.bfloat16)
    act = ops.silu_mul(gu.to(DEV))
    ref = torch.nn.functional.silu(gu[:, :n].float()) * gu[:, n:].float()
    assert act.shape == (B, n)
    assert (act.float().cpu() - ref).abs().max().item() <= 2e-2 * max(1.0, ref.abs().max().item())


def test_glue_argument_errors(ops):
    with pytest.raises(Exception):
        ops.silu_mul(torch.zeros(1, 20, dtype=torch.bfloat16, device=DEV))       # F = 10 is not a multiple of 8
    with pytest.raises(Exception):
        ops.add_rmsnorm(torch.zeros(1, 64, dtype=torch.bfloat16, device=DEV), None,
                        torch.zeros(32, dtype=torch.bfloat16, device=DEV))


def test_stage_timing_inside_a_replayed_graph(ops):
    """Launches captured while timing is on are bracketed by event nodes that every replay stamps again."""
    from pariskv_b200 import _lib
    gu = torch.randn(4, 2 * 4096, device=DEV).to(torch.bfloat16)
    ops.silu_mul(gu)                                   # first use outside the capture
    torch.cuda.synchronize()
    _lib.timing_clear_graph()
    _lib.timing_enable(True)
    try:
        g = torch.cuda.CUDAGraph()
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            g.capture_begin()
            out = ops.silu_mul(gu)
            out2 = ops.silu_mul(gu)
            g.capture_end()
        torch.cuda.current_stream().wait_stream(side)
    finally:
        _lib.timing_enable(False)
    for _ in range(3):
        g.replay()
        torch.cuda.synchronize()
        got = _lib.timing_read_graph()
        assert got["glue"][1] == 2 and 0.0 < got["glue"][0] < 50.0      # two launches, milliseconds
    assert torch.equal(out, out2)
    del g
    _lib.timing_clear_graph()
    assert _lib.timing_read_graph() == {}


@pytest.mark.parametrize("O,I", [(6144, 4096), (4096, 12288), (1001, 520), (2, 8)])
def test_gemv_against_fp32(ops, O, I):
    """One-token projection: fp32 accumulation, one bf16 rounding; plain and gated ([gate; up] stacked, silu in the
    epilogue, rounded like the separate launches)."""
    g = torch.Generator().manual_seed(O + I)
    W = (torch.randn(O, I, generator=g) * 0.05).to(torch.bfloat16)
    x = torch.randn(1, I, generator=g).to(torch.bfloat16)
    y = ops.gemv(W.to(DEV), x.to(DEV))
    ref = x.float() @ W.float().t()
    assert y.shape == (1, O)
    assert (y.float().cpu() - ref).abs().max().item() <= 1e-2 * max(1.0, ref.abs().max().item())
    if O % 2 == 0:
        act = ops.gemv(W.to(DEV), x.to(DEV), gated=True)
        gu = ref.to(torch.bfloat16).float()
        want = torch.nn.functional.silu(gu[:, :O // 2]).to(torch.bfloat16).float() * gu[:, O // 2:]
        assert act.shape == (1, O // 2)
        assert (act.float().cpu() - want).abs().max().item() <= 3e-2 * max(1.0, want.abs().max().item())


# Every number of pieces per lane and several splits of the columns over the warps, rows that do not divide by the blocks, fewer
# rows than blocks, and more than one panel of 128 rows per block (148 blocks on B200).
@pytest.mark.parametrize("O,I", [(1, 8), (7, 256), (150, 264), (148 * 3 + 1, 1024), (600, 1280), (300, 12288), (290, 2048 + 16), (333, 9000), (444, 5120),
                                 (298, 15000), (150, 24576), (148 * 2 * 131, 32), (148 * 300 + 7, 136)])
def test_gemv_splits_against_fp64(ops, O, I):
    """fp32 sums of I products and one rounding to bf16 (2^-8 of the value): the sums' error is below I * 2^-24 of the sum of
    magnitudes whatever their order."""
    g = torch.Generator().manual_seed(O + I)
    W = (torch.randn(O, I, generator=g) * 0.05).to(torch.bfloat16)
    x = torch.randn(1, I, generator=g).to(torch.bfloat16)
    W[0, :] = 0.0
    if O > 2:
        W[O - 1] = 1.0
    y = ops.gemv(W.to(DEV), x.to(DEV)).double().cpu()
    ref, mag = x.double() @ W.double().t(), x.double().abs() @ W.double().abs().t()
    assert ((y - ref).abs() <= 2.0 ** -8 * ref.abs() + I * 2.0 ** -24 * mag + 1e-30).all()
    if O % 2 == 0:
        act = ops.gemv(W.to(DEV), x.to(DEV), gated=True).double().cpu()
        gate, up = ref[:, :O // 2], ref[:, O // 2:]
        want = torch.nn.functional.silu(gate) * up
        # two roundings of either factor (gate, silu(gate); up), one of the product; silu's slope is below 1.1
        err = 2.0 ** -8 * (1.1 * gate.abs() * up.abs() + 3 * want.abs()) + I * 2.0 ** -22 * (mag[:, :O // 2] * up.abs() + mag[:, O // 2:] * gate.abs() + 1)
        assert ((act - want).abs() <= err).all()


# Slices of the most elements that are kept in shared memory (16-bit counts of 512 bins; all of them in one bin, or nearly) and one
# group more (32-bit counts of 256 bins), on the largest cluster and on one CTA; slices around 4096 (512 and 1024 threads).
@pytest.mark.parametrize("rows,L", [(1, 16 * 32768), (1, 16 * 32768 + 1), (150, 32768), (150, 32769), (3, 16 * 511), (2, 5000), (1, 16 * 4064),
                                    (1, 16 * 4064 + 1), (150, 4064), (150, 4065)])
@pytest.mark.parametrize("kind", ["equal", "two values", "one off", "wide ints", "floats", "floats with inf and nan"])
def test_topk_bins_at_the_edges_of_a_slice(ops, rows, L, kind):
    g = torch.Generator(device=DEV).manual_seed(L + rows)
    if kind == "equal":
        x = torch.full((rows, L), 7, dtype=torch.int32, device=DEV)
    elif kind == "two values":
        x = torch.randint(0, 2, (rows, L), generator=g, device=DEV, dtype=torch.int32)
    elif kind == "one off":
        x = torch.zeros(rows, L, device=DEV)
        x[:, L // 3] = 1e30
    elif kind == "wide ints":
        x = torch.randint(-2 ** 31, 2 ** 31 - 1, (rows, L), generator=g, device=DEV, dtype=torch.int32)
    else:
        x = torch.randn(rows, L, generator=g, device=DEV)
        if "nan" in kind:
            x[:, L // 2], x[:, L // 5], x[:, 11] = float("inf"), float("nan"), -float("inf")
    for k in (1, 100, L // 50 + 1):
        got = ops.topk(x, k)
        key = x.double() if x.dtype == torch.int32 else torch.where(x.isnan(), torch.full_like(x, float("inf")), x).double()
        if "nan" in kind:
            key[:, L // 5] = 3e38 * 10   # above infinity
            key[:, L // 2] = 3e38 * 5
        want = torch.sort(key, dim=1, descending=True, stable=True).indices[:, :k].sort(dim=1).values
        assert torch.equal(got, want), (kind, k)


# Fewer selected rows than the launch is sized for, in the streaming, the cluster and the one-tile form: a head's rows are spread
# anew over its blocks, at counts around the edges of their shares.
@pytest.mark.parametrize("bs,H,G,K,n_window", [(8, 8, 4, 4000, 70), (16, 8, 2, 2048, 132), (1, 8, 4, 4096, 20), (3, 2, 5, 2000, 0), (2, 8, 8, 900, 200), (1, 2, 12, 700, 33)])
@pytest.mark.parametrize("on_device", [False, True])
def test_attention_spreads_the_rows_that_there_are(ops, bs, H, G, K, n_window, on_device):
    g = torch.Generator(device=DEV).manual_seed(K)
    cap, cap_w = K + 500, n_window + 50
    q = torch.randn(bs, 1, H * G, 128, generator=g, device=DEV).to(torch.bfloat16)
    wk, wv = (torch.randn(bs, H, cap_w, 128, generator=g, device=DEV).to(torch.bfloat16) for _ in range(2))
    store = torch.randn(bs, H, cap, 2, 128, generator=g, device=DEV).to(torch.bfloat16)
    sel = torch.rand(bs, H, cap, generator=g, device=DEV).argsort(-1)[..., :K].sort(-1).values.contiguous()
    edges = [0, 1, 63, 64, 65, 127, 128, 129, 191, 192, 193, 250, 384, 500, 640, 641, 767, 768, 769, K - 64, K - 1, K]
    n_sel = torch.tensor([max(0, min(K, edges[i % len(edges)])) for i in range(bs * H)], dtype=torch.int32, device=DEV).view(bs, H)
    rows_dev = torch.tensor([n_window - 3], dtype=torch.int32, device=DEV)
    more = dict(n_window_dev=rows_dev, n_window_add=3) if on_device else {}
    out = ops.sparse_attention(q, wk, wv, cap_w if on_device else n_window, store[..., 0, :], store[..., 1, :], sel, n_sel=n_sel, **more)
    for b in range(bs):
        for h in range(H):
            idx = sel[b, h, :int(n_sel[b, h])]
            k = torch.cat([store[b, h, idx, 0], wk[b, h, :n_window]]).double()
            v = torch.cat([store[b, h, idx, 1], wv[b, h, :n_window]]).double()
            got = out[b, 0, h * G:(h + 1) * G].double()
            if k.shape[0] == 0:
                assert not got.any()
                continue
            p = torch.softmax(q[b, 0, h * G:(h + 1) * G].double() @ k.t() / 128 ** 0.5, -1)
            # fp32 sums and probabilities of 17 bits, then one rounding to bf16: 2^-9 of the value, 2^-14 of the weighted magnitudes
            assert ((got - p @ v).abs() <= 2.0 ** -8 * (p @ v).abs() + 2.0 ** -14 * (p @ v.abs())).all()


# As many rows as SMs (148 on B200) and more, at slices around 4096 elements, around the most of which two blocks share an SM
# (2 * (16384 + 8192 + 1152 + 4 n + 2048) = 228 KB: n = 22240) and around those kept in shared memory: blocks of 512 and 1024 threads.
@pytest.mark.parametrize("rows", [148, 149, 300])
@pytest.mark.parametrize("L", [4064, 4065, 22240, 22241, 32768, 32769])
@pytest.mark.parametrize("dtype", [torch.int32, torch.float32])
def test_topk_more_rows_than_fit_at_once(ops, rows, L, dtype):
    g = torch.Generator(device=DEV).manual_seed(rows + L)
    x = torch.randint(-40, 40, (rows, L), generator=g, device=DEV, dtype=torch.int32) if dtype is torch.int32 else torch.randn(rows, L, generator=g, device=DEV)
    x[:, L // 2] = x[:, 3]
    for k in (1, L // 20, L):
        want = torch.sort(x.double(), dim=1, descending=True, stable=True).indices[:, :k].sort(dim=1).values
        assert torch.equal(ops.topk(x, k), want)


# Rows dealt out a step at a time from 8 steps of 148 blocks on (a step is 16 outputs at 2048 columns, 8 at 4096 and 5120, 2 at 12288
# and 13824, half of that gated, 1 at 24576 gated): one output fewer, just as many, a last step of one output and of some blocks only.
@pytest.mark.parametrize("I,step,gated", [(2048, 16, False), (4096, 8, False), (4096, 4, True), (5120, 8, False), (5120, 4, True), (12288, 2, False),
                                          (13824, 2, False), (13824, 1, True), (24576, 1, True), (24576, 1, False)])
@pytest.mark.parametrize("more", [-1, 0, 1, 7])
def test_gemv_rows_in_turn_against_fp64(ops, I, step, gated, more):
    """The bounds of test_gemv_splits_against_fp64."""
    n = 8 * 148 * step + (more if more < 7 else 7 + 70 * step)
    g = torch.Generator(device=DEV).manual_seed(I + n)
    W = (torch.randn(2 * n if gated else n, I, generator=g, device=DEV) * 0.05).to(torch.bfloat16)
    x = torch.randn(1, I, generator=g, device=DEV).to(torch.bfloat16)
    ref = torch.cat([x.double() @ part.double().t() for part in W.split(4096)], 1)
    mag = torch.cat([x.double().abs() @ part.double().abs().t() for part in W.split(4096)], 1)
    y = ops.gemv(W, x, gated=gated).double()
    if gated:
        gate, up = ref[:, :n], ref[:, n:]
        want = torch.nn.functional.silu(gate) * up
        err = 2.0 ** -8 * (1.1 * gate.abs() * up.abs() + 3 * want.abs()) + I * 2.0 ** -22 * (mag[:, :n] * up.abs() + mag[:, n:] * gate.abs() + 1)
        assert ((y - want).abs() <= err).all()
    else:
        assert ((y - ref).abs() <= 2.0 ** -8 * ref.abs() + I * 2.0 ** -24 * mag + 1e-30).all()


@pytest.mark.parametrize("bs,H,G,K", [(8, 8, 4, 4000), (1, 8, 4, 2048), (2, 2, 8, 900), (1, 2, 12, 700)])
@pytest.mark.parametrize("count", [-33, -1000, -2 ** 31])
def test_attention_takes_a_count_below_zero_for_no_rows(ops, bs, H, G, K, count):
    """The rows of a head are counted from words on the device: one so far below zero that the window rows do not make up for it
    leaves the head without rows, an output of zeros, in every form; the heads beside it are not touched."""
    g = torch.Generator(device=DEV).manual_seed(K)
    q = torch.randn(bs, 1, H * G, 128, generator=g, device=DEV).to(torch.bfloat16)
    w = torch.randn(bs, H, 40, 128, generator=g, device=DEV).to(torch.bfloat16)
    store = torch.randn(bs, H, K, 2, 128, generator=g, device=DEV).to(torch.bfloat16)
    sel = torch.arange(K, device=DEV).expand(bs, H, K).contiguous()
    n_sel = torch.full((bs, H), K, dtype=torch.int32, device=DEV)
    want = ops.sparse_attention(q, w, w, 33, store[..., 0, :], store[..., 1, :], sel, n_sel=n_sel)
    n_sel[0, 1] = count
    got = ops.sparse_attention(q, w, w, 33, store[..., 0, :], store[..., 1, :], sel, n_sel=n_sel)
    assert not got[0, 0, G:2 * G].any()
    got[0, 0, G:2 * G] = want[0, 0, G:2 * G]
    assert torch.equal(got, want)


@pytest.mark.parametrize("hidden,ffn", [(1024, 3072), (4096, 12288)])
def test_gemv_with_early_loads_gives_the_same_bits(ops, hidden, ffn):
    """norm -> gate and up -> down, each launch reading what the one before it wrote: with early loads the weights are read before the
    wait, x never is.  Plain launches give the values."""
    from pariskv_b200 import _lib
    g = torch.Generator(device=DEV).manual_seed(hidden)
    gu, down = ((torch.randn(o, i, generator=g, device=DEV) * 0.03).to(torch.bfloat16) for o, i in ((2 * ffn, hidden), (hidden, ffn)))
    norm = torch.ones(hidden, dtype=torch.bfloat16, device=DEV)
    xs = torch.randn(24, 1, hidden, generator=g, device=DEV).to(torch.bfloat16)

    def run():
        h, out = torch.zeros(1, hidden, dtype=torch.bfloat16, device=DEV), []
        for x in xs:
            h, n = ops.add_rmsnorm(x, h, norm)
            h = ops.gemv(down, ops.gemv(gu, n, gated=True))
            out.append(h)
        return torch.cat(out)

    try:
        _lib.set_dependent_launch(False)
        want = run()
        _lib.set_dependent_launch(True)
        assert torch.equal(run(), want)
        _lib.set_pdl(True)
        for _ in range(5):
            assert torch.equal(run(), want)
    finally:
        _lib.set_dependent_launch(True)
