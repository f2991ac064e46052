"""The one-launch prompt ingestion against the oracle: window rows, zone records, histogram, store rows, value norms and
position words, at prompt lengths around the edges of the window and of a block's rounds."""
import pytest
import torch

from conftest import bits_of

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("offload", [True, False])
@pytest.mark.parametrize("P", [1, 20, 21, 51, 84, 85, 700, 4301])
def test_prefill_matches_oracle(oracle, P, offload):
    from pariskv_b200.cache_hub.polar_cache_adaptivek_varlen import polar_cache
    H, sink, local, bs = 3, 4, 16, 2
    cache = polar_cache(valid_start=[5, 5], layer_num=1, batch_size=bs, max_length=P + 5 + 32, num_key_value_heads=H,
                        num_heads=2 * H, head_dim=128, dtype=torch.bfloat16, layer_mapping={"0": DEV}, max_new_length=32,
                        sink_size=sink, local_size=local, final_topk=16, dynamic_update_interval=8, enable_offload=offload)
    g = torch.Generator().manual_seed(P)
    k = torch.randn(bs, P + 5, H, 128, generator=g)
    k[..., [7, 37, 71, 101]] *= 8.0
    k[:, 5, 0] = 0.0                                   # a zero key
    k = (k * torch.exp(0.5 * torch.randn(bs, P + 5, H, 1, generator=g))).to(torch.bfloat16)
    v = torch.randn(bs, P + 5, H, 128, generator=g).to(torch.bfloat16)
    for _ in range(2):                                 # the second prompt overwrites the first one's histogram
        cache.prefill_update_kv_cache(None, k.to(DEV), v.to(DEV), 0, 0)
    cache.sync(0, 0)
    torch.cuda.synchronize()
    N = max(0, P - sink - local)
    n_win = sink + local if N else P
    assert cache._layer_state[0].tolist() == [n_win, 0, 0, 0] + [N] * bs
    kt, vt = k[:, 5:].transpose(1, 2), v[:, 5:].transpose(1, 2)                       # [bs,H,P,128]
    win = list(range(P)) if N == 0 else list(range(sink)) + list(range(P - local, P))
    cb, w, pk = oracle.encode(kt.contiguous(), cache.srht_diagonal_signs.cpu())       # [bs,H,16,P(,4)]
    assert torch.equal(cache.unified_keys_gpu[0][:, :, :n_win].cpu(), kt[:, :, win])
    assert torch.equal(cache.unified_values_gpu[0][:, :, :n_win].cpu(), vt[:, :, win])
    assert torch.equal(cache._win_codes[0][:, :, :n_win].cpu().permute(0, 1, 3, 2), cb[..., win])
    assert torch.equal(bits_of(cache._win_weight[0][:, :, :n_win].cpu().permute(0, 1, 3, 2)), bits_of(w[..., win]))
    assert torch.equal(cache._win_4bit[0][:, :, :n_win].cpu().permute(0, 1, 3, 2, 4), pk[..., win, :])
    norm = vt.float().norm(dim=-1)
    assert torch.allclose(cache._win_vnorm[0][:, :, :n_win].cpu(), norm[:, :, win], rtol=1e-5)
    zone = slice(sink, sink + N)
    assert torch.equal(cache.codebook_gpu[0][..., :N].cpu(), cb[..., zone])
    assert torch.equal(bits_of(cache.key_block_weight_gpu[0][..., :N].cpu()), bits_of(w[..., zone]))
    assert torch.equal(cache.key_4bit_packed_gpu[0][..., :N, :].cpu(), pk[..., zone, :])
    assert torch.allclose(cache.value_norm_gpu[0][..., :N].cpu(), norm[..., zone], rtol=1e-5)
    assert torch.equal(cache._store_k[0][:, :, :N].cpu(), kt[:, :, zone])
    assert torch.equal(cache._store_v[0][:, :, :N].cpu(), vt[:, :, zone])
    counts = oracle.cluster_counts(cb[..., zone].contiguous()) if N else torch.zeros(bs, H, 16, 256, dtype=torch.int32)
    assert torch.equal(cache.cluster_key_counts_gpu[0].cpu(), counts)


def test_short_prompts_on_several_streams_share_no_buffer():
    """Prompts whose rows are copied on the caller's own stream: another stream may fill the next layer at the same time, so
    their staging rows come from the allocator, not from the cache's pair of buffers."""
    from pariskv_b200.cache_hub.polar_cache import polar_cache
    n, H, layers = 600, 2, 4
    cache = polar_cache(valid_start=0, layer_num=layers, batch_size=1, max_length=n + 64, num_key_value_heads=H, num_heads=4 * H,
                        head_dim=128, dtype=torch.bfloat16, layer_mapping={str(i): DEV for i in range(layers)}, max_new_length=64,
                        sink_size=4, local_size=16, final_topk=64, dynamic_update_interval=32, enable_offload=True)
    g = torch.Generator(device=DEV).manual_seed(1)
    kv = [[torch.randn(1, n, H, 128, generator=g, device=DEV).to(torch.bfloat16) for _ in range(2)] for _ in range(layers)]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    for l in range(layers):
        with torch.cuda.stream(streams[l & 1]):
            cache.prefill_update_kv_cache(None, kv[l][0], kv[l][1], l, 0)
    torch.cuda.synchronize()
    assert all(buf is None for buf, _ in cache._staging)
    for l in range(layers):
        for rows, store in zip(kv[l], (cache.unified_keys_cpu[l], cache.unified_values_cpu[l])):
            assert torch.equal(store[0, :, :n - 20], rows[0, 4:n - 16].transpose(0, 1).cpu())


def _prompt(g, layout, bs, P, H):
    """[bs,P,H,128] with the given order in memory: tokens outermost, heads outermost, one head's rows for all heads, or K
    one way and V the other."""
    def rows(kind):
        if kind == "heads":
            return torch.randn(bs, H, P, 128, generator=g).to(torch.bfloat16).to(DEV).transpose(1, 2)
        if kind == "expanded":
            return torch.randn(bs, P, 1, 128, generator=g).to(torch.bfloat16).to(DEV).expand(bs, P, H, 128)
        if kind == "slice":     # the K or V columns of a wider row, whose first column lies 16 bytes into it
            wide = torch.randn(bs, P, (H + 1) * 128 + 8, generator=g).to(torch.bfloat16).to(DEV)
            return wide[..., 8:8 + H * 128].unflatten(-1, (H, 128))
        return torch.randn(bs, P, H, 128, generator=g).to(torch.bfloat16).to(DEV)
    return [rows(kind) for kind in (("tokens", "heads") if layout == "mixed" else (layout, layout))]


# Row by row (up to 16384 keys): zone rows around the edges of a tile of 96, windows of one tile and of two.  By TMA: the same edges,
# one tile per block and several (both stages in turn), every layout; K and V in different orders and expanded heads go row by row.
@pytest.mark.parametrize("P,H,local,layout", [
    (115, 3, 16, "tokens"), (116, 3, 16, "heads"), (117, 3, 16, "mixed"), (211, 2, 16, "slice"), (213, 2, 16, "expanded"),
    (228, 1, 128, "tokens"), (95, 2, 91, "tokens"), (96, 2, 91, "tokens"), (2048 + 20, 8, 16, "tokens"),
    (2049 + 20, 8, 16, "tokens"), (8255 + 20, 8, 16, "heads"), (8256 + 20, 8, 16, "slice"), (8257 + 20, 8, 16, "tokens"),
    (9001, 8, 64, "expanded"), (9000, 8, 300, "mixed"), (90001, 1, 64, "slice"), (13900, 5, 100, "heads"), (40000, 2, 128, "tokens")])
def test_prefill_tiles_match_oracle(oracle, P, H, local, layout):
    from pariskv_b200.cache_hub.polar_cache_adaptivek_varlen import polar_cache
    sink, bs = 4, 1
    g = torch.Generator().manual_seed(P)
    k, v = _prompt(g, layout, bs, P, H)
    cache = polar_cache(valid_start=0, layer_num=1, batch_size=bs, max_length=P + 32, num_key_value_heads=H, num_heads=H, head_dim=128,
                        dtype=torch.bfloat16, layer_mapping={"0": DEV}, max_new_length=32, sink_size=sink, local_size=local,
                        final_topk=16, dynamic_update_interval=8, enable_offload=False)
    cache.prefill_update_kv_cache(None, k, v, 0, 0)
    cache.check_status()
    N = max(0, P - sink - local)
    kt, vt = k.transpose(1, 2).cpu(), v.transpose(1, 2).cpu()
    win = list(range(P)) if N == 0 else list(range(sink)) + list(range(P - local, P))
    cb, w, pk = oracle.encode(kt.contiguous(), cache.srht_diagonal_signs.cpu())
    n, zone, norm = len(win), slice(sink, sink + N), vt.float().norm(dim=-1)
    for got, want in [(cache.unified_keys_gpu[0][:, :, :n], kt[:, :, win]), (cache.unified_values_gpu[0][:, :, :n], vt[:, :, win]),
                      (cache._win_codes[0][:, :, :n].permute(0, 1, 3, 2), cb[..., win]),
                      (cache._win_4bit[0][:, :, :n].permute(0, 1, 3, 2, 4), pk[..., win, :]),
                      (cache.codebook_gpu[0][..., :N], cb[..., zone]), (cache.key_4bit_packed_gpu[0][..., :N, :], pk[..., zone, :]),
                      (cache._store_k[0][:, :, :N], kt[:, :, zone]), (cache._store_v[0][:, :, :N], vt[:, :, zone])]:
        assert torch.equal(got.cpu(), want)
    assert torch.equal(bits_of(cache._win_weight[0][:, :, :n].cpu().permute(0, 1, 3, 2)), bits_of(w[..., win]))
    assert torch.equal(bits_of(cache.key_block_weight_gpu[0][..., :N].cpu()), bits_of(w[..., zone]))
    # sums of 128 squares in fp32, whatever the order: at most 127 roundings of 2^-24 each in the sum, half of it in the root
    assert torch.allclose(cache._win_vnorm[0][:, :, :n].cpu(), norm[:, :, win], rtol=1e-5)
    assert torch.allclose(cache.value_norm_gpu[0][..., :N].cpu(), norm[..., zone], rtol=1e-5)
    counts = oracle.cluster_counts(cb[..., zone].contiguous()) if N else torch.zeros(bs, H, 16, 256, dtype=torch.int32)
    assert torch.equal(cache.cluster_key_counts_gpu[0].cpu(), counts)
    if N:   # rows behind the zone's end are untouched
        assert not cache._store_kv[0][:, :, N:].any() and not cache.codebook_gpu[0][..., N:].any()


@pytest.mark.parametrize("P", [700, 12000])    # row by row; by TMA
@pytest.mark.parametrize("empty", [False, True])
def test_report_of_one_sample_outlives_the_next(P, empty):
    """All samples of a layer share one error word: the host sets it, as sample 0 would, and sample 1 leaves it alone, a sample
    without tokens too.  A new prompt for sample 0 starts clean."""
    from pariskv_b200.cache_hub.polar_cache import polar_cache
    g = torch.Generator().manual_seed(P)
    k, v = _prompt(g, "tokens", 1, P, 2)
    cache = polar_cache(valid_start=0, layer_num=2, batch_size=2, max_length=P + 32, num_key_value_heads=2, num_heads=2, head_dim=128,
                        dtype=torch.bfloat16, layer_mapping={"0": DEV, "1": DEV}, max_new_length=32, sink_size=4, local_size=16,
                        final_topk=16, dynamic_update_interval=8, enable_offload=False)
    cache._prefill_sample(k[0], v[0], 1, 0, 0)
    cache.check_status()
    cache._layer_state[1][3] = 1
    cache._prefill_sample(k[0], v[0], 1, 1, P if empty else 0)
    with pytest.raises(RuntimeError, match=r"layers \[1\]"):
        cache.check_status()
    cache._prefill_sample(k[0], v[0], 1, 0, P if empty else 0)
    cache.check_status()
    cache._prefill_sample(k[0], v[0], 1, 1, 0)
    cache.check_status()


# On both sides of the line between the two forms, and of the widths around it: 148 SMs x 4/3 = 198 blocks; one tile a block (25
# tiles x 8 heads = 200 blocks by TMA, 24 x 8 = 192 row by row), two (4000 x 8: 168 row by row, 5000 x 8: 216 by TMA), three.
@pytest.mark.parametrize("P,H", [(2300, 8), (2400, 8), (4000, 8), (5000, 8), (12300, 2), (24000, 1), (32768, 1)])
@pytest.mark.parametrize("cls,offload,record", [("topk", True, 128), ("topk", False, 96), ("adaptive", True, 96), ("adaptive", False, 128)])
def test_prompts_of_a_batch_match_oracle(oracle, P, H, cls, offload, record):
    """Two samples of different valid_start, prefilled twice into the same cache: the bases of sample 1, a prompt that starts inside
    its tensor, the staging rows behind the stores of the launch before, no value norms, both sizes of a key record."""
    from pariskv_b200.cache_hub import polar_cache_adaptivek_varlen
    from pariskv_b200.cache_hub.polar_cache import polar_cache
    make = polar_cache if cls == "topk" else polar_cache_adaptivek_varlen.polar_cache
    sink, local, starts, g = 4, 64, [3, 90], torch.Generator().manual_seed(P + H)
    cache = make(valid_start=starts, layer_num=1, batch_size=2, max_length=P + 32, num_key_value_heads=H, num_heads=H, head_dim=128,
                 dtype=torch.bfloat16, layer_mapping={"0": DEV}, max_new_length=32, sink_size=sink, local_size=local, final_topk=16,
                 dynamic_update_interval=8, enable_offload=offload, key_record_bytes=record)
    for _ in range(2):
        k, v = _prompt(g, "tokens", 2, P, H)
        cache.prefill_update_kv_cache(None, k, v, 0, 0)
    cache.sync(0, 0)
    torch.cuda.synchronize()
    cache.check_status()
    for b in range(2):
        kt, vt = k[b:b + 1, starts[b]:].transpose(1, 2).cpu(), v[b:b + 1, starts[b]:].transpose(1, 2).cpu()
        n = kt.shape[2]
        N, one, zone = n - sink - local, slice(b, b + 1), slice(sink, n - local)
        win = list(range(sink)) + list(range(n - local, n))
        cb, w, pk = oracle.encode(kt.contiguous(), cache.srht_diagonal_signs.cpu())
        w_n = sink + local
        assert cache._layer_state[0].tolist()[:4] == [w_n, 0, 0, 0] and int(cache._layer_state[0][4 + b]) == N
        for got, want in [(cache.unified_keys_gpu[0][one, :, :w_n], kt[:, :, win]), (cache.unified_values_gpu[0][one, :, :w_n], vt[:, :, win]),
                          (cache._win_codes[0][one, :, :w_n].permute(0, 1, 3, 2), cb[..., win]),
                          (cache._win_4bit[0][one, :, :w_n].permute(0, 1, 3, 2, 4), pk[..., win, :]),
                          (cache.codebook_gpu[0][one, ..., :N], cb[..., zone]), (cache.key_4bit_packed_gpu[0][one, ..., :N, :], pk[..., zone, :]),
                          (cache._store_k[0][one, :, :N], kt[:, :, zone]), (cache._store_v[0][one, :, :N], vt[:, :, zone])]:
            assert torch.equal(got.cpu(), want)
        assert torch.equal(bits_of(cache._win_weight[0][one, :, :w_n].cpu().permute(0, 1, 3, 2)), bits_of(w[..., win]))
        assert torch.equal(bits_of(cache.key_block_weight_gpu[0][one, ..., :N].cpu()), bits_of(w[..., zone]))
        # sums of 128 squares in fp32, as above
        norm = vt.float().norm(dim=-1)
        assert torch.allclose(cache._win_vnorm[0][one, :, :w_n].cpu(), norm[:, :, win], rtol=1e-5)
        if cls == "adaptive":
            assert torch.allclose(cache.value_norm_gpu[0][one, ..., :N].cpu(), norm[..., zone], rtol=1e-5)
        assert torch.equal(cache.cluster_key_counts_gpu[0][one].cpu(), oracle.cluster_counts(cb[..., zone].contiguous()))
