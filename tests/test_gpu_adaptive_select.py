"""The adaptive selection kernel at the edges of its paths: one candidate, thread and register-batch remainders, lists that do
not fit in shared memory, equal benefits, benefits of zero, benefits over very many octaves."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def ops():
    from pariskv_b200 import ops
    return ops


@pytest.mark.parametrize("C,K_out", [(1, 1), (33, 7), (1025, 1024), (8192, 4096), (8193, 4096), (33000, 4096)])
@pytest.mark.parametrize("kind", ["plain", "equal", "few", "zeros", "octaves"])
def test_selection_equals_the_oracle(ops, oracle, C, K_out, kind):
    g = torch.Generator().manual_seed(C + K_out)
    bs, H, S = 1, 3, 77
    cl = torch.randn(bs, H, C, generator=g)
    if kind == "equal":
        cl[:] = 0.5
    elif kind == "few":        # a handful of distinct benefits: buckets of hundreds
        cl = torch.randint(0, 5, (bs, H, C), generator=g).float()
    elif kind == "zeros":      # most candidates carry no weight: the lowest positions fill the selection
        cl[torch.rand(bs, H, C, generator=g) < 0.8] = float("-inf")
    elif kind == "octaves":
        cl *= 25.0
    sl, slv = torch.randn(bs, H, S, generator=g), torch.rand(bs, H, S, generator=g)
    cv = torch.ones(bs, H, C) if kind in ("equal", "few") else torch.rand(bs, H, C, generator=g) + 0.1
    ci = torch.stack([torch.randperm(C + 9, generator=g)[:C] for _ in range(H)])[None]
    k_o, idx_o = oracle.adaptive_topk(sl, slv, cl, cv, ci, 0.9, K_out)
    k, idx = ops.adaptive_topk(sl.to(DEV), cl.to(DEV), 1.0, slv.to(DEV), ci.to(DEV), cv.to(DEV), 0.9, K_out)
    assert torch.equal(k.cpu(), k_o) and torch.equal(idx.cpu(), idx_o)


@pytest.mark.parametrize("S,filled", [(5, 5), (130, 68), (300, 299)])
def test_window_logits_and_caps(oracle, S, filled):
    from pariskv_b200 import _lib
    g = torch.Generator().manual_seed(S)
    bs, H, C, K_out, scale = 2, 3, 700, 256, 0.088
    q = torch.randn(bs, H, 128, generator=g).to(torch.bfloat16)
    wk = torch.randn(bs, H, S + 3, 128, generator=g).to(torch.bfloat16)
    cs, cap = torch.randn(bs, H, C, generator=g) * 9, torch.randint(1, K_out, (bs, H), generator=g, dtype=torch.int32)
    slv, vn = torch.rand(bs, H, S, generator=g), torch.rand(bs, H, C + 50, generator=g)
    ci = torch.stack([torch.stack([torch.randperm(C + 50, generator=g)[:C] for _ in range(H)]) for _ in range(bs)])
    args = [t.to(DEV) for t in (q, wk, torch.tensor([filled], dtype=torch.int32), cs, cap, slv, ci, vn)]
    ak, idx, n_sel, sl = _lib.native().adaptive_select(args[0], args[1], args[2], S, args[3], args[4], scale, args[5], args[6],
                                                       args[7], 0.9, K_out, 1, K_out)
    want = torch.einsum("bhd,bhkd->bhk", q.float(), wk[:, :, :S].float()) * scale
    assert torch.isinf(sl[:, :, filled:]).all()
    assert (sl.cpu() - want)[:, :, :filled].abs().max() <= 2.0 ** -8 * want.abs().max()
    cl = cs.to(torch.bfloat16).float() * torch.tensor(scale, dtype=torch.float32)
    k_o, idx_o = oracle.adaptive_topk(sl.cpu(), slv, cl, torch.gather(vn, 2, ci), ci, 0.9, K_out)
    assert torch.equal(idx.cpu(), idx_o)
    assert torch.equal(ak.cpu(), torch.minimum(k_o, cap.long())) and torch.equal(n_sel.cpu().long(), ak.cpu())
