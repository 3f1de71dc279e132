"""DeepSeek-V4 sparse_flash_mla front door (window + compressed tokens + sinks) on the GPU against the oracle."""
import importlib

import numpy as np
import pytest
import torch

from gpu_util import assert_close_fp, check_status
from oracle import dsa_oracle as orc

pytestmark = pytest.mark.gpu


def _paged(dense: torch.Tensor, block_size: int, rng) -> tuple:
    """[B, S, D] -> (pool [blocks, block_size, 1, D] with the sequences' blocks shuffled, block table [B, n])."""
    B, S, D = dense.shape
    n = (S + block_size - 1) // block_size
    perm = rng.permutation(B * n + 2)[: B * n]          # two blocks of the pool stay unused
    pool = torch.zeros((B * n + 2, block_size, 1, D), dtype=dense.dtype)
    table = torch.from_numpy(perm.reshape(B, n).astype(np.int32))
    for b in range(B):
        for j in range(n):
            chunk = dense[b, j * block_size:(j + 1) * block_size]
            pool[int(table[b, j]), : chunk.shape[0], 0] = chunk
    return pool, table


def _case(seed, B, S, S_kv, N1, D, K, ratio, act_q, act_kv):
    g = torch.Generator().manual_seed(seed)
    q = torch.randn((B, S, N1, D), generator=g).to(torch.bfloat16)
    k = torch.randn((B, S_kv, D), generator=g).to(torch.bfloat16)
    c = torch.randn((B, S_kv // ratio, D), generator=g).to(torch.bfloat16)
    sinks = torch.randn((N1,), generator=g)
    rng = np.random.default_rng(seed)
    ci = np.full((B, S, 1, K), -1, dtype=np.int32)
    for b in range(B):
        for s in range(act_q[b]):
            n = int(rng.integers(0, K + 1))
            ci[b, s, 0, :n] = rng.choice(S_kv // ratio, size=n, replace=False) if n <= S_kv // ratio else rng.integers(0, S_kv // ratio, size=n)
    return q, k, c, sinks, torch.from_numpy(ci), rng


@pytest.mark.parametrize("scenario", [1, 2, 3])
@pytest.mark.parametrize("layout", ["TND", "BSND"])
def test_sparse_flash_mla_matches_oracle(scenario, layout):
    import tilelang_ascend_b200 as dsa
    B, S, S_kv, N1, D, K, ratio, win = 2, 9, 300, 64, 512, 32, 4, 127
    act_q, act_kv = [9, 5], [300, 171]
    q, k, c, sinks, ci, rng = _case(scenario, B, S, S_kv, N1, D, K, ratio, act_q, act_kv)
    scale = D ** -0.5
    kw = {}
    if scenario >= 2:
        kw.update(cmp_k=c, cmp_ratio=ratio)
    if scenario == 3:
        kw.update(cmp_sparse_indices=ci[:, :, 0, :])
    ref_out, ref_lse = orc.sparse_flash_mla_v4(q, k, sinks, act_q_lens=act_q, act_kv_lens=act_kv, softmax_scale=scale, ori_win_left=win, **kw)

    ori_pool, ori_bt = _paged(k, 128, rng)
    cmp_pool, cmp_bt = _paged(c, 16, rng)
    cu = torch.tensor([0, act_q[0], act_q[0] + act_q[1]], dtype=torch.int32)
    args = dict(ori_kv=ori_pool.cuda(), ori_block_table=ori_bt.cuda(), seqused_kv=torch.tensor(act_kv, dtype=torch.int32).cuda(), sinks=sinks.cuda(),
                softmax_scale=scale, ori_win_left=win, layout_q=layout, return_softmax_lse=True, cu_seqlens_q=cu.cuda())
    if scenario >= 2:
        args.update(cmp_kv=cmp_pool.cuda(), cmp_block_table=cmp_bt.cuda(), cmp_ratio=ratio)
    if layout == "TND":
        q_in = torch.cat([q[b, : act_q[b]] for b in range(B)]).cuda()
        if scenario == 3:
            args.update(cmp_sparse_indices=torch.cat([ci[b, : act_q[b]] for b in range(B)]).cuda())
        out, lse = dsa.sparse_flash_mla(q_in, **args)
        check_status()
        ref_o = torch.cat([ref_out[b, : act_q[b]] for b in range(B)])
        ref_l = torch.cat([ref_lse[b, : act_q[b]] for b in range(B)])
    else:
        if scenario == 3:
            args.update(cmp_sparse_indices=ci.cuda())
        out, lse = dsa.sparse_flash_mla(q.cuda(), **args)
        check_status()
        ref_o, ref_l = ref_out, ref_lse       # rows beyond a sequence's length are zero on both sides
    assert_close_fp(out.cpu(), ref_o, f"out, scenario {scenario} {layout}")
    assert_close_fp(lse.cpu(), ref_l, f"lse, scenario {scenario} {layout}")


def test_sink_combine_single_partial_without_sink_is_identity():
    import tilelang_ascend_b200 as dsa
    g = torch.Generator().manual_seed(0)
    out = torch.randn((5, 8, 64), generator=g).to(torch.bfloat16).cuda()
    lse = torch.randn((5, 8), generator=g).cuda()
    o2, l2 = dsa.sink_combine_raw(out, lse, None, None, None, 8)
    assert torch.equal(o2, out) and torch.allclose(l2, lse, rtol=1e-6, atol=1e-6)


@pytest.mark.parametrize("H,win,K,T", [(64, 127, 512, 3), (64, 0, 64, 200), (100, 63, 96, 9), (160, 127, 0, 5), (16, 127, 512, 40)])
def test_joined_lists_match_two_passes(H, win, K, T, monkeypatch):
    """One pass over the window and the compressed keys against the two-pass route it replaces: short and long calls (shares of a
    split unit and whole units), several head blocks, tokens without any key, a sink far above and far below the scores, table
    entries outside the pools.  The two routes round at different places: each is within 2^-8 of the exact row (bf16), so the
    relative 2-norm of their difference is below 2^-7."""
    import tilelang_ascend_b200 as dsa
    mod = importlib.import_module("tilelang_ascend_b200.sparse_flash_mla")   # (the package re-exports the function by that name)
    g = torch.Generator().manual_seed(H + K)
    n_kv, ratio = 4000, 4
    q = torch.randn((T, H, 512), generator=g).to(torch.bfloat16).cuda()
    pool = torch.randn((32, 128, 1, 512), generator=g).to(torch.bfloat16).cuda()
    cpool = torch.randn((70, 16, 1, 512), generator=g).to(torch.bfloat16).cuda()
    bt = torch.randperm(32, generator=g).to(torch.int32)[None]
    cbt = torch.randperm(70, generator=g).to(torch.int32)[None]
    cbt[0, 3], cbt[0, 5] = -1, 70            # padding / beyond the pool: those keys take no part
    sinks = torch.randn((H,), generator=g)
    sinks[0], sinks[1] = 300.0, -300.0
    kw = dict(ori_kv=pool, ori_block_table=bt.cuda(), cu_seqlens_q=torch.tensor([0, T], dtype=torch.int32).cuda(), sinks=sinks.cuda(),
              seqused_kv=torch.tensor([n_kv if T < 100 else T - 2], dtype=torch.int32).cuda(), softmax_scale=512 ** -0.5, ori_win_left=win,
              return_softmax_lse=True)
    if K:
        ci = torch.randint(0, n_kv // ratio, (T, 1, K), generator=g).sort(dim=-1).values.to(torch.int32)
        ci[0] = -1
        kw.update(cmp_kv=cpool, cmp_block_table=cbt.cuda(), cmp_ratio=ratio, cmp_sparse_indices=ci.cuda())
    out, lse = dsa.sparse_flash_mla(q, **kw)
    monkeypatch.setattr(mod, "_JOINED_MAX_KEYS", 0)
    ref, ref_lse = dsa.sparse_flash_mla(q, **kw)
    check_status()
    assert torch.isfinite(lse).all() and torch.isfinite(out.float()).all()
    assert ((out.float() - ref.float()).norm() / ref.float().norm()).item() < 2 ** -7
    # the parts' log-sum-exps are fp32 sums of at most 640 bf16-weighted terms; merged with fast logarithms
    assert (lse - ref_lse).abs().max().item() < 2e-3
