"""Performance cases of the DeepSeek-sparse-attention path: what a serving or training program has this package do, through
its public entry points.

Kinds (each is one public call, or one forward + backward):

* ``select``         stand-alone top-k selector (``simple_topk_selector``) on fp32 score rows
* ``index_prefill``  lightning indexer of a prompt chunk, dense keys, causal (``lightning_indexer``, BSND)
* ``index_decode``   lightning indexer of decode tokens against a paged key cache (``lightning_indexer``, PA_BSND)
* ``prefill``        sparse MLA forward of a prompt chunk on causal index lists (``sparse_attention_fwd``)
* ``decode``         sparse MLA forward of decode tokens against a paged latent cache (``sparse_attn_tilelang``)
* ``dense_decode``   dense MLA decode, every key of the cache (``mla_decode``)
* ``v4``             DeepSeek-V4 window + compressed-token attention with sinks (``sparse_flash_mla``), prefill and decode
* ``hisa``           block-sparse indexer logits of a long context (``block_sparse_mqa_attn_return_logits``)
* ``train``          differentiable sparse MLA, forward and backward (``sparse_mla`` + autograd)

Tensors are seeded N(0, 1) (weights scaled as an averaging over heads); index lists are distinct and causal, cache blocks are
shuffled, sequence lengths of a batch are ragged.
"""
import torch

import tilelang_ascend_b200 as dsa

_DT = {"bf16": torch.bfloat16, "fp16": torch.float16}
_DV, _ROPE = 512, 64
_D = _DV + _ROPE
_BLOCK = 128        # keys per block of the paged caches and of the block-sparse logits


def listed():
    return [
        # the selector on its own at the size of the reference example's test: a few dozen short rows, latency bound
        dict(name="select_64x4096", kind="select", rows=64, n=4096, topk=2048),
        # scores + top-2048 of a 4096-token prompt chunk against 8192 keys (one layer's indexer in prefill)
        dict(name="index_prefill_4096x8192", kind="index_prefill", B=1, S=4096, S_kv=8192, H=64, topk=2048, dtype="bf16"),
        # one decode step's indexer: 32 sequences, ragged caches of up to 48 K keys in shuffled blocks
        dict(name="index_decode_32x49152", kind="index_decode", B=32, S=1, S_kv=49152, H=64, topk=2048, dtype="bf16"),
        # the headline prefill: 4096 queries, 128 heads, top-2048
        dict(name="prefill_4096", kind="prefill", B=1, S=4096, S_kv=4096, H=128, topk=2048, dtype="bf16"),
        # a ragged chunk of two prompts on a tensor-parallel half of the heads, fp16, shorter lists
        dict(name="prefill_2x777_h64_fp16", kind="prefill", B=2, S=777, S_kv=2501, H=64, topk=1024, dtype="fp16"),
        # decode step of a full batch and of a nearly empty one
        dict(name="decode_64", kind="decode", B=64, S=1, S_kv=32768, H=128, topk=2048, dtype="bf16"),
        dict(name="decode_4", kind="decode", B=4, S=1, S_kv=20000, H=128, topk=2048, dtype="bf16"),
        # dense MLA decode at the largest shape of the reference's layered test
        dict(name="dense_decode_132x8192", kind="dense_decode", B=132, S_kv=8192, H=128, dtype="fp16"),
        # V4 layers: prefill of an 8192-token prompt and a decode step of 16 sequences, window 128 + 512 compressed tokens
        dict(name="v4_prefill_8192", kind="v4", mode="csa", B=1, S=8192, S_kv=8192, H=64, topk=512, dtype="bf16"),
        dict(name="v4_decode_16", kind="v4", mode="csa", B=16, S=1, S_kv=8193, H=64, topk=512, dtype="bf16"),
        # block-sparse logits of the last 1024 queries of a 128 K context, 64 selected blocks each
        dict(name="hisa_1024x131072", kind="hisa", S=1024, S_kv=131072, H=32, topk=64, dtype="fp16"),
        # one training step's attention: forward and backward at the prefill shape
        dict(name="train_4096", kind="train", S=4096, S_kv=4096, H=128, topk=2048, dtype="bf16"),
    ]


def _log(rng, lo, hi):
    """A whole number spread over the logarithm of [lo, hi]; odd ones as likely as even ones."""
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["select", "index_prefill", "index_decode", "prefill", "decode", "dense_decode", "v4", "hisa", "train"])
    dtype = rng.choice(["bf16", "fp16"])
    if kind == "select":
        n = _log(rng, 512, 131072)
        return dict(kind=kind, rows=_log(rng, 1, min(4096, (1 << 25) // n)), n=n, topk=min(n, rng.choice([128, 512, 1024, 2048])))
    if kind == "index_prefill":
        S = _log(rng, 128, 4096)
        return dict(kind=kind, B=rng.choice([1, 1, 2]), S=S, S_kv=_log(rng, S, 8192), H=rng.choice([16, 32, 64, 64]), topk=rng.choice([512, 1024, 2048]),
                    dtype=dtype)
    if kind == "index_decode":
        return dict(kind=kind, B=_log(rng, 1, 64), S=rng.choice([1, 1, 2]), S_kv=_log(rng, 3000, 65536), H=rng.choice([32, 64, 64]),
                    topk=rng.choice([1024, 2048]), dtype=dtype)
    if kind == "prefill":
        S = _log(rng, 64, 4096)
        return dict(kind=kind, B=rng.choice([1, 1, 2]), S=S, S_kv=_log(rng, S, 8192), H=rng.choice([32, 64, 128, 128]), topk=rng.choice([512, 1024, 2048]),
                    dtype=dtype)
    if kind == "decode":
        return dict(kind=kind, B=_log(rng, 1, 128), S=rng.choice([1, 1, 2]), S_kv=_log(rng, 2500, 32768), H=rng.choice([32, 64, 128, 128]),
                    topk=rng.choice([1024, 2048]), dtype=dtype)
    if kind == "dense_decode":
        return dict(kind=kind, B=_log(rng, 1, 132), S_kv=_log(rng, 500, 8192), H=rng.choice([64, 128]), dtype=dtype)
    if kind == "v4":
        mode = rng.choice(["swa", "hca", "csa", "csa"])
        if rng.random() < 0.5:
            S = _log(rng, 256, 8192)
            return dict(kind=kind, mode=mode, B=1, S=S, S_kv=_log(rng, S, 16384), H=64, topk=512, dtype=dtype)
        return dict(kind=kind, mode=mode, B=_log(rng, 1, 64), S=rng.choice([1, 1, 2]), S_kv=_log(rng, 4000, 32768), H=64, topk=512, dtype=dtype)
    if kind == "hisa":
        return dict(kind=kind, S=_log(rng, 64, 1024), S_kv=_log(rng, 16384, 131072), H=rng.choice([32, 64]), topk=rng.choice([16, 32, 64]), dtype=dtype)
    S = _log(rng, 128, 3000)
    return dict(kind=kind, S=S, S_kv=_log(rng, S, 4096), H=rng.choice([64, 128]), topk=rng.choice([512, 1024, 2048]), dtype=dtype)


# ----------------------------------------------------------------------------------------------------------- inputs
def _causal_lists(g, S, S_kv, topk, dev, limits=None):
    """[S, topk] int32: distinct keys in random order below each query's limit, -1 behind them."""
    if limits is None:
        limits = torch.arange(S, device=dev) + (S_kv - S + 1)
    keys = torch.rand((S, S_kv), generator=g, device=dev)
    keys = torch.where(torch.arange(S_kv, device=dev)[None, :] < limits[:, None], keys, torch.full_like(keys, -1.0))
    k = min(topk, S_kv)
    val, idx = keys.topk(k, dim=1)
    idx = torch.where(val < 0, torch.full_like(idx, -1), idx).to(torch.int32)
    if k < topk:
        idx = torch.cat((idx, torch.full((S, topk - k), -1, dtype=torch.int32, device=dev)), dim=1)
    return idx.contiguous()


def _lengths(g, B, S, S_kv, dev):
    """Ragged sequence lengths in [S_kv / 2, S_kv], the first one S_kv."""
    n = (S_kv * (0.5 + 0.5 * torch.rand((B,), generator=g, device=dev))).to(torch.int32).clamp(min=S, max=S_kv)
    n[0] = S_kv
    return n


def _block_table(g, B, S_kv, dev):
    nb = -(-S_kv // _BLOCK)
    return torch.randperm(B * nb, generator=g, device=dev).to(torch.int32).view(B, nb).contiguous()


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    g = torch.Generator(device=dev).manual_seed(int(seed))
    c = dict(case)
    kind = c["kind"]
    dt = _DT[c.get("dtype", "bf16")]

    def randn(*shape, dtype=dt):
        return torch.randn(shape, generator=g, device=dev, dtype=dtype)

    if kind == "select":
        return dict(kind=kind, x=randn(c["rows"], c["n"], dtype=torch.float32), kernel=dsa.simple_topk_selector(c["rows"], c["n"], c["topk"], 512))
    if kind in ("index_prefill", "index_decode"):
        B, S, S_kv, H = c["B"], c["S"], c["S_kv"], c["H"]
        w = randn(B, S, H, dtype=torch.float32).abs() / H
        s = dict(kind=kind, q=randn(B, S, H, 128), w=w, topk=c["topk"])
        if kind == "index_prefill":
            s.update(k=randn(B, S_kv, 1, 128))
        else:
            bt = _block_table(g, B, S_kv, dev)
            s.update(k=randn(bt.numel(), _BLOCK, 1, 128), bt=bt, aq=torch.full((B,), S, dtype=torch.int32, device=dev), ak=_lengths(g, B, S, S_kv, dev))
        return s
    if kind in ("prefill", "train"):
        B, S, S_kv, H, topk = c.get("B", 1), c["S"], c["S_kv"], c["H"], c["topk"]
        idx = torch.stack([_causal_lists(g, S, S_kv, topk, dev) for _ in range(B)]).view(B, S, 1, topk)
        s = dict(kind=kind, q=randn(B, S, H, _D), kv=randn(B, S_kv, 1, _D), idx=idx)
        if kind == "prefill":
            s["kernel"] = dsa.sparse_attention_fwd(H, _DV, _ROPE, topk, 1, dtype="bfloat16" if dt == torch.bfloat16 else "float16", return_softmax_lse=True)
        else:
            s["q"].requires_grad_(True)
            s["kv"].requires_grad_(True)
            s["d_out"] = randn(B, S, H, _DV)
        return s
    if kind == "decode":
        B, S, S_kv, H, topk = c["B"], c["S"], c["S_kv"], c["H"], c["topk"]
        ak = _lengths(g, B, S, S_kv, dev)
        limits = (ak[:, None] - S + 1 + torch.arange(S, device=dev)[None, :]).reshape(B * S)
        bt = _block_table(g, B, S_kv, dev)
        return dict(kind=kind, q=randn(B, S, H, _DV), q_rope=randn(B, S, H, _ROPE), k=randn(bt.numel(), _BLOCK, 1, _DV), k_rope=randn(bt.numel(), _BLOCK, 1, _ROPE),
                    idx=_causal_lists(g, B * S, S_kv, topk, dev, limits).view(B, S, 1, topk), bt=bt, ak=ak,
                    aq=torch.full((B,), S, dtype=torch.int32, device=dev))
    if kind == "dense_decode":
        B, N, H = c["B"], c["S_kv"], c["H"]
        return dict(kind=kind, q=randn(B, H, _DV), q_rope=randn(B, H, _ROPE), kv=randn(B, N, 1, _DV), k_rope=randn(B, N, 1, _ROPE),
                    kernel=dsa.mla_decode(B, H, 1, N, _DV, _ROPE))
    if kind == "v4":
        B, S, S_kv, H, K, mode = c["B"], c["S"], c["S_kv"], c["H"], c["topk"], c["mode"]
        ratio = 128 if mode == "hca" else 4
        used = _lengths(g, B, S, S_kv, dev)
        ori_bt, n_cmp = _block_table(g, B, S_kv, dev), max(S_kv // ratio, 1)
        kw = dict(ori_kv=randn(ori_bt.numel(), _BLOCK, 1, _DV), ori_block_table=ori_bt, cu_seqlens_q=torch.arange(B + 1, dtype=torch.int32, device=dev) * S,
                  seqused_kv=used, sinks=randn(H, dtype=torch.float32), softmax_scale=_DV ** -0.5, return_softmax_lse=True)
        if mode != "swa":
            cmp_bt = _block_table(g, B, n_cmp, dev)
            kw.update(cmp_kv=randn(cmp_bt.numel(), _BLOCK, 1, _DV), cmp_block_table=cmp_bt, cmp_ratio=ratio)
        if mode == "hca":
            kw.update(topk_cmp=n_cmp)      # the caller's upper bound of the compressed tokens of a sequence
        if mode == "csa":
            pos = (used[:, None] - S + torch.arange(S, device=dev)[None, :]).reshape(B * S)
            kw.update(cmp_sparse_indices=_causal_lists(g, B * S, n_cmp, K, dev, (pos + 1) // ratio).view(B * S, 1, K))
        return dict(kind=kind, q=randn(B * S, H, _DV), kw=kw)
    S, S_kv, H, topk = c["S"], c["S_kv"], c["H"], c["topk"]   # hisa
    ke = torch.arange(S, dtype=torch.int32, device=dev) + (S_kv - S + 1)
    blk = _causal_lists(g, S, -(-S_kv // _BLOCK), topk, dev, (ke + _BLOCK - 1) // _BLOCK)
    return dict(kind=kind, q=randn(S, H, 128), k=randn(S_kv, 128), w=(randn(S, H, dtype=torch.float32).abs() / H).to(dt), ks=torch.zeros_like(ke), ke=ke, blk=blk,
                kernel=dsa.block_sparse_mqa_attn_return_logits(S, S_kv, _BLOCK, topk, H, 128))


# -------------------------------------------------------------------------------------------------------- the calls
def run(s):
    kind = s["kind"]
    if kind == "select":
        return s["kernel"](s["x"])
    if kind == "index_prefill":
        return dsa.lightning_indexer(s["q"], s["k"], s["w"], sparse_count=s["topk"], sparse_mode=3)[0]
    if kind == "index_decode":
        return dsa.lightning_indexer(s["q"], s["k"], s["w"], actual_seq_lengths_query=s["aq"], actual_seq_lengths_key=s["ak"], block_table=s["bt"],
                                     layout_key="PA_BSND", sparse_count=s["topk"], sparse_mode=3)[0]
    if kind == "prefill":
        return s["kernel"](s["q"], s["kv"], s["idx"])
    if kind == "decode":
        return dsa.sparse_attn_tilelang(s["q"], s["k"], s["k"], s["idx"], _D ** -0.5, 1, s["aq"], s["ak"], query_rope=s["q_rope"], key_rope=s["k_rope"],
                                        layout_kv="PA_BSND", block_table=s["bt"], return_softmax_lse=True)
    if kind == "dense_decode":
        return s["kernel"](s["q"], s["q_rope"], s["kv"], s["k_rope"])
    if kind == "v4":
        return dsa.sparse_flash_mla(s["q"], **s["kw"])
    if kind == "hisa":
        return s["kernel"](s["q"], s["k"], s["blk"], s["w"], s["ks"], s["ke"])
    out, lse = dsa.sparse_mla(s["q"], s["kv"], s["idx"])
    d_q, d_kv = torch.autograd.grad(out, (s["q"], s["kv"]), s["d_out"])
    return dict(out=out.detach(), lse=lse.detach(), d_q=d_q, d_kv=d_kv)


# ------------------------------------------------------------------------------------------------- what a pass needs
def _causal_pairs(S, S_kv, topk):
    """Sum over queries of min(topk, candidates)."""
    return sum(min(topk, S_kv - S + 1 + t) for t in range(S))


def work(case):
    """Compulsory bytes (inputs read once, outputs written once; of a ragged batch three quarters of the longest length) and
    floating-point operations of the contractions."""
    c = dict(case)
    kind, H, topk = c["kind"], c.get("H", 0), c.get("topk", 0)
    if kind == "select":
        return dict(bytes=c["rows"] * (c["n"] + topk) * 4, flops=0)
    if kind == "index_prefill":
        B, S, S_kv = c["B"], c["S"], c["S_kv"]
        return dict(bytes=B * (S * H * 260 + S_kv * 256 + S * topk * 4), flops=B * _causal_pairs(S, S_kv, S_kv) * H * 256)
    if kind == "index_decode":
        B, S, n = c["B"], c["S"], 0.75 * c["S_kv"]
        return dict(bytes=B * (S * H * 260 + n * 256 + S * topk * 4), flops=B * S * n * H * 256)
    if kind == "prefill":
        B, S, S_kv = c["B"], c["S"], c["S_kv"]
        return dict(bytes=B * (S * (H * ((_D + _DV) * 2 + 4) + topk * 4) + S_kv * _D * 2), flops=B * _causal_pairs(S, S_kv, topk) * H * 2 * (_D + _DV))
    if kind == "train":
        S, S_kv = c["S"], c["S_kv"]
        pairs = _causal_pairs(S, S_kv, topk)
        # forward: S, O; backward: S again, dP, dQ and the two parts of dKV
        return dict(bytes=S * (H * (4 * _D + 5 * _DV) + topk * 4 + 4 * H) + S_kv * _D * 4, flops=pairs * H * 2 * (3 * _D + 2 * _DV + _D + _DV))
    if kind == "decode":
        B, S, n = c["B"], c["S"], min(topk, 0.75 * c["S_kv"])
        return dict(bytes=B * S * (n * _D * 2 + H * ((_D + _DV) * 2 + 4) + topk * 4), flops=B * S * n * H * 2 * (_D + _DV))
    if kind == "dense_decode":
        B, n = c["B"], c["S_kv"]
        return dict(bytes=B * (n * _D * 2 + H * (_D + _DV) * 2), flops=B * n * H * 2 * (_D + _DV))
    if kind == "v4":
        B, S, S_kv, mode = c["B"], c["S"], c["S_kv"], c["mode"]
        n = S_kv if B == 1 else 0.75 * S_kv
        pos = n - S / 2
        cmp_keys = {"swa": 0, "hca": pos / 128, "csa": min(topk, pos / 4)}[mode]
        pairs = B * S * (min(128, n) + cmp_keys)
        rows = B * min(n, S + 127) + B * min(n / (128 if mode == "hca" else 4), S * cmp_keys if cmp_keys else 0)
        return dict(bytes=B * S * (H * (2 * _DV * 2 + 4) + (topk * 4 if mode == "csa" else 0)) + rows * _DV * 2, flops=pairs * H * 4 * _DV)
    S, S_kv = c["S"], c["S_kv"]
    return dict(bytes=S * (H * 258 + topk * 4 + topk * _BLOCK * 4) + min(S_kv, S * topk * _BLOCK) * 256, flops=S * topk * _BLOCK * H * 256)


def tolerance(case):
    """About four times the distance of these paths from the same computation in 64 bits: indexer orders differ from the fp64
    order at 6e-4 of the places (neighbouring scores closer than fp32 sums resolve; the index sets agree), fp32 logits by 2e-7,
    attention outputs and gradients by 2.6e-3 (bf16) / 3.3e-4 (fp16), largest difference 1.6e-2 / 1.9e-3."""
    kind = case["kind"]
    if kind == "select":
        return "exact"
    if kind in ("index_prefill", "index_decode"):
        return {"rel": 1e-6, "differ": 0.0025}
    if kind == "hisa":
        return {"rel": 1e-6, "max": 1e-5}
    return {"rel": 1e-2, "max": 6e-2} if case["dtype"] == "bf16" else {"rel": 1.5e-3, "max": 8e-3}
