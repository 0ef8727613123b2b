"""What the performance of this framework is measured on: attention-layer steps of a serving engine through the plugin
surface (HorizonFp4Builder's metadata, HorizonFp4Impl.do_kv_cache_update, HorizonFp4Impl.forward) and the bulk cache
fill through kernels.write.

A "step" case is one layer of one engine step over a paged NVFP4 cache:

  n_dec, ctx_lo, ctx_hi   decode requests and their context lengths, log-uniform quantiles of [ctx_lo, ctx_hi]
  q_tokens                query tokens of a decode request (1, or 1 + draft tokens to verify)
  n_pre, new_lo, new_hi   prefill requests and their numbers of new tokens, log-uniform quantiles
  prior_lo, prior_hi      tokens already cached before those new ones (0: a fresh prompt; else a chunk of a long prompt
                          or a prefix-cache hit)
  head_dim, kv_heads, group, page, order, k8, had   the model's shape and the cache's options
  graph                   the step is captured once and replayed, as an engine does with uniform decode batches

A "write" case quantises n_tokens tokens into random slots (one launch of kernels.write).

Values: q and v ~ N(0, 1), k ~ N(0, 1) with four outlier channels per head scaled by 20, global scales amax / (6 * 448),
pages scattered at random over the pool. The context lengths follow from the case alone, everything else from the seed.
"""
import math
import os
from types import SimpleNamespace

import torch

os.environ.setdefault("HORIZON_KVFP4_STANDALONE", "1")       # the plugin classes without importing vLLM

from horizon_kernels_b200 import backend as BE  # noqa: E402
from horizon_kernels_b200 import kernels as K  # noqa: E402
from horizon_kernels_b200 import layout as Lt  # noqa: E402

OUTLIER = 20.0
GK = OUTLIER * 5.5 / (6 * 448)                                # amax / (6 * 448) at 5.5 sigma
GV = 5.5 / (6 * 448)
SHAPES = {"8b": dict(head_dim=128, kv_heads=8, group=4),     # Llama-3-8B-shaped: 32 query heads over 8 kv heads
          "70b": dict(head_dim=128, kv_heads=8, group=8),    # 70B-shaped: 64 query heads over 8 kv heads
          "hybrid": dict(head_dim=256, kv_heads=2, group=8),
          "dense256": dict(head_dim=256, kv_heads=4, group=6)}


def _step(name, shape, n_dec=0, ctx=(1, 1), q_tokens=1, n_pre=0, new=(1, 1), prior=(0, 0), page=16, order="LBHNC",
          k8=False, had=False, graph=False):
    c = dict(kind="step", n_dec=n_dec, ctx_lo=ctx[0], ctx_hi=ctx[1], q_tokens=q_tokens, n_pre=n_pre, new_lo=new[0],
             new_hi=new[1], prior_lo=prior[0], prior_hi=prior[1], page=page, order=order, k8=k8, had=had, graph=graph,
             **SHAPES[shape])
    return dict(c, name=name) if name else c


def _write(name, shape, n_tokens, page=16, search=True):
    c = dict(kind="write", n_tokens=n_tokens, page=page, search=search, **SHAPES[shape])
    return dict(c, name=name) if name else c


def listed():
    return [
        # a few users of one chat server between prompts: four requests, two thousand tokens each; launches and host
        # calls are most of it
        _step("decode_four", "8b", 4, (2048, 2048)),
        # a busy chat server's decode step, captured in a graph: 64 requests of 1k to 8k tokens
        _step("decode_batch", "8b", 64, (1024, 8192), graph=True),
        # long documents: eight requests of 131072 tokens
        _step("decode_long", "70b", 8, (131072, 131072)),
        # a large hybrid batch at head_dim 256, contexts from 128 to 32k tokens, captured in a graph
        _step("decode_hybrid", "hybrid", 512, (128, 32768), graph=True),
        # speculative decoding: four tokens per request are verified at once (sixteen query rows per kv head)
        _step("verify_draft", "8b", 32, (1024, 8192), q_tokens=4),
        # the same at head_dim 256 with one draft token and Hadamard-rotated keys
        _step("verify_rotated", "hybrid", 96, (512, 16384), q_tokens=2, had=True),
        # positions-outermost pages of 64 tokens (the other page order that the backend advertises)
        _step("decode_nhd", "dense256", 48, (512, 16384), page=64, order="LBNHC"),
        # FP8 keys with FP4 values
        _step("decode_k8v4", "hybrid", 128, (512, 16384), k8=True),
        # one fresh prompt
        _step("prefill_prompt", "8b", n_pre=1, new=(6144, 6144)),
        # a chunk of a long prompt over its cached part
        _step("prefill_chunk", "hybrid", n_pre=1, new=(2048, 2048), prior=(30000, 30000)),
        # continuous batching: prompts of several lengths join a running decode batch, some with a cached prefix
        _step("mixed_step", "8b", 48, (700, 9000), n_pre=4, new=(90, 1500), prior=(0, 3000)),
        # the fill of a cache by prompts: 32768 tokens into random slots
        _write("write_fill", "8b", 32768),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def draw(rng):
    kind = rng.choice(("decode", "decode", "decode", "verify", "options", "prefill", "prefill", "mixed", "mixed",
                       "write"))
    shape = rng.choice(("8b", "8b", "70b", "hybrid", "dense256"))
    row = SHAPES[shape]["kv_heads"] * SHAPES[shape]["head_dim"]        # values of one token and side
    page = rng.choice((16, 16, 32, 64))
    if kind == "write":
        return _write(None, shape, _log(rng, 1, 32768 * 1024 // row), page, rng.random() < 0.75)
    if kind in ("decode", "verify", "options"):
        hi = _log(rng, 128, 131072)
        lo = _log(rng, max(1, hi // 64), hi)
        n = _log(rng, 1, max(1, min(512, 2 ** 30 // row // hi)))        # up to 2^30 cached values per side
        q = rng.choice((2, 3, 4)) if kind == "verify" else 1
        opt = {}
        if kind == "options":
            opt = rng.choice(({"order": "LBNHC"}, {"had": True}, {"k8": True}))
            if "k8" in opt and SHAPES[shape]["head_dim"] != 256:
                shape = "hybrid"
        return _step(None, shape, n, (lo, hi), q, page=page, graph=rng.random() < 0.4, **opt)
    if kind == "prefill":
        # one to four prompts or chunks; the attended pairs of all of them stay below those of prefill_chunk
        n = rng.choice((1, 1, 2, 4))
        new = _log(rng, 16, 6144 // n)
        prior = 0 if rng.random() < 0.5 else _log(rng, 64, 32000)
        while n * new * (prior + new) * SHAPES[shape]["group"] * row > 2048 * 32048 * 8 * 512:
            new, prior = max(16, new * 2 // 3), prior * 2 // 3
        return _step(None, shape, n_pre=n, new=(max(4, new // 2), new), prior=(prior // 2, prior), page=page,
                     had=rng.random() < 0.15, order="LBNHC" if rng.random() < 0.15 else "LBHNC")
    hi = _log(rng, 256, 16384)
    new = _log(rng, 16, 2048)
    return _step(None, shape, _log(rng, 1, 96), (max(1, hi // 8), hi), rng.choice((1, 1, 2)), rng.choice((1, 2, 3, 4)),
                 (max(4, new // 6), new), (0, _log(rng, 16, 4096)), page)


# ------------------------------------------------------------------------------------------------------------ lengths
def _quantiles(n, lo, hi):
    """n values of a log-uniform law on [lo, hi] (lo = 0 counts as 1, less one), by their quantiles"""
    off = 1 if lo == 0 else 0
    a, b = math.log(lo + off), math.log(hi + off)
    return [int(round(math.exp(a + (b - a) * (i + 0.5) / n))) - off for i in range(n)]


def _requests(case):
    """[(query tokens, context length with them)] of the step's requests, decode requests first"""
    q = case["q_tokens"]
    reqs = [(q, max(q, L)) for L in _quantiles(case["n_dec"], case["ctx_lo"], case["ctx_hi"])]
    new = _quantiles(case["n_pre"], case["new_lo"], case["new_hi"])
    prior = _quantiles(case["n_pre"], case["prior_lo"], case["prior_hi"])
    # the shortest prompt has the longest cached part; a prefill has more new tokens than a decode request has
    reqs += [(max(q + 1, n), max(q + 1, n) + p) for n, p in zip(new, reversed(prior))]
    return reqs


# ------------------------------------------------------------------------------------------------------------ prepare
def _kv(n, case, g):
    H, D = case["kv_heads"], case["head_dim"]
    k = torch.randn(n, H, D, generator=g, device="cuda")
    k[:, :, torch.tensor([3, D // 4 + 3, D // 2 + 3, 3 * D // 4 + 3], device="cuda")] *= OUTLIER
    v = torch.randn(n, H, D, generator=g, device="cuda")
    return k.to(torch.bfloat16), v.to(torch.bfloat16)


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed * 7919 + 17)
    H, D, PS = case["kv_heads"], case["head_dim"], case["page"]
    if case["kind"] == "write":
        n = case["n_tokens"]
        pages = (n + PS - 1) // PS + 7
        cache = Lt.alloc_cache(pages, PS, H, D, device="cuda")
        slots = torch.randperm(pages * PS, generator=g, device="cuda")[:n].contiguous()
        k, v = _kv(n, case, g)
        kv = torch.cat((k.view(n, H * D), v.view(n, H * D)), dim=1)     # slices of one projection's rows
        flat, strides = Lt.flat_views(*Lt.slot_views(cache, H, D))
        return SimpleNamespace(kind="write", k=kv[:, :H * D].view(n, H, D), v=kv[:, H * D:].view(n, H, D), flat=flat,
                               strides=strides, page=PS, slots=slots, search=case["search"], cache=cache,
                               gk=torch.full((H,), GK, device="cuda"), gv=torch.full((H,), GV, device="cuda"))
    reqs = _requests(case)
    rng = torch.Generator().manual_seed(seed + 5)
    n_dec = case["n_dec"]
    perm = torch.randperm(n_dec, generator=rng).tolist()
    reqs = [reqs[i] for i in perm] + reqs[n_dec:]
    B, T, HQ = len(reqs), sum(q for q, _ in reqs), H * case["group"]
    n_pages = [(L + PS - 1) // PS for _, L in reqs]
    total = sum(n_pages)
    slot = Lt.k8_slot_bytes(D) if case["k8"] else Lt.slot_bytes(D)
    heads = H if case["k8"] else 2 * H
    if case["order"] == "LBNHC":
        phys = torch.zeros((total + 1, PS, heads, slot), dtype=torch.uint8, device="cuda")
        cache = phys.permute(0, 2, 1, 3)
    else:
        phys = cache = torch.zeros((total + 1, heads, PS, slot), dtype=torch.uint8, device="cuda")
    pool = torch.randperm(total, generator=g, device="cuda") + 1            # page 0 stays unused
    bt = torch.zeros((B, max(n_pages)), dtype=torch.int32, device="cuda")
    lens = torch.tensor([L for _, L in reqs], device="cuda")
    n_pages_t = torch.tensor(n_pages, device="cuda")
    first = torch.cumsum(n_pages_t, 0) - n_pages_t
    col = torch.arange(bt.shape[1], device="cuda")
    have = col[None, :] < n_pages_t[:, None]
    bt[have] = pool[(first[:, None] + col[None, :])[have]].to(torch.int32)

    saved = {k: os.environ.get(k) for k in ("HORIZON_KVFP4_HAD", "HORIZON_KVFP4_K8")}
    os.environ["HORIZON_KVFP4_HAD"] = "1" if case["had"] else "0"
    os.environ["HORIZON_KVFP4_K8"] = "1" if case["k8"] else "0"
    spec = case["q_tokens"] - 1
    impl = BE.HorizonFp4Impl(HQ, D, D ** -0.5, num_kv_heads=H, kv_cache_dtype="nvfp4", max_num_seqs=512,
                             num_speculative_tokens=spec)
    for k, val in saved.items():
        if val is None:
            os.environ.pop(k)
        else:
            os.environ[k] = val
    builder = BE.HorizonFp4Builder(vllm_config=SimpleNamespace(
        speculative_config=SimpleNamespace(num_speculative_tokens=spec)))
    layer = SimpleNamespace(_k_scale_float=GK, _v_scale_float=GV, layer_name="model.layers.0.self_attn.attn")
    # every page is filled as prompts fill it
    for i in range(0, total, 4096):
        pgs = pool[i:i + 4096]
        sl = (pgs[:, None] * PS + torch.arange(PS, device="cuda")[None, :]).reshape(-1)
        k, v = _kv(sl.numel(), case, g)
        impl.do_kv_cache_update(layer, k, v, cache, sl)
    # the step's tokens: the last q of every request
    qlens = torch.tensor([q for q, _ in reqs], device="cuda")
    qsl_cpu = torch.tensor([0] + [q for q, _ in reqs], dtype=torch.int64).cumsum(0).to(torch.int32)
    req_of = torch.repeat_interleave(torch.arange(B, device="cuda"), qlens)
    pos = torch.arange(T, device="cuda") - qsl_cpu[:-1].cuda().long()[req_of] + (lens - qlens)[req_of]
    slots = bt[req_of, pos // PS].long() * PS + pos % PS
    k, v = _kv(T, case, g)
    kv = torch.cat((k.view(T, H * D), v.view(T, H * D)), dim=1)         # slices of one projection's rows
    seq_lens = lens.to(torch.int32)
    cam = SimpleNamespace(num_reqs=B, num_actual_tokens=T, query_start_loc=qsl_cpu.cuda(), query_start_loc_cpu=qsl_cpu,
                          seq_lens=seq_lens, seq_lens_cpu_upper_bound=seq_lens.cpu(), block_table_tensor=bt,
                          slot_mapping=slots)
    s = SimpleNamespace(kind="step", impl=impl, layer=layer, k=kv[:, :H * D], v=kv[:, H * D:], cache=cache, phys=phys,
                        slots=slots, meta=builder.build(0, cam), graph=None, n_decode=n_dec * case["q_tokens"],
                        q=torch.randn(T, HQ * D, generator=g, device="cuda").to(torch.bfloat16),
                        out=torch.zeros(T, HQ * D, dtype=torch.bfloat16, device="cuda"))
    if case["graph"]:
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            _layer_step(s)
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=side):
                _layer_step(s)
        torch.cuda.current_stream().wait_stream(side)
        s.graph = graph
    return s


def _layer_step(s):
    s.impl.do_kv_cache_update(s.layer, s.k, s.v, s.cache, s.slots)
    s.impl.forward(s.layer, s.q, s.k, s.v, s.cache, s.meta, s.out)


def run(state):
    s = state
    if s.kind == "write":
        K.write(s.k, s.v, s.flat, s.strides, s.page, s.slots, s.gk, s.gv, s.search)
        return {"cache": s.cache}
    if s.graph is not None:
        s.graph.replay()
    else:
        _layer_step(s)
    return {"decode": s.out[:s.n_decode], "prefill": s.out[s.n_decode:], "cache": s.phys}


# ------------------------------------------------------------------------------------------------------ work, tolerance
def work(case):
    H, D = case["kv_heads"], case["head_dim"]
    slot = Lt.k8_slot_bytes(D) if case.get("k8") else 2 * Lt.slot_bytes(D)     # cached bytes of a token and kv head
    if case["kind"] == "write":
        return {"bytes": case["n_tokens"] * (H * (4 * D + slot) + 8), "flops": 0}
    HQ = H * case["group"]
    n = flops = 0
    for q, L in _requests(case):
        n += q * (H * (4 * D + slot) + 8 + 4 * HQ * D)      # new k, v read and cached, slot id, query, output
        n += (L - q) * H * slot                             # cached context read (the new tokens are counted above)
        flops += 4 * D * HQ * (q * (L - q) + q * (q + 1) // 2)
    return {"bytes": n, "flops": flops}


def tolerance(case):
    """the cache bytes are exact. The attention output is bf16, from probabilities that are rounded to fp16 before the
    value product: against the same attention in 64 bits over the same cache it is off by 1.66e-3 to 1.68e-3 (2-norm)
    and by at most 4.4e-3 of a value or of the root mean square, most of it the output's own rounding (measured on every
    listed case); four times that"""
    if case["kind"] == "write":
        return "exact"
    return {"rel": 7e-3, "max": 1.8e-2, "differ": 0.0}


# --------------------------------------------------------------------------------------------------------------- exact
def _e4m3(b):
    return b.contiguous().view(torch.float8_e4m3fn).double()


def _e2m1(b):
    """codes, two to a byte (the first in the low nibble), in blocks of sixteen -> (.., blocks, 16)"""
    table = torch.tensor([0, 0.5, 1, 1.5, 2, 3, 4, 6, -0.0, -0.5, -1, -1.5, -2, -3, -4, -6], dtype=torch.float64,
                         device=b.device)
    codes = torch.stack((b & 15, b >> 4), dim=-1).long()
    return table[codes].reshape(*b.shape[:-1], b.shape[-1] // 8, 16)


def _fp4(slots, D):
    return (_e2m1(slots[..., :D // 2]) * _e4m3(slots[..., D // 2:])[..., None]).reshape(*slots.shape[:-1], D)


def exact(case, seed):
    """The attention of the step in 64 bits over the bytes that the cache holds once the step's tokens are in it (those
    bytes have a tolerance of their own, none, and no value here). Decode rows are scaled by the value scale twice, as
    their entry point's two arguments are, prefill rows once."""
    if case["kind"] == "write":
        return None
    s = prepare(case, seed)
    s.impl.do_kv_cache_update(s.layer, s.k, s.v, s.cache, s.slots)
    H, D, G, PS = case["kv_heads"], case["head_dim"], case["group"], case["page"]
    q_all = s.q.view(-1, H * G, D).double()
    if case["had"]:
        signs = torch.randint(0, 2, (D,), generator=torch.Generator().manual_seed(0x6B7634)) * 2 - 1
        had = torch.ones((1, 1), dtype=torch.float64)
        while had.shape[0] < D:
            had = torch.cat((torch.cat((had, had), 1), torch.cat((had, -had), 1)))
        q_all = (q_all * signs.cuda()) @ (had * D ** -0.5).cuda()
    out = torch.zeros_like(q_all)
    qsl, lens, bt = s.meta.query_start_loc.tolist(), s.meta.seq_lens.tolist(), s.meta.block_table
    for b, L in enumerate(lens):
        t0, t1 = qsl[b], qsl[b + 1]
        pages = bt[b, :(L + PS - 1) // PS].long()
        lim = torch.arange(L - (t1 - t0) + 1, L + 1, device="cuda").repeat_interleave(G)
        for h in range(H):
            rows = s.cache[pages, h].reshape(-1, s.cache.shape[3])[:L]
            if case["k8"]:
                k, v = _e4m3(rows[:, :D]), _fp4(rows[:, D:], D)
            else:
                k, v = _fp4(rows, D), _fp4(s.cache[pages, H + h].reshape(-1, rows.shape[1])[:L], D)
            qh = q_all[t0:t1, h * G:(h + 1) * G].reshape(-1, D)
            step = max(1, 2 ** 27 // L)
            o = []
            for r in range(0, qh.shape[0], step):
                w = qh[r:r + step] @ k.T * (D ** -0.5 * GK)
                w.masked_fill_(torch.arange(L, device="cuda")[None, :] >= lim[r:r + step, None], -math.inf)
                o.append(torch.softmax(w, dim=1) @ v)
            out[t0:t1, h * G:(h + 1) * G] = torch.cat(o).view(t1 - t0, G, D) * (GV * GV if t0 < s.n_decode else GV)
    out = out.view(out.shape[0], H * G * D)
    return {"decode": out[:s.n_decode], "prefill": out[s.n_decode:], "cache": None}
