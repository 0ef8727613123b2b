"""The prefill kernels (csrc/hkv_prefill.cu) against attention in fp64 over the same cache bytes, at the sizes where they
can go wrong: row tiles and key tiles with remainders, groups that do not divide 128, row tiles whose keys are divided
among CTAs, contexts longer than the chunk, many requests in one call, query tokens without any visible key."""
import numpy as np
import pytest
import torch

import synth
from cases import bf16_tensor
from horizon_kernels_b200 import _lib
from horizon_kernels_b200 import kernels as K
from horizon_kernels_b200 import layout as Lt
from oracle import kvfp4 as O

pytestmark = pytest.mark.gpu


def run_case(qls, lens, KVH, G, D, PS=16, chunk=65536, q_dtype=torch.bfloat16, out_dtype=torch.bfloat16, seed=5, qk_scale=None):
    c = synth.paged_case(seed + D, lens, KVH, G, D, PS, outliers=True, ql_list=qls)
    dev = torch.device("cuda")
    gk = torch.full((KVH,), 0.04, device=dev)
    gv = torch.full((KVH,), 1.0, device=dev)
    cache = Lt.alloc_cache(c["NP"], PS, KVH, D, device=dev, fill=0x7F)
    flat, strides = Lt.flat_views(*Lt.slot_views(cache, KVH, D))
    K.write(bf16_tensor(c["key"]), bf16_tensor(c["val"]), flat, strides, PS, torch.from_numpy(c["slots"]).to(dev), gk, gv)
    q = bf16_tensor(c["q"]).to(q_dtype)                  # (exact: the values are ordinary)
    NT = q.shape[0]
    out = torch.full((NT + 3, KVH * G, D), 5.0, dtype=out_dtype, device=dev)
    qsl = [int(x) for x in c["qsl"]]
    rows = [(b, qsl[b], qsl[b + 1], L) for b, L in enumerate(lens)]
    sm = D ** -0.5 if qk_scale is None else qk_scale
    ws = K.alloc_workspace(4, KVH, min(G, 8), D)
    K.prefill(q, flat, strides, PS, torch.from_numpy(c["bt"]).to(dev), rows, sm * 0.04, 1.0, KVH, out, chunk=chunk,
              workspace=ws)
    assert K.workspace_status(ws) == 0
    assert (out[NT:] == 5.0).all()
    lay = O.Layout.slots(PS, KVH, D)
    ref, _ = O.attention(c["q"], cache.cpu().numpy().reshape(-1), lay, c["bt"], c["seq_lens"], c["qsl"], KVH, sm,
                         np.full(KVH, 0.04, np.float32), np.ones(KVH, np.float32), 1.0)
    got, want = out[:NT].float().cpu().numpy().astype(np.float64), np.asarray(ref, np.float64)
    # probabilities and the output are each rounded to 11 and 8 bits: 2^-9 of a value from the latter, less from the
    # former; four times the sum of both roundings' root mean squares (1.7e-3)
    rel = np.linalg.norm(got - want) / max(np.linalg.norm(want), 1e-30)
    assert rel <= 2.5e-3, rel
    return out, rows, want


SIZES = [
    ([1], [1]), ([5], [5]), ([128], [128]), ([129], [129]), ([31], [4000]), ([300], [777]), ([64, 33, 2, 257], [64, 1000, 300, 257]),
]


@pytest.mark.parametrize("qls,lens", SIZES)
@pytest.mark.parametrize("KVH,G,D", [(2, 4, 128), (2, 8, 256)])
def test_sizes(qls, lens, KVH, G, D):
    run_case(qls, lens, KVH, G, D)


@pytest.mark.parametrize("KVH,G,D,PS", [(1, 1, 128, 16), (3, 6, 128, 32), (1, 12, 256, 64), (4, 6, 256, 16), (1, 64, 128, 16)])
def test_groups_and_pages(KVH, G, D, PS):
    run_case([70, 9], [200, 513], KVH, G, D, PS)


@pytest.mark.parametrize("chunk", [1, 128, 300, 1024])
@pytest.mark.parametrize("KVH,G,D", [(2, 4, 128), (1, 8, 256)])
def test_chunks_keep_a_state(KVH, G, D, chunk):
    """contexts of several chunks, alone and among requests that share a launch; fp32 output"""
    run_case([150, 20, 40], [1500, 260, 900], KVH, G, D, chunk=chunk, out_dtype=torch.float32)


@pytest.mark.parametrize("D", [128, 256])
def test_divided_row_tiles(D):
    """one short request over a long context: every CTA has a part of the same row tiles"""
    run_case([3], [20000], 1, 4, D)


def test_fp16_queries():
    run_case([100], [500], 2, 4, 128, q_dtype=torch.float16)


@pytest.mark.parametrize("D", [128, 256])
def test_negative_and_zero_scale(D):
    run_case([40], [300], 1, 4, D, qk_scale=-0.05)
    run_case([40], [300], 1, 4, D, qk_scale=0.0)


@pytest.mark.parametrize("D", [128, 256])
def test_tokens_without_keys(D):
    """more query tokens than context: the first ones see no key and give zeros"""
    dev = torch.device("cuda")
    KVH, G, PS, ql, L = 2, 4, 16, 200, 37
    cache = torch.randint(0, 120, (4, 2 * KVH, PS, Lt.slot_bytes(D)), dtype=torch.uint8, device=dev)
    flat, strides = Lt.flat_views(*Lt.slot_views(cache, KVH, D))
    q = torch.randn(ql, KVH * G, D, device=dev).to(torch.bfloat16)
    out = torch.full_like(q, 3.0)
    K.prefill(q, flat, strides, PS, torch.arange(4, dtype=torch.int32, device=dev).view(1, 4), [(0, 0, ql, L)], 1e-3, 1.0,
              KVH, out)
    assert (out[:ql - L] == 0).all() and torch.isfinite(out.float()).all() and (out[ql - L:] != 0).any()


def test_many_requests():
    """more requests than one launch takes"""
    rng = np.random.default_rng(3)
    qls = [int(x) for x in rng.integers(2, 40, 70)]
    lens = [q + int(x) for q, x in zip(qls, rng.integers(0, 200, 70))]
    run_case(qls, lens, 1, 4, 128)


def test_graph_capture_and_repeat():
    """captured once and replayed: the same bits as the eager call"""
    dev = torch.device("cuda")
    KVH, G, D, PS, ql, L = 2, 4, 128, 16, 130, 700
    cache = torch.randint(0, 120, (64, 2 * KVH, PS, Lt.slot_bytes(D)), dtype=torch.uint8, device=dev)
    flat, strides = Lt.flat_views(*Lt.slot_views(cache, KVH, D))
    q = torch.randn(ql, KVH * G, D, device=dev).to(torch.bfloat16)
    bt = torch.randperm(64, device=dev)[:L // PS + 1].to(torch.int32).view(1, -1)
    eager, out = torch.zeros_like(q), torch.zeros_like(q)
    call = lambda o: K.prefill(q, flat, strides, PS, bt, [(0, 0, ql, L)], 1e-3, 1.0, KVH, o)  # noqa: E731
    call(eager)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        call(out)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=side):
            call(out)
    torch.cuda.current_stream().wait_stream(side)
    out.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, eager)


def filled(KVH, D, L, k, v, gk, PS=16, nhd=False, k8=False, signs=None):
    """cache of one request of L tokens with the given keys and values: (flat, strides), block table"""
    dev = torch.device("cuda")
    per = (L + PS - 1) // PS
    heads, slot = (KVH, Lt.k8_slot_bytes(D)) if k8 else (2 * KVH, Lt.slot_bytes(D))
    if nhd:
        cache = torch.full((per + 2, PS, heads, slot), 0x7F, dtype=torch.uint8, device=dev).permute(0, 2, 1, 3)
    else:
        cache = torch.full((per + 2, heads, PS, slot), 0x7F, dtype=torch.uint8, device=dev)
    flat, strides = Lt.k8_flat_views(*Lt.k8_views(cache, D)) if k8 else Lt.flat_views(*Lt.slot_views(cache, KVH, D))
    bt = torch.randperm(per, generator=torch.Generator().manual_seed(L)).to(torch.int32).view(1, per).to(dev)
    pos = torch.arange(L, device=dev)
    slots = bt[0, pos // PS].long() * PS + pos % PS
    one = torch.ones(KVH, device=dev)
    K.write(k.to(torch.bfloat16), v.to(torch.bfloat16), flat, strides, PS, slots, gk * one, one, signs=signs, k8=k8)
    return flat, strides, bt


def attend64(q, flat, strides, PS, bt, rows, KVH, sm, f16_probabilities=False, k8=False):
    """per (token, head) in 64 bits: the output, sum_j w_j |v_j|, and the largest score (log2) of every 128 keys; optionally
    with the probabilities rounded to f16 under the row's exact maximum before the value product"""
    NT, HQ, D = q.shape
    G = HQ // KVH
    out, absv = (torch.zeros(NT, HQ, D, dtype=torch.float64, device=q.device) for _ in range(2))
    tops = {}
    for b, q0, q1, L in rows:
        kk, vv = (torch.empty(L, KVH, D, dtype=torch.float16, device=q.device) for _ in range(2))
        K.dequant_tokens(flat, strides, PS, bt[b].contiguous(), 0, L, kk, vv, k8=k8)
        ql = q1 - q0
        hidden = torch.arange(L, device=q.device)[None] >= torch.arange(L - ql + 1, L + 1, device=q.device).repeat_interleave(G)[:, None]
        for h in range(KVH):
            s = q[q0:q1, h * G:(h + 1) * G].reshape(ql * G, D).double() @ kk[:, h].double().T * sm
            s.masked_fill_(hidden, -float("inf"))
            p = torch.exp(s - s.amax(dim=1, keepdim=True))
            pn = p.half().double() if f16_probabilities else p
            den = p.sum(dim=1, keepdim=True)
            out[q0:q1, h * G:(h + 1) * G] = (pn @ vv[:, h].double() / den).view(ql, G, D)
            absv[q0:q1, h * G:(h + 1) * G] = (p @ vv[:, h].double().abs() / den).view(ql, G, D)
            pad = torch.nn.functional.pad(s, (0, -L % 128), value=-float("inf"))
            tops[b, h] = pad.view(ql * G, -1, 128).amax(dim=2) * 1.4426950408889634
    return out, absv, tops


@pytest.mark.parametrize("KVH,G,D,ql,L,amp", [(2, 4, 128, 700, 3000, 1.0), (2, 8, 256, 256, 5000, 1.0), (1, 4, 128, 5, 9000, 1.0),
                                              (2, 4, 128, 512, 4000, 0.3), (2, 4, 256, 300, 4000, 0.1)])
def test_error_is_that_of_probabilities_under_the_exact_maximum(KVH, G, D, ql, L, amp):
    """fp32 output against 64 bits: what the products lose is the rounding of the probabilities to f16. Where few keys have most
    of the weight it is small if the largest probability is exactly 1, as under the row's exact maximum, and two to three times
    that under a maximum that lags behind. The bound is the error of 64-bit attention with probabilities rounded to f16 under the
    exact maximum, plus a tenth (the running maximum rounds the earlier keys on another grid)"""
    g = torch.Generator(device="cuda").manual_seed(D + ql)
    k, v = torch.randn(2, L, KVH, D, generator=g, device="cuda")
    k[:, :, [3, D // 4 + 3, D // 2 + 3, 3 * D // 4 + 3]] *= 20.0 * amp
    flat, strides, bt = filled(KVH, D, L, k, v, 0.04)
    q = torch.randn(ql, KVH * G, D, generator=g, device="cuda").to(torch.bfloat16)
    rows, sm = [(0, 0, ql, L)], D ** -0.5 * 0.04
    out = torch.zeros(ql, KVH * G, D, device="cuda")
    K.prefill(q, flat, strides, 16, bt, rows, sm, 1.0, KVH, out)
    want, _, _ = attend64(q, flat, strides, 16, bt, rows, KVH, sm)
    f16, _, _ = attend64(q, flat, strides, 16, bt, rows, KVH, sm, f16_probabilities=True)
    err, bound = (out.double() - want).norm() / want.norm(), (f16 - want).norm() / want.norm()
    assert err <= 1.1 * bound, (float(err), float(bound))


@pytest.mark.parametrize("KVH,G,D,ql,L,chunk", [(2, 4, 128, 1100, 2200, 65536), (2, 4, 128, 1100, 2200, 512), (1, 4, 128, 9, 1700, 65536),
                                                (2, 8, 256, 560, 1700, 65536), (2, 8, 256, 560, 1700, 512), (1, 8, 256, 9, 1700, 65536),
                                                (1, 8, 256, 9, 1700, 900)])
def test_maxima_that_rise_in_every_tile(KVH, G, D, ql, L, chunk):
    """keys that grow along the context: for every other query head each tile's largest score exceeds all before it by more than
    14 (log2), for the rest it falls, so that in every tile some rows of a warp rescale the output and others do not; row tiles
    whole (6 tiles and more), divided among CTAs, and chunk by chunk. Every element against 64 bits"""
    g = torch.Generator(device="cuda").manual_seed(D + ql + chunk)
    u = torch.nn.functional.normalize(torch.randn(KVH, D, generator=g, device="cuda"), dim=1)
    grow = (torch.arange(L, device="cuda") // 128 + 1).float()[:, None, None]
    k = u * grow * 3.0 + 0.02 * torch.randn(L, KVH, D, generator=g, device="cuda")
    v = torch.randn(L, KVH, D, generator=g, device="cuda")
    flat, strides, bt = filled(KVH, D, L, k, v, float(k.abs().max()) / 2688)
    sign = 1.0 - 2.0 * (torch.arange(KVH * G, device="cuda") % 2)
    q = (u.repeat_interleave(G, dim=0) * sign[:, None] + 0.01 * torch.randn(ql, KVH * G, D, generator=g, device="cuda")).to(torch.bfloat16)
    rows, sm = [(0, 0, ql, L)], 6.0 * float(k.abs().max()) / 2688
    out = torch.zeros(ql, KVH * G, D, device="cuda")
    K.prefill(q, flat, strides, 16, bt, rows, sm, 1.0, KVH, out, chunk=chunk)
    want, absv, tops = attend64(q, flat, strides, 16, bt, rows, KVH, sm)
    for t in tops.values():                              # [token x head][tile]; the first eight tiles are whole for every row
        t = t.view(ql, G, -1)[:, :, :8]
        assert (t[:, 0::2].diff(dim=2) > 14).all() and (t[:, 1::2].diff(dim=2) < 0).all()
    # a weight is off by 2^-11 from f16 and by less than 2^-12 from its exponent (scores below 500 (log2), fp32 sums of products);
    # probabilities below f16's normal range by 2^-25 of the largest
    bound = absv * (2.0 ** -11 + 2.0 ** -12) + L * 2.0 ** -25 * float(v.abs().max()) * 2
    bad = ((out.double() - want).abs() > bound).sum()
    assert bad == 0, int(bad)


@pytest.mark.parametrize("ql,L,chunk", [(300, 900, 65536), (6, 3000, 65536), (200, 1000, 256)])
@pytest.mark.parametrize("D", [128, 256])
def test_non_finite_queries_and_scales(D, ql, L, chunk):
    """row tiles whole, divided and chunk by chunk: a query row with a NaN or an infinity gives NaN, as softmax over its scores
    does, and changes no other row; a NaN scale gives NaN"""
    KVH, G = 1, 4
    g = torch.Generator(device="cuda").manual_seed(D + ql)
    k, v = torch.randn(2, L, KVH, D, generator=g, device="cuda")
    flat, strides, bt = filled(KVH, D, L, k, v, 0.01)
    q = torch.randn(ql, KVH * G, D, generator=g, device="cuda").to(torch.bfloat16)
    call = lambda q, a, b: K.prefill(q, flat, strides, 16, bt, [(0, 0, ql, L)], a, b, KVH, torch.zeros_like(q), chunk=chunk)  # noqa: E731
    want, bad = call(q, D ** -0.5, 1.0), q.clone()
    bad[0, 1, 5], bad[3, 0, 0], bad[ql - 1, 3, D - 1] = float("nan"), float("inf"), float("-inf")
    hit = torch.zeros(ql, KVH * G, dtype=torch.bool, device="cuda")
    hit[0, 1] = hit[3, 0] = hit[ql - 1, 3] = True
    got = call(bad, D ** -0.5, 1.0)
    assert got[hit].isnan().all() and torch.equal(got[~hit], want[~hit]) and torch.isfinite(want.float()).all()
    for a, b in ((float("nan"), 1.0), (1.0, float("nan"))):
        assert call(q, a, b).isnan().all(), (a, b)


@pytest.mark.parametrize("own", [True, False])
@pytest.mark.parametrize("D,chunk", [(128, 65536), (256, 65536), (128, 256)])
def test_a_wait_that_runs_out_ends_the_launch_and_is_reported(D, chunk, own):
    """the give-up path of the attention kernel: every CTA stops fetching early, its waits run out after a millisecond, the
    launches end and the status word of the workspace (without one: of the library's own) says so, once; the same call then
    works, to the bit"""
    import ctypes as C
    KVH, G, ql, L = 2, 4, 700, 1500
    k, v = torch.randn(2, L, KVH, D, device="cuda")
    flat, strides, bt = filled(KVH, D, L, k, v, 0.01)
    q = torch.randn(ql, KVH * G, D, device="cuda").to(torch.bfloat16)
    ws = K.alloc_workspace(1, KVH, G, D) if own else None
    want, out = torch.zeros_like(q), torch.zeros_like(q)
    K.prefill(q, flat, strides, 16, bt, [(0, 0, ql, L)], D ** -0.5, 1.0, KVH, want, chunk=chunk, workspace=ws)
    assert K.workspace_status(ws) == 0
    lib, p = _lib.load(), lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    host_rows = (C.c_int32 * 4)(0, 0, ql, L)
    nb = lib.hkv_prefill_scratch_bytes(host_rows, 1, ql, KVH, G, D, chunk, 0)
    scratch = torch.empty(nb, dtype=torch.uint8, device="cuda")
    call = lambda f: f(p(q), 0, *(p(t) for t in flat), (C.c_int64 * 6)(*strides), 16, p(bt), *bt.shape, host_rows, 1, ql, KVH, G, D,  # noqa: E731
                       D ** -0.5, 1.0, None, 0, chunk, p(scratch), nb, p(out), 0, p(ws) if own else None,
                       C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert call(lib.hkv_selftest_prefill_timeout) == 0
    assert K.workspace_status(ws) == -8                  # HKV_ERR_DEVICE_WAIT, cleared by the read
    assert K.workspace_status(ws) == 0
    assert call(lib.hkv_prefill) == 0
    assert K.workspace_status(ws) == 0
    assert torch.equal(out, want)


@pytest.mark.parametrize("chunk", [65536, 384])
@pytest.mark.parametrize("KVH,G,D,PS", [(2, 4, 128, 16), (3, 2, 128, 32), (1, 8, 128, 64), (2, 8, 256, 16), (3, 4, 256, 64)])
def test_positions_outermost_pages(KVH, G, D, PS, chunk):
    """vLLM's other page order: the bits of head-major pages of the same tokens (odd kv head counts put token rows off the
    16-byte grid at head_dim 128)"""
    ql, L = 150, 1300
    g = torch.Generator(device="cuda").manual_seed(D + PS)
    k, v = torch.randn(2, L, KVH, D, generator=g, device="cuda")
    q = torch.randn(ql, KVH * G, D, generator=g, device="cuda").to(torch.bfloat16)
    got = []
    for nhd in (False, True):
        flat, strides, bt = filled(KVH, D, L, k, v, 0.01, PS, nhd=nhd)
        got.append(K.prefill(q, flat, strides, PS, bt, [(0, 0, ql, L)], 0.01 * D ** -0.5, 1.0, KVH, torch.zeros_like(q), chunk=chunk))
    assert torch.equal(got[0], got[1]) and got[0].any()


@pytest.mark.parametrize("chunk", [65536, 1000, 384])
@pytest.mark.parametrize("D,option", [(128, "rotated"), (256, "rotated"), (256, "k8"), (128, "f16"), (256, "f16")])
def test_options_over_chunks(D, option, chunk):
    """rotated keys, FP8 keys and f16 queries in one and in several chunks, every element against 64 bits"""
    KVH, G, ql, L = 2, 4, 150, 1700
    g = torch.Generator(device="cuda").manual_seed(D + ql)
    k, v = torch.randn(2, L, KVH, D, generator=g, device="cuda")
    k[:, :, [3, D // 2 + 3]] *= 20.0
    q = torch.randn(ql, KVH * G, D, generator=g, device="cuda").to(torch.float16 if option == "f16" else torch.bfloat16)
    signs = K.hadamard_signs(D, device="cuda") if option == "rotated" else None
    k8 = option == "k8"
    gk = 0.25 if k8 else 0.04
    flat, strides, bt = filled(KVH, D, L, k, v, gk, k8=k8, signs=signs)
    rows, sm, out = [(0, 0, ql, L)], D ** -0.5 * gk, torch.zeros(ql, KVH * G, D, device="cuda")
    K.prefill(q, flat, strides, 16, bt, rows, sm, 1.0, KVH, out, chunk=chunk, signs=signs, k8=k8)
    q64 = q if signs is None else K.rotate(q, signs).to(torch.bfloat16)
    want, absv, _ = attend64(q64, flat, strides, 16, bt, rows, KVH, sm, k8=k8)
    # as in test_maxima_that_rise_in_every_tile
    bound = absv * (2.0 ** -11 + 2.0 ** -12) + L * 2.0 ** -25 * float(v.abs().max()) * 2
    assert ((out.double() - want).abs() <= bound).all()
