"""GPU parity of the quantize-on-write kernel, through the C ABI: every cache byte must equal what the reference's
PyTorch writer produced (golden fixtures) and what the CPU oracle produces on the same inputs. Mirrors the reference's
write gates (scripts/kernels/kvfp4/test_kvfp4_gpu.py G1 and test_kvfp4_serving_gpu.py S4 in the reference tree)."""
import os

import numpy as np
import pytest
import torch

import synth
from cases import Cache, bf16_tensor, gpu_write
from oracle import kvfp4 as O

pytestmark = pytest.mark.gpu


def dev_t(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("name", ["a", "b"])
def test_write_golden(golden_dir, name):
    z = np.load(os.path.join(golden_dir, "write.npz"))
    KVH, D, PS, NP = (int(v) for v in z[f"{name}_geom"])
    key, val = bf16_tensor(z[f"{name}_key"]), bf16_tensor(z[f"{name}_val"])
    for search in (0, 1):
        for kind in ("region", "hnd", "nhd"):
            cache = Cache(NP, PS, KVH, D, kind, fill=0xA5)
            gpu_write(cache, key, val, dev_t(z[f"{name}_slots"]), dev_t(z[f"{name}_gk"]), dev_t(z[f"{name}_gv"]),
                      bool(search))
            got, want = cache.bytes(), z[f"{name}_{kind}_s{search}"]
            assert np.array_equal(got, want), (name, kind, search, int((got != want).sum()))


def kv_tokens(seed, NT, KVH, D, kind):
    k = synth.normal(seed, (NT, KVH, D))
    v = synth.normal(seed + 1, (NT, KVH, D)) * np.exp(0.5 * synth.normal(seed + 2, (NT, 1, 1)))
    if kind == "outlier":
        ch = [0, 1, D // 4, D // 4 + 1, D // 2 - 2, D // 2 - 1, D - 56, D - 55]
        k[:, :, ch] = k[:, :, ch] * 6 + 10
        k[0] *= 8
    elif kind == "edge":
        if NT > 0: k[0] = 0
        if NT > 1: v[1] = 0
        if NT > 2: k[2] *= 1e-30
        if NT > 3: v[3] *= 1e30
        if NT > 4: k[4, :, :16] = 300.0
        if NT > 5: v[5, :, ::3] = -0.0
        ties = np.tile(np.array([0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0, 6.0, -0.25, -0.75, -1.25, -1.75, -2.5, -3.5, -5.0,
                                 -6.0]), D // 16)          # quotients exactly on the rounding boundaries
        if NT > 6: k[6] = ties
        if NT > 7: v[7] = ties * 0.125
        if NT > 8: k[8] = ties * 3.0
        if NT > 9: v[9] = ties * (1.0 + 2.0 ** -7)
    return synth.to_bf16_bits(k), synth.to_bf16_bits(v)


@pytest.mark.parametrize("D,KVH,PS", [(128, 8, 16), (256, 2, 16), (256, 4, 64)])
@pytest.mark.parametrize("kind", ["random", "outlier", "edge"])
def test_write_matches_oracle(D, KVH, PS, kind):
    # 60 tokens hold every edge row and go four lanes to a block; `line` is the last count that does, the next goes one lane
    # to a block, as 300 do
    line = 19000 // (2 * KVH * D // 16)
    for NT in (1, 7, 60, line, line + 1, 300):
        NP = (NT + PS - 1) // PS + 3
        slots = synth.permutation(5 + NT, NP * PS)[:NT].astype(np.int64)
        slots[synth.uniform(6 + NT, NT) < 0.1] = -1
        kb, vb = kv_tokens(100 + NT, NT, KVH, D, kind)
        gk = np.array([1.0, 0.5, 2.0, 1.0, 0.3, 1.7, 0.01, 5.0][:KVH], np.float32)
        gv = np.array([1.0, 1.0, 0.25, 4.0, 2.0, 0.5, 0.02, 3.0][:KVH], np.float32)
        for search in (1, 0):
            for lay in ("hnd", "region"):
                cache = Cache(NP, PS, KVH, D, lay, fill=0xA5)
                want = np.full(cache.bytes().shape, 0xA5, np.uint8)
                O.write(kb, vb, want, cache.olay, slots, gk, gv, bool(search))
                args = (cache, bf16_tensor(kb), bf16_tensor(vb), dev_t(slots), dev_t(gk), dev_t(gv), bool(search))
                gpu_write(*args)
                got = cache.bytes().copy()
                assert np.array_equal(got, want), (D, kind, NT, search, lay, int((got != want).sum()))
                cache.phys.fill_(0xA5)                     # determinism: a second run writes the same bytes
                gpu_write(*args)
                assert np.array_equal(cache.bytes(), got)


@pytest.mark.parametrize("kind", ["edge", "outlier"])
@pytest.mark.parametrize("D,KVH", [(128, 8), (256, 2)])
def test_large_launch_one_lane_per_block_matches_oracle(D, KVH, kind):
    """many more than 19000 blocks: the launch gives every block to ONE lane, which scores the four scale candidates itself
    (packed fp32 pairs, quotients by multiply-adds) and falls back to IEEE divisions for zero blocks, tiny and huge
    scales; the edge rows (zeros, 1e-30, 1e30, -0.0, exact ties) go through both paths. The edge tokens are repeated
    across the launch so that whole warps and single lanes of a warp meet them."""
    PS, NT = 16, 4100 + 37
    NP = (NT + PS - 1) // PS + 2
    kb, vb = kv_tokens(640 + D, NT, KVH, D, kind)
    if kind == "edge":
        ek, ev = kv_tokens(641, 10, KVH, D, "edge")
        for t0 in (0, 1000, 1000 + 5, 2048, 4096, NT - 10):
            kb[t0:t0 + 10], vb[t0:t0 + 10] = ek, ev
    slots = synth.permutation(7 + D, NP * PS)[:NT].astype(np.int64)
    slots[synth.uniform(8 + D, NT) < 0.05] = -1
    gk = np.array([1.0, 0.5, 2.0, 1.0, 0.3, 1.7, 0.01, 5.0][:KVH], np.float32)
    gv = np.array([1.0, 1.0, 0.25, 4.0, 2.0, 0.5, 0.02, 3.0][:KVH], np.float32)
    for search in (True, False):
        cache = Cache(NP, PS, KVH, D, "hnd", fill=0xA5)
        want = np.full(cache.bytes().shape, 0xA5, np.uint8)
        O.write(kb, vb, want, cache.olay, slots, gk, gv, search)
        gpu_write(cache, bf16_tensor(kb), bf16_tensor(vb), dev_t(slots), dev_t(gk), dev_t(gv), search)
        got = cache.bytes()
        assert np.array_equal(got, want), (D, kind, search, int((got != want).sum()))


def test_write_from_strided_qkv_and_fewer_slots_than_tokens():
    """key / value are column slices of a fused qkv projection output; tokens beyond len(slot_mapping) are ignored"""
    NT, HQ, KVH, D, PS = 37, 32, 8, 128, 16
    qkv = (synth.normal(77, (NT, (HQ + 2 * KVH) * D)) * 2).astype(np.float32)
    t = bf16_tensor(synth.to_bf16_bits(qkv))
    key = t[:, HQ * D:(HQ + KVH) * D].view(NT, KVH, D)
    val = t[:, (HQ + KVH) * D:].view(NT, KVH, D)
    assert not key.is_contiguous()
    n_sl = 30
    NP = 5
    slots = synth.permutation(78, NP * PS)[:n_sl].astype(np.int64)
    gk = np.full(KVH, 0.01, np.float32)
    gv = np.full(KVH, 0.02, np.float32)
    cache = Cache(NP, PS, KVH, D, "hnd", fill=0x5A)
    gpu_write(cache, key, val, dev_t(slots), dev_t(gk), dev_t(gv), True)
    want = np.full(cache.bytes().shape, 0x5A, np.uint8)
    kb = synth.to_bf16_bits(qkv[:, HQ * D:(HQ + KVH) * D].reshape(NT, KVH, D))
    vb = synth.to_bf16_bits(qkv[:, (HQ + KVH) * D:].reshape(NT, KVH, D))
    O.write(kb[:n_sl], vb[:n_sl], want, cache.olay, slots, gk, gv, True)
    assert np.array_equal(cache.bytes(), want)


def test_write_graph_replay():
    NT, KVH, D, PS, NP = 64, 8, 128, 16, 8
    kb, vb = kv_tokens(300, NT, KVH, D, "outlier")
    slots = synth.permutation(301, NP * PS)[:NT].astype(np.int64)
    cache = Cache(NP, PS, KVH, D, "hnd", fill=0xA5)
    args = (cache, bf16_tensor(kb), bf16_tensor(vb), dev_t(slots), dev_t(np.full(KVH, 0.5, np.float32)),
            dev_t(np.full(KVH, 2.0, np.float32)), True)
    gpu_write(*args)
    torch.cuda.synchronize()
    first = cache.bytes().copy()
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        gpu_write(*args)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            gpu_write(*args)
    for _ in range(2):
        cache.phys.fill_(0xA5)
        g.replay()
        torch.cuda.synchronize()
        assert np.array_equal(cache.bytes(), first)


@pytest.mark.parametrize("search", [True, False])
def test_config3_fill_then_appends(search):
    """benchmark configuration 3 at full size: a prefill write of 32768 tokens x 8 kv heads x 128 into random pages, then 256
    steps appending one token to each of 128 sequences (crossing page boundaries); every cache byte, canaries of the
    untouched pages included, equal to the oracle's, with the scale search on and off"""
    KVH, D, PS = 8, 128, 16
    NT, NSEQ, STEPS = 32768, 128, 256
    app_pp = (STEPS + 9 + PS - 1) // PS                        # pages an appended sequence touches
    NP = NT // PS + NSEQ * app_pp + 8
    kb, vb = kv_tokens(400, NT, KVH, D, "outlier")
    perm = synth.permutation(401, NP)
    pre_pages = perm[:NT // PS]
    slots = (pre_pages[:, None] * PS + np.arange(PS)[None, :]).reshape(-1).astype(np.int64)
    gk = np.full(KVH, synth.tensor_scale(kb), np.float32)
    gv = np.full(KVH, synth.tensor_scale(vb), np.float32)
    cache = Cache(NP, PS, KVH, D, "hnd", fill=0xA5)
    want = np.full(cache.bytes().shape, 0xA5, np.uint8)
    gpu_write(cache, bf16_tensor(kb), bf16_tensor(vb), dev_t(slots), dev_t(gk), dev_t(gv), search)
    O.write(kb, vb, want, cache.olay, slots, gk, gv, search)
    app_pages = perm[NT // PS:NT // PS + NSEQ * app_pp].reshape(NSEQ, app_pp)
    ak, av = kv_tokens(500, NSEQ * STEPS, KVH, D, "random")
    ak, av = ak.reshape(STEPS, NSEQ, KVH, D), av.reshape(STEPS, NSEQ, KVH, D)
    dk, dv, dgk, dgv = bf16_tensor(ak), bf16_tensor(av), dev_t(gk), dev_t(gv)
    all_sl = []
    for step in range(STEPS):
        pos = 9 + step
        sl = (app_pages[np.arange(NSEQ), pos // PS] * PS + pos % PS).astype(np.int64)
        all_sl.append(sl)
        gpu_write(cache, dk[step], dv[step], dev_t(sl), dgk, dgv, search)
    O.write(ak.reshape(-1, KVH, D), av.reshape(-1, KVH, D), want, cache.olay, np.concatenate(all_sl), gk, gv, search)
    assert np.array_equal(cache.bytes(), want)


def test_config3_full_size_roundtrip():
    """32768 tokens x 8 kv heads x 128: the dequantised cache is within the format's error of the input and the
    written scales never exceed the saturating code (size-independent properties; the byte-exact check runs on a
    1024-token sample of the same launch)"""
    KVH, D, PS, NT = 8, 128, 16, 32768
    NP = NT // PS + 4
    g = torch.Generator(device="cuda").manual_seed(7)
    key = torch.randn(NT, KVH, D, generator=g, device="cuda")
    key[:, :, [3, 35, 67, 99]] *= 20.0
    key = key.to(torch.bfloat16)
    val = torch.randn(NT, KVH, D, generator=g, device="cuda").to(torch.bfloat16)
    slots = torch.randperm(NP * PS, generator=g, device="cuda")[:NT].to(torch.int64)
    gk = torch.full((KVH,), float(key.float().abs().max()) / (6 * 448), device="cuda")
    gv = torch.full((KVH,), float(val.float().abs().max()) / (6 * 448), device="cuda")
    cache = Cache(NP, PS, KVH, D, "hnd", fill=0xA5)
    gpu_write(cache, key, val, slots, gk, gv, True)
    torch.cuda.synchronize()
    phys = cache.phys                                           # (NP, 2 KVH, PS, 72)
    sl = slots.cpu().numpy()
    host = phys.cpu().numpy()
    sample = np.arange(0, NT, 32)
    from cases import bf16_bits
    kb, vb = bf16_bits(key[sample]), bf16_bits(val[sample])
    want = np.full(host.size, 0xA5, np.uint8)
    O.write(kb, vb, want, cache.olay, sl[sample], gk.cpu().numpy(), gv.cpu().numpy(), True)
    want = want.reshape(host.shape)
    pg, ps = sl[sample] // PS, sl[sample] % PS
    assert np.array_equal(host[pg, :, ps, :], want[pg, :, ps, :])
    sf = host[sl // PS, :, sl % PS, 64:]
    assert sf.max() <= 0x7E
    deq = O.dequantize_rows(host[sl // PS, :KVH, sl % PS, :64], host[sl // PS, :KVH, sl % PS, 64:],
                            gk.cpu().numpy()[None, :].astype(np.float64))
    x = key.float().cpu().numpy().astype(np.float64)
    rel = np.linalg.norm(deq - x) / np.linalg.norm(x)
    assert rel < 0.12, rel
