"""The native side of the host wrappers (csrc/hkv_host.cpp) against their Python path: the same bytes and bits for
arguments that only the latter takes, the same refusals, the current stream."""
from types import SimpleNamespace

import pytest
import torch

from horizon_kernels_b200 import _lib
from horizon_kernels_b200 import backend as BE
from horizon_kernels_b200 import kernels as K
from horizon_kernels_b200 import layout as Lt

pytestmark = pytest.mark.gpu

KVH, G, D, PS, B = 2, 4, 128, 16, 3


def _state():
    dev = torch.device("cuda")
    cache = Lt.alloc_cache(24, PS, KVH, D, device=dev)
    flat, strides = Lt.flat_views(*Lt.slot_views(cache, KVH, D))
    k, v = torch.randn(2, 300, KVH, D, device=dev).to(torch.bfloat16)
    g = torch.full((KVH,), 0.01, device=dev)
    bt = torch.arange(24, dtype=torch.int32, device=dev).view(B, 8)
    return dict(cache=cache, flat=flat, strides=strides, k=k, v=v, g=g, bt=bt, slots=torch.arange(300, device=dev),
                lens=torch.tensor([100, 7, 128], dtype=torch.int32, device=dev),
                qsl=torch.arange(B + 1, dtype=torch.int32, device=dev),
                q=torch.randn(B, KVH * G, D, device=dev).to(torch.bfloat16),
                ws=K.alloc_workspace(B, KVH, G, D))


def _decode(s, out, PS=PS, scale=0.05, **kw):
    return K.decode_ragged(s["q"], s["flat"], s["strides"], PS, s["bt"], s["lens"], s["qsl"], scale, 1.0, s["g"], s["g"],
                           1, out, s["ws"], **kw)


def _prefill(s, out, rows, PS=PS, chunk=65536, **kw):
    return K.prefill(s["q"], s["flat"], s["strides"], PS, s["bt"], rows, 0.05, 1.0, KVH, out, chunk=chunk, **kw)


class AnInt(int):
    pass


def test_both_paths_give_the_same(monkeypatch):
    s = _state()
    native, python, calls = torch.zeros_like(s["q"]), torch.zeros_like(s["q"]), []
    K.write(s["k"], s["v"], s["flat"], s["strides"], PS, s["slots"], s["g"], s["g"])
    want = s["cache"].clone()
    s["cache"].zero_()
    K.write(s["k"], s["v"], s["flat"], s["strides"], AnInt(PS), s["slots"], s["g"], s["g"], search=1)   # the Python path
    assert torch.equal(s["cache"], want) and want.any()
    h = _lib.host()
    spy = type("Spy", (), {n: staticmethod(lambda *a, n=n: (calls.append((n, getattr(h, n)(*a))), calls[-1][1])[1])
                           for n in ("write", "decode", "prefill")})
    monkeypatch.setattr(_lib, "_host", spy)
    _decode(s, native)
    _decode(s, python, PS=AnInt(PS))
    assert torch.equal(native, python) and native.any()
    rows = [(0, 0, 2, 100), (2, 2, 3, 128)]
    _prefill(s, native.zero_(), rows)
    _prefill(s, python.zero_(), tuple(rows), PS=AnInt(PS))
    assert torch.equal(native, python) and native.any()
    assert calls == [("decode", 0), ("decode", None), ("prefill", 0), ("prefill", None)]


def test_refusals_are_the_python_ones():
    s = _state()
    out = torch.zeros_like(s["q"])
    with pytest.raises(TypeError):
        K.write(s["k"].float(), s["v"], s["flat"], s["strides"], PS, s["slots"], s["g"], s["g"])
    with pytest.raises(ValueError):
        K.write(s["k"], s["v"], s["flat"], s["strides"], PS, torch.arange(301, device="cuda"), s["g"], s["g"])
    with pytest.raises(ValueError):
        _decode(s, out[:2])
    with pytest.raises(RuntimeError):
        _decode(s, out.cpu())
    with pytest.raises(_lib.HkvError):
        _decode(s, out, PS=24)
    with pytest.raises(ValueError, match="beyond the block-table row"):
        _prefill(s, out, [(0, 0, 2, 129)])
    with pytest.raises(ValueError):
        _prefill(s, out, [(3, 0, 2, 100)])
    with pytest.raises(ValueError):
        _prefill(s, out, [(0, 1, 4, 100)])
    with pytest.raises(RuntimeError):                    # the status word is written by the kernel
        _prefill(s, out, [(0, 0, 2, 100)], workspace=s["ws"].cpu())
    with pytest.raises(ValueError, match="workspace"):
        _prefill(s, out, [(0, 0, 2, 100)], workspace=s["ws"][:32])
    with pytest.raises(_lib.HkvError):
        _prefill(s, out, [(0, 0, 2, 100)], workspace=s["ws"][4:])
    assert not out.any()


def test_the_current_stream_is_used():
    """a launch on a side stream waits for that stream's work, not for the default stream's"""
    s = _state()
    K.write(s["k"], s["v"], s["flat"], s["strides"], PS, s["slots"], s["g"], s["g"])
    want = _decode(s, torch.zeros_like(s["q"])).clone()
    torch.cuda.synchronize()
    side, q, out = torch.cuda.Stream(), s["q"].clone(), torch.zeros_like(s["q"])
    s["q"].zero_()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        torch.cuda._sleep(20_000_000)
        s["q"].copy_(q)
        _decode(s, out)
    side.synchronize()
    assert torch.equal(out, want)


@pytest.mark.parametrize("order", ["heads", "positions"])
@pytest.mark.parametrize("opt", ["", "HAD", "K8"])
@pytest.mark.parametrize("flat_rows", [True, False])
def test_layer_calls_give_the_same(monkeypatch, order, opt, flat_rows):
    """the backend's cache update and decode on the engine's own tensors, (tokens, heads * D) or (tokens, heads, D), new keys
    and values as slices of one projection, fewer step tokens than rows: the same bytes and bits as through views and the
    wrappers; what has another form is left to those, which serve or refuse it"""
    if opt == "K8" and order == "positions":
        pytest.skip("the K8V4 decode takes head-major pages only")
    for name in ("HAD", "K8"):
        monkeypatch.setenv(f"HORIZON_KVFP4_{name}", "1" if name == opt else "0")
    D, k8 = 256 if opt == "K8" else 128, opt == "K8"
    impl = BE.HorizonFp4Impl(KVH * G, D, D ** -0.5, num_kv_heads=KVH, kv_cache_dtype="nvfp4", max_num_seqs=8)
    layer = SimpleNamespace(_k_scale_float=0.01, _v_scale_float=0.02)
    slot, heads = (Lt.k8_slot_bytes(D), KVH) if k8 else (Lt.slot_bytes(D), 2 * KVH)
    shape = (24, heads, PS, slot) if order == "heads" else (24, PS, heads, slot)
    n = 200
    kv = torch.randn(n, 2 * KVH * D, device="cuda").to(torch.bfloat16)
    k, v = kv[:, :KVH * D], kv[:, KVH * D:]
    q = torch.randn(B + 2, KVH * G * D, device="cuda").to(torch.bfloat16)
    if not flat_rows:
        k, v, q = k.view(n, KVH, D), v.view(n, KVH, D), q.view(B + 2, KVH * G, D)
    slots = torch.randperm(24 * PS, device="cuda")[:n - 3]
    meta = SimpleNamespace(num_reqs=B, num_actual_tokens=B, has_decode=True, prefill_rows=[], qlmax=1,
                           block_table=torch.arange(24, dtype=torch.int32, device="cuda").view(B, 8),
                           seq_lens=torch.tensor([100, 7, 128], dtype=torch.int32, device="cuda"),
                           query_start_loc=torch.arange(B + 1, dtype=torch.int32, device="cuda"))
    h, answers = _lib.host(), []

    def logical(phys):
        return phys if order == "heads" else phys.permute(0, 2, 1, 3)

    def step(native):
        def call(name):
            def f(*a):
                answers.append(getattr(h, name)(*a) if native else None)
                return answers[-1]
            return staticmethod(f)
        monkeypatch.setattr(_lib, "_host", type("H", (), dict(
            layer_write=call("layer_write"), layer_decode=call("layer_decode"), write=staticmethod(h.write),
            decode=staticmethod(h.decode), prefill=staticmethod(h.prefill))))
        phys, out = torch.zeros(shape, dtype=torch.uint8, device="cuda"), torch.zeros_like(q)
        impl.do_kv_cache_update(layer, k, v, logical(phys), slots)
        assert impl.forward(layer, q, k, v, logical(phys), meta, out) is out
        return phys, out

    want, got = step(False), step(True)
    assert answers == [None, None, 0, 0]
    assert torch.equal(want[0], got[0]) and want[0].any()
    assert torch.equal(want[1], got[1]) and want[1][:B].any() and not want[1][B:].any()
    cache = logical(got[0])
    args = [k, v, cache, slots, impl._gk, impl._gv, D, True, None, k8]
    wide = logical(torch.zeros(*shape[:3], 2 * slot, dtype=torch.uint8, device="cuda"))[..., ::2]
    for i, bad in ((0, k.float()), (1, v[:-1]), (2, cache[:, 1:]), (2, wide), (3, slots.int()), (4, impl._gk[:1]), (6, 64),
                   (8, impl._gk)):
        assert h.layer_write(*args[:i], bad, *args[i + 1:]) is None
    with pytest.raises(ValueError):
        impl.do_kv_cache_update(layer, k, v, cache[:, 1:], slots)
    with pytest.raises(TypeError):
        impl.forward(layer, q.float(), k, v, cache, meta, torch.zeros_like(q))
    with pytest.raises(ValueError):
        impl.forward(layer, q, k, v, cache, meta, torch.zeros_like(q)[:1])
