"""The native side of the host wrappers (csrc/hkv_host.cpp) against their Python path: the same bytes and bits for
arguments that only the latter takes, the same refusals, the current stream."""
import pytest
import torch

from horizon_kernels_b200 import _lib
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
