"""The decode kernels read 16 bytes at a time: a pointer that does not start on 16 bytes is an error code before
anything is launched, and a block whose weights do not start there runs on the library path."""
import ctypes

import pytest
import torch

import rwkv_infctx_trainer_b200._lib as L

_vp, _i, _f = ctypes.c_void_p, ctypes.c_int, ctypes.c_float


class Decode6(ctypes.Structure):        # wkvx_decode6_t of csrc/wkv_internal.h
    _fields_ = ([(n, _i) for n in ("M", "H", "rank", "decay_rank")] + [("x", _vp), ("shift", _vp), ("maa_x", _vp), ("maa", _vp * 5), ("maa_dtype", _i)]
                + [(n, _vp) for n in ("w1", "w2", "decay", "d1", "d2", "u")] + [("proj", _vp * 5), ("ln_w", _vp), ("ln_b", _vp), ("ln_dtype", _i), ("eps", _f)]
                + [(n, _vp) for n in ("state_in", "t1", "xs", "rkvg", "dd", "normed", "out", "new_shift", "state_out")])


class Decode5(ctypes.Structure):        # wkvx_decode5_t
    _fields_ = ([(n, _i) for n in ("M", "H", "C")] + [("x", _vp), ("shift", _vp), ("mix", _vp * 4), ("mix_dtype", _i), ("decay", _vp), ("decay_dtype", _i),
                ("u", _vp), ("proj", _vp * 5), ("ln_w", _vp), ("ln_b", _vp), ("ln_dtype", _i), ("eps", _f)]
                + [(n, _vp) for n in ("state_in", "rkvg", "normed", "out", "new_shift", "state_out")])


@pytest.mark.skipif(torch.cuda.is_available(), reason="made-up addresses: for a machine where nothing could be launched on them")
@pytest.mark.parametrize("version", [5, 6])
def test_misaligned_pointer_is_an_error_code(version):
    lib = L.load()
    a = Decode6(M=1, H=2, rank=32, decay_rank=64) if version == 6 else Decode5(M=1, H=2, C=128)
    fn = lib.wkvx_decode6 if version == 6 else lib.wkvx_decode5
    fn.argtypes = [_vp, _vp]
    base = 1 << 20
    for name, ty in a._fields_:
        if ty is _vp:
            setattr(a, name, base)
        elif ty not in (_i, _f):
            setattr(a, name, ty(*[base] * ty._length_))
    wide = ["x", "shift", "state_in", "rkvg", "normed", "new_shift", "state_out"] + (["w1", "w2", "d1", "xs"] if version == 6 else [])
    for name in wide:
        setattr(a, name, base + 2)
        assert fn(ctypes.addressof(a), None) == 4, name
        setattr(a, name, base)
    for i in range(5):
        a.proj[i] = base + 8
        assert fn(ctypes.addressof(a), None) == 4, i
        a.proj[i] = base


@pytest.mark.gpu
@pytest.mark.parametrize("cls", ["RWKV_TimeMix6_0", "RWKV_TimeMix"])
def test_weights_that_start_on_an_odd_element(cls):
    """one decoded token of a block whose projections sit at odd offsets of larger buffers, against the same block with
    its own storage (the two run on different kernels: bf16 roundings of one projection apart)"""
    import rwkv_infctx_trainer_b200 as W
    C, H, B = 256, 4, 2
    torch.manual_seed(5)
    blk = getattr(W, cls)(1, 4, C, H, 64, C).cuda().bfloat16()
    x = torch.randn((B, 1, C), device="cuda").bfloat16()
    state = (torch.randn((B, C), device="cuda").bfloat16(), torch.randn((B, H, 64, 64), device="cuda"))
    rel = lambda a, b: float((a.float() - b.float()).norm() / b.float().norm())
    with torch.no_grad():
        want, (_, ws) = blk(x, state)
        for lin in (blk.receptance, blk.key, blk.value, blk.gate, blk.output):
            buf = torch.empty(C * C + 8, device="cuda", dtype=torch.bfloat16)
            odd = buf[1:1 + C * C].view(C, C)
            odd.copy_(lin.weight)
            assert odd.data_ptr() % 16 == 2 and odd.is_contiguous()
            lin.weight = torch.nn.Parameter(odd)
        got, (_, s) = blk(x, state)
    assert rel(got, want) < 1e-2 and rel(s, ws) < 5e-3
