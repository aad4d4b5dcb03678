"""The low-rank maps of a decoded v6 token go through tanh: its bf16 result is tanh in 64 bits rounded once, from the
smallest values to saturation."""
import ctypes

import pytest
import torch

import test_decode_alignment as DA
from rwkv_infctx_trainer_b200 import _lib as L

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


@pytest.mark.parametrize("M", [1, 3])
def test_tanh_of_the_low_rank_map(M):
    """x has a single 1, so that a column's sum is one weight: 160 magnitudes per call, both signs, from 1e-37 to 30"""
    lib = L.load()
    lib.wkvx_decode6.argtypes = [ctypes.c_void_p, ctypes.c_void_p]
    H, C, R, DR = 2, 128, 32, 64
    z = lambda *s, dt=BF: torch.zeros(s, device="cuda", dtype=dt)
    mags = torch.cat((torch.logspace(-37, -6, 80), torch.logspace(-6, 1.48, 80))).double()
    for sign in (1.0, -1.0):
        t = dict(x=z(M, C), shift=z(M, C), maa_x=z(C), w1=z(C, 5 * R), w2=z(5, R, C), decay=z(C), d1=z(C, DR), d2=z(DR, C), u=z(H, 64),
                 ln_w=z(C), ln_b=z(C), state_in=z(M, H, 64, 64, dt=torch.float32), t1=z(M, 5 * R), xs=z(5, M, C), rkvg=z(4, M, C),
                 dd=z(M, DR), normed=z(M, C), out=z(M, C), new_shift=z(M, C), state_out=z(M, H, 64, 64, dt=torch.float32))
        t["x"][:, 5] = 1
        t["w1"][5] = (sign * mags).to("cuda", BF)
        t["d1"][5] = (sign * mags[40:40 + DR]).to("cuda", BF)
        mixes, proj = [z(C) for _ in range(5)], [z(C, C) for _ in range(5)]
        a = DA.Decode6(M=M, H=H, rank=R, decay_rank=DR, maa_dtype=L.WKV_BF16, ln_dtype=L.WKV_BF16, eps=1e-3)
        for n, x in t.items():
            setattr(a, n, x.data_ptr())
        for i in range(5):
            a.maa[i], a.proj[i] = mixes[i].data_ptr(), proj[i].data_ptr()
        assert lib.wkvx_decode6(ctypes.addressof(a), torch.cuda.current_stream().cuda_stream) == 0
        torch.cuda.synchronize()
        for got, w in ((t["t1"], t["w1"][5]), (t["dd"], t["d1"][5])):
            want = torch.tanh(w.double()).expand_as(got)
            # bf16 has 8 significant bits: half a step is at most 2^-8 of the value (just above a power of two), and the
            # fp32 value in front of the rounding is a few 2^-24 off
            bad = (got.double() - want).abs() > want.abs() * (2.0 ** -8 + 2.0 ** -20)
            assert not bad.any(), [(float(x), float(y)) for x, y in zip(want[bad][:5], got[bad][:5])]
