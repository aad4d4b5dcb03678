"""A host thread that has made no CUDA call yet calls an op on buffers the allocator already holds (what an autograd
thread does from the second step on): the same result as on the thread that set everything up."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["v6", "v5", "v4", "block"])
def test_op_on_a_thread_that_is_new_to_cuda(kind):
    import rwkv_infctx_trainer_b200 as W
    B, T, H = 2, 130, 2
    C = H * 64
    bf = lambda *s: torch.randn(s, device="cuda").bfloat16()
    r, k, v, gy = (bf(B, T, C) for _ in range(4))
    u, s0 = bf(H, 64), torch.randn((B, H, 64, 64), device="cuda")
    if kind == "v6":
        w = bf(B, T, C)
        call = lambda: W.WKV6.apply(B, T, C, H, r, k, v, w, u, s0)
    elif kind == "v5":
        w = -torch.rand((H, 64), device="cuda")
        call = lambda: W.WKV5.apply(B, T, C, H, r, k, v, w, u, s0)
    elif kind == "v4":
        w, s4 = -torch.rand(C, device="cuda"), torch.rand((B, C, 3), device="cuda")
        call = lambda: W.wkv_op(w, u.flatten(), k, v, s4)
    else:
        blk = W.RWKV_TimeMix6_0(1, 4, C, H, 64, C).cuda().bfloat16()
        shift = bf(B, C)
        call = lambda: (blk(r, (shift, s0))[0],)

    def step():
        x = v if kind != "block" else r
        x.requires_grad_(True)
        y = call()[0]
        return y.detach(), torch.autograd.grad(y, x, gy)[0]

    step()
    want = step()          # (both buffers of a step are in the allocator's cache now)
    got = []

    def work():
        try:
            with torch.no_grad():
                got.append(call()[0])
            got.extend(step())
        except Exception as e:      # noqa: BLE001 (handed to the test's own thread)
            got.append(e)

    t = threading.Thread(target=work)
    t.start()
    t.join()
    assert not isinstance(got[-1], Exception), got[-1]
    torch.cuda.synchronize()
    for a, b in zip(got, (want[0],) + want):
        assert torch.equal(a, b)
