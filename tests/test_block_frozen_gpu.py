"""A block's backward pass forms the gradients that are asked for: the same bits as the full pass gives, and no
matrix product whose result nobody wants.  (v4 without the state's gradient: the kernel carries the gradient between
its tiles with another exponent then, so a bf16 result may fall to the other side of a rounding here and there.)"""
import pytest
import torch

import test_block_checks as BC

pytestmark = pytest.mark.gpu
PROJ = {4: ("key", "value", "receptance", "output"), 5: ("receptance", "key", "value", "gate", "output"),
        6: ("receptance", "key", "value", "gate", "output")}


def backward(version, blk, leaves, x, shift, state, gy, gs):
    """gradients of `leaves` and the names of the operators the backward pass ran"""
    out = BC.call(version, blk, x, shift, state)
    s = out[1].wkv_state if version == 4 else out[1][1]
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]) as prof:
        g = torch.autograd.grad((out[0], s), leaves, (gy, gs))
        torch.cuda.synchronize()
    ops = {e.key: e.count for e in prof.key_averages()}
    return g, ops.get("aten::mm", 0) + ops.get("aten::bmm", 0)


@pytest.mark.parametrize("version", [4, 5, 6])
def test_only_what_is_asked_for_is_formed(version):
    B, C, H, T = BC.B, BC.C, BC.H, 70
    blk = BC.make(version, "cuda").bfloat16()
    with torch.no_grad():
        for n, p in blk.named_parameters():
            if "w1" in n or "w2" in n:
                p.normal_(0, 0.1)
    x, gy = torch.randn((B, T, C), device="cuda").bfloat16(), torch.randn((B, T, C), device="cuda").bfloat16()
    shift = torch.randn((B, C), device="cuda").bfloat16()
    state = BC.good_state(version, "cuda")
    state = torch.rand_like(state) + 0.5
    gs = torch.randn_like(state) * 0.1
    shared = {"x": x, "shift": shift, "state": state}
    params = dict(blk.named_parameters())

    def run(wanted):
        for n, t in {**params, **shared}.items():
            t.requires_grad_(n in wanted)
        leaves = [params[n] if n in params else shared[n] for n in wanted]
        g, n = backward(version, blk, leaves, x, shift, state, gy, gs)
        return dict(zip(wanted, g)), n

    def same(a, b, wanted):
        if version == 4 and "state" not in wanted:
            return float((a.float() - b.float()).norm() / b.float().norm()) < 2.0 ** -9
        return torch.equal(a, b)

    everything = list(shared) + list(params)
    full, products = run(everything)
    proj = [n + ".weight" for n in PROJ[version]]
    for wanted, fewer in (([n for n in everything if n not in proj], len(proj)),      # frozen projections
                          (["x"], None), (["shift"], None), (["state"], None)):
        got, n = run(wanted)
        for k, g in got.items():
            assert same(g, full[k], wanted), (wanted, k)
        assert n == products - fewer if fewer else n < products - len(proj) + 1, (wanted, n, products)
    for name in params:                                                               # each parameter alone
        got, n = run([name])
        assert same(got[name], full[name], [name]), name
        assert n < products, (name, n, products)
    assert run(["output.weight"])[1] == 1       # nothing behind the last product is wanted
