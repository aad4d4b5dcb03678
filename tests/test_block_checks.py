"""The time-mix blocks look at their arguments before they launch anything.  Shapes are looked at before
devices, so most of this runs without a GPU: a call that would read or write out of range raises ValueError."""
import pytest
import torch

BLOCKS = {4: "RWKV_TimeMix_v4", 5: "RWKV_TimeMix", 6: "RWKV_TimeMix6_0"}
C, H, B = 128, 2, 3


def make(version, device="cpu"):
    import rwkv_infctx_trainer_b200 as W
    torch.manual_seed(version)
    cls = getattr(W, BLOCKS[version])
    return (cls(1, 4, C, C) if version == 4 else cls(1, 4, C, H, 64, C)).to(device)


def call(version, blk, x, shift, state):
    import rwkv_infctx_trainer_b200 as W
    return blk(x, W.TimeMixState(shift, state) if version == 4 else (shift, state))


def good_state(version, device="cpu"):
    return torch.zeros((B, C, 3) if version == 4 else (B, H, 64, 64), device=device)


@pytest.mark.parametrize("version", [4, 5, 6])
@pytest.mark.parametrize("T", [1, 20])
@pytest.mark.parametrize("grad", [False, True])
def test_state_of_another_size_is_refused(version, T, grad):
    blk = make(version)
    x, shift = torch.zeros((B, T, C)), torch.zeros((B, C))
    ok = good_state(version)
    with torch.set_grad_enabled(grad):
        for bad in (ok[:1], torch.cat((ok, ok)), ok[:, :1], ok[..., :1]):
            with pytest.raises(ValueError, match="wkv state"):
                call(version, blk, x, shift, bad)
        with pytest.raises(RuntimeError, match="CUDA"):      # the right one gets as far as the device check
            call(version, blk, x, shift, ok)


def _param(blk, name):
    owner, _, leaf = name.rpartition(".")
    return (blk.get_submodule(owner) if owner else blk), leaf


@pytest.mark.parametrize("version", [4, 5, 6])
@pytest.mark.parametrize("T", [1, 20])
def test_width_or_parameter_of_another_size_is_refused(version, T):
    blk = make(version)
    state = good_state(version)
    with torch.no_grad():
        for width in (C - 64, C + 64, C + 1):        # an input of another width than the parameters
            with pytest.raises(ValueError):
                call(version, blk, torch.zeros((B, T, width)), torch.zeros((B, width)), state)
        x, shift = torch.zeros((B, T, C)), torch.zeros((B, C))
        for name, p in list(blk.named_parameters()):  # one parameter with an element (or row) missing
            owner, leaf = _param(blk, name)
            flat = p.dim() < 2 or p.shape[0] == 1 or name == "time_faaaa" or (version == 5 and name == "time_decay")
            setattr(owner, leaf, torch.nn.Parameter(p.detach().flatten()[1:] if flat else p.detach()[1:]))
            with pytest.raises(ValueError):
                call(version, blk, x, shift, state)
            setattr(owner, leaf, p)
        with pytest.raises(RuntimeError, match="CUDA"):
            call(version, blk, x, shift, state)


@pytest.mark.gpu
@pytest.mark.parametrize("version", [4, 5, 6])
def test_parameter_on_another_device_is_refused(version):
    """every parameter, not the first alone: one left on the host raises before any kernel sees its address"""
    blk = make(version, "cuda")
    x, shift, state = torch.zeros((B, 1, C), device="cuda"), torch.zeros((B, C), device="cuda"), good_state(version, "cuda")
    with torch.no_grad():
        for name, p in list(blk.named_parameters()):
            owner, leaf = _param(blk, name)
            setattr(owner, leaf, torch.nn.Parameter(p.detach().cpu()))
            with pytest.raises(RuntimeError, match="CUDA"):
                call(version, blk, x, shift, state)
            setattr(owner, leaf, p)
        call(version, blk, x, shift, state)


@pytest.mark.gpu
@pytest.mark.parametrize("version", [4, 5, 6])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_parameters_that_are_slices_of_a_flat_buffer(version, dtype):
    """every parameter one element past a 16-byte boundary: a training segment gives what it gives with the
    parameters in buffers of their own"""
    x, gy = torch.randn((B, 20, C), device="cuda").bfloat16(), torch.randn((B, 20, C), device="cuda").bfloat16()
    shift, state = torch.randn((B, C), device="cuda").bfloat16(), torch.ones_like(good_state(version, "cuda"))
    blk = make(version, "cuda").to(dtype)

    def run():
        out = call(version, blk, x, shift, state)[0]
        params = [p for _, p in sorted(blk.named_parameters())]
        return [out] + list(torch.autograd.grad(out, params, gy))

    want = run()
    for name, p in list(blk.named_parameters()):
        owner, leaf = _param(blk, name)
        buf = torch.empty(p.numel() + 8, device="cuda", dtype=dtype)
        odd = buf[1:1 + p.numel()].view(p.shape)
        odd.copy_(p.detach())
        setattr(owner, leaf, torch.nn.Parameter(odd))
        assert getattr(owner, leaf).data_ptr() % 16 != 0
    rel = lambda a, b: float((a.float() - b.float()).norm() / b.float().norm().clamp_min(1e-30))
    for a, b in zip(run(), want):
        assert a.shape == b.shape and rel(a.detach(), b.detach()) < 1e-2      # (a library GEMM may pick another kernel for such an operand)


@pytest.mark.gpu
@pytest.mark.parametrize("version", [5, 6])
@pytest.mark.parametrize("T", [1, 20])
@pytest.mark.parametrize("shape", [(B * H, 64, 64), (B * H, 1, 64, 64), (B, H * 64 * 64)])
def test_state_of_the_same_size_in_another_shape(version, T, shape):
    """the state is taken by its elements; what comes back is [B,H,64,64], and its gradient has the shape it was given in"""
    blk = make(version, "cuda").bfloat16()
    x, shift = torch.randn((B, T, C), device="cuda").bfloat16(), torch.randn((B, C), device="cuda").bfloat16()
    state = torch.randn((B, H, 64, 64), device="cuda")
    with torch.no_grad():
        want, (_, ws) = call(version, blk, x, shift, state)
        got, (_, s) = call(version, blk, x, shift, state.view(shape))
        assert s.shape == ws.shape == (B, H, 64, 64) and torch.equal(got, want) and torch.equal(s, ws)
    grads = []
    for st in (state, state.view(shape)):
        leaf = st.clone().requires_grad_(True)
        out, (_, s) = call(version, blk, x, shift, leaf)
        grads += torch.autograd.grad((out, s), leaf, (torch.ones_like(out), torch.ones_like(s)))
    assert grads[1].shape == shape and torch.equal(grads[0].view(shape), grads[1])
