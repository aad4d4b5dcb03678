"""What the speed of this package is measured on: the work a user has it do, through its public
entry points.

A case is one call chain of the WKV op or of a time-mix block:

  unit      "op"     the op itself: WKV6 / WKV5 (their `apply`), `wkv_op` (v4), or, with api
                     "dropin", the wrappers named as in the trainer this package serves
                     (RUN_WKV6STATE_CUDA / RUN_WKV5_CUDA, state updated in place)
            "block"  RWKV_TimeMix6_0 / RWKV_TimeMix / RWKV_TimeMix_v4 with bf16 parameters
  mode      "train"  forward over the segments with the state carried, then the gradients of
                     everything that has one
            "infer"  forward alone, without autograd (prefill; T = 1 is a decode step)
  T, segment         tokens of a row, and how many of them a call takes (the last may be shorter)
  truncated          "train" only: the backward pass of a segment runs right after its forward pass
                     and no gradient crosses a segment boundary
  dtype              of the activations (the state is fp32 always)
  B, H               rows; heads of 64 channels (v4: C = 64 H channels)

Distributions: r, k, v and the incoming gradients N(0, 1); v6 decay activation N(-0.6, 0.5) per
token; v5 decay parameter U(-6, -1) and v4 time_decay U(-5, 1) per channel; bonus U(-1, 1).
"""
import math

import torch

import rwkv_infctx_trainer_b200 as W

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
N = 64                                   # head size


def _case(name, unit, version, mode, B, T, H, segment=None, dtype="bf16", api="function", truncated=False):
    return {"name": name, "unit": unit, "version": version, "mode": mode, "B": B, "T": T, "H": H,
            "segment": segment or T, "dtype": dtype, "api": api, "truncated": truncated}


def listed():
    return [
        # training the 7B shape: the benchmark's headline workload, 4 BPTT segments, full gradient chain
        _case("v6_train_7b", "op", 6, "train", 4, 16384, 64, segment=4096),
        # what one of eight GPUs holds of the 3B shape's million-token stream: 5 of its 40 heads, one row,
        # truncated back-propagation (8 of the stream's 256 segments)
        _case("v6_stream_5_heads", "op", 6, "train", 1, 32768, 5, segment=4096, truncated=True),
        # training the v5 1.5B shape
        _case("v5_train_1b5", "op", 5, "train", 8, 4096, 32, segment=2048),
        # v4 at full precision
        _case("v4_train_fp32", "op", 4, "train", 8, 4096, 32, segment=2048, dtype="fp32"),
        # v4 in bf16 on rows whose length fits no tile
        _case("v4_train_ragged", "op", 4, "train", 3, 1001, 12),
        # the small fp32 job that numerics are checked on
        _case("v5_train_fp32_small", "op", 5, "train", 2, 512, 4, segment=128, dtype="fp32"),
        # the drop-in wrapper, with the segment lengths the v6 trainer cuts: ceil(T / 3) + 2, last one shorter
        _case("v6_dropin_ragged", "op", 6, "train", 2, 3001, 16, segment=1003, api="dropin"),
        # a prompt
        _case("v6_prefill", "op", 6, "infer", 1, 1999, 40),
        # one decode step of a small batch
        _case("v6_decode", "op", 6, "infer", 8, 1, 64),
        # a layer's time-mix block in training, one segment of the 3B shape
        _case("block6_train_3b", "block", 6, "train", 1, 4096, 40),
        # the same block, one decode step of one row
        _case("block6_decode", "block", 6, "infer", 1, 1, 40),
        # a small v5 model's block in training, short ragged rows
        _case("block5_train_small", "block", 5, "train", 3, 510, 12),
    ]


def draw(rng):
    def spread(lo, hi):
        return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))

    unit = rng.choice(["op", "op", "op", "block"])
    version = rng.choice([4, 5, 5, 6, 6, 6])
    mode = rng.choice(["train", "train", "infer"])
    dtype = "bf16" if unit == "block" else rng.choice(["bf16"] * 5 + ["fp32", "fp32", "fp16"])
    api = rng.choice(["function", "function", "dropin"]) if unit == "op" and version != 4 else "function"
    if mode == "infer" and rng.random() < 0.5:
        B, T, H, segments, truncated = spread(1, 64), 1, spread(1, 64), 1, False
    else:
        B, T, H = rng.randint(1, 8), spread(16, 16384), spread(1, 64)
        segments = rng.randint(1, 4) if mode == "train" and T >= 512 else 1
        truncated = segments > 1 and (api == "dropin" or rng.random() < 0.3)
    # no drawn case is larger than the largest listed one of its kind
    if unit == "block":
        fits = lambda: B * T * H * H <= 4096 * 40 * 40      # (the projections grow with the square of the width)
    elif dtype == "bf16" or version == 4:
        fits = lambda: B * T * H * (1 if dtype == "bf16" else 2) <= 4 * 16384 * 64 // (4 if version == 4 else 1)
    else:
        fits = lambda: T <= 1024 and B * T * H <= 64 * 1024  # full-precision v5 / v6: numerics checks
    while not fits():
        if T > 1024:
            T -= T // 3
        elif B > 1:
            B -= 1
        else:
            H -= 1 + H // 8
    segment = -(-T // segments) + (2 if segments > 1 else 0)
    case = _case("", unit, version, mode, B, T, H, segment, dtype, api, truncated)
    del case["name"]
    return case


# ---------------------------------------------------------------------------------------------
# inputs

def _segments(case):
    return [(t, min(case["T"], t + case["segment"])) for t in range(0, case["T"], case["segment"])]


def _op_inputs(case, g, train):
    B, H, version = case["B"], case["H"], case["version"]
    C, dt, dev = H * N, DTYPES[case["dtype"]], "cuda"

    def normal(*shape, mean=0.0, std=1.0, dtype=dt):
        return torch.randn(shape, generator=g, device=dev, dtype=torch.float32).mul_(std).add_(mean).to(dtype)

    def uniform(*shape, lo, hi, dtype):
        return torch.rand(shape, generator=g, device=dev).mul_(hi - lo).add_(lo).to(dtype)

    names = ("k", "v") if version == 4 else ("r", "k", "v")
    s = {"segs": []}
    for a, b in _segments(case):
        seg = {n: normal(B, b - a, C) for n in names}
        if version == 6:
            seg["w"] = normal(B, b - a, C, mean=-0.6, std=0.5)
        for t in seg.values():
            t.requires_grad_(train)
        if train:
            seg["gy"] = normal(B, b - a, C)
        s["segs"].append(seg)
    if version == 4:
        s["w"] = uniform(C, lo=-5.0, hi=1.0, dtype=torch.float32)
        s["u"] = uniform(C, lo=-1.0, hi=1.0, dtype=dt)
        # what a row carries after some text: (numerator, denominator, exponent)
        q = uniform(B, C, lo=0.5, hi=4.0, dtype=torch.float32)
        s["state"] = torch.stack((q * normal(B, C, std=0.5, dtype=torch.float32), q,
                                  normal(B, C, mean=1.0, std=0.5, dtype=torch.float32)), -1).contiguous()
    else:
        if version == 5:
            s["w"] = uniform(H, N, lo=-6.0, hi=-1.0, dtype=torch.float32)
        s["u"] = uniform(H, N, lo=-1.0, hi=1.0, dtype=dt)
        s["state"] = normal(B, H, N, N, std=0.5, dtype=torch.float32)
    for n in ("u", "w"):
        if n in s:
            s[n].requires_grad_(True)    # (parameters, under no_grad in inference)
    s["state"].requires_grad_(train and case["api"] == "function" and not case["truncated"])
    return s


_BLOCKS = {6: W.RWKV_TimeMix6_0, 5: W.RWKV_TimeMix}


def _block_inputs(case, g, train):
    B, H, version = case["B"], case["H"], case["version"]
    C, dev, bf = H * N, "cuda", torch.bfloat16

    def normal(*shape, std=1.0, dtype=bf):
        return torch.randn(shape, generator=g, device=dev).mul_(std).to(dtype)

    with torch.device(dev):
        block = W.RWKV_TimeMix_v4(1, 4, C, C) if version == 4 else _BLOCKS[version](1, 4, C, H, N, C)
    block = block.to(bf)
    with torch.no_grad():
        for name, p in block.named_parameters():     # (the constructor's values do not depend on the seed)
            if p.dim() >= 2 and p.shape[-1] > 1 and p.shape[0] > 1 and "faaaa" not in name and name != "time_decay":
                p.copy_(normal(*p.shape, std=0.02 if "w1" in name or "w2" in name else p.shape[-1] ** -0.5))
    state = normal(B, C), (torch.stack((normal(B, C, std=0.5, dtype=torch.float32),
                                        torch.ones(B, C, device=dev), torch.ones(B, C, device=dev)), -1).contiguous()
                           if version == 4 else normal(B, H, N, N, std=0.5, dtype=torch.float32))
    s = {"block": block, "state": state, "segs": []}
    for t in state:
        t.requires_grad_(train and not case["truncated"])
    for a, b in _segments(case):
        seg = {"x": normal(B, b - a, C).requires_grad_(train)}
        if train:
            seg["gy"] = normal(B, b - a, C)
        s["segs"].append(seg)
    return s


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    train = case["mode"] == "train"
    s = _block_inputs(case, g, train) if case["unit"] == "block" else _op_inputs(case, g, train)
    s["case"] = case
    return s


# ---------------------------------------------------------------------------------------------
# one pass

def _call_op(case, s, seg, state):
    """-> (y, state after the segment)"""
    version, B, C, H = case["version"], case["B"], case["H"] * N, case["H"]
    T = seg["k"].shape[1]
    if version == 4:
        y, state = W.wkv_op(s["w"], s["u"], seg["k"], seg["v"], state)
        return y, state
    w = seg["w"] if version == 6 else s["w"]
    if case["api"] == "dropin":          # (the state is updated in place)
        if version == 6:
            return W.RUN_WKV6STATE_CUDA(B, T, C, H, seg["r"], seg["k"], seg["v"], w, s["u"], state), state
        return W.RUN_WKV5_CUDA(B, T, C, H, state, seg["r"], seg["k"], seg["v"], w, s["u"]), state
    fn = W.WKV6 if version == 6 else W.WKV5
    return fn.apply(B, T, C, H, seg["r"], seg["k"], seg["v"], w, s["u"], state)


def _call_block(case, s, seg, state):
    if case["version"] == 4:
        out, state = s["block"](seg["x"], W.TimeMixState(*state))
        return out, (state.shift_state, state.wkv_state)
    return s["block"](seg["x"], state)


def _leaves(case, s, seg):
    if case["unit"] == "block":
        return [seg["x"]]
    return [seg[n] for n in ("r", "k", "v", "w") if n in seg]


def _shared_leaves(case, s):
    if case["unit"] == "block":
        return list(s["block"].parameters())
    return [s[n] for n in ("u", "w") if n in s]


def run(s):
    case = s["case"]
    call = _call_block if case["unit"] == "block" else _call_op
    state = s["state"]
    if case["mode"] == "infer":
        with torch.no_grad():
            if case["api"] == "dropin":
                state = state.clone()
            out = []
            for seg in s["segs"]:
                y, state = call(case, s, seg, state)
                out.append(y)
            return out, state

    if case["api"] == "dropin":
        state = state.clone()
    shared = _shared_leaves(case, s)
    ys, grads = [], []
    if case["truncated"]:
        for seg in s["segs"]:
            y, state = call(case, s, seg, state)
            state = tuple(t.detach() for t in state) if isinstance(state, tuple) else state.detach()
            grads.append(torch.autograd.grad(y, _leaves(case, s, seg) + shared, seg["gy"]))
            ys.append(y.detach())
        # (what a trainer accumulates over the segments: the parameters' gradients)
        n = len(shared)
        total = [sum(g[len(g) - n + i] for g in grads) for i in range(n)]
        return ys, state, [g[:len(g) - n] for g in grads], total
    leaves = list(shared)
    for seg in s["segs"]:
        y, state = call(case, s, seg, state)
        ys.append(y)
        leaves += _leaves(case, s, seg)
    carried = [t for t in (s["state"] if isinstance(s["state"], tuple) else (s["state"],)) if t.requires_grad]
    grads = torch.autograd.grad(ys, leaves + carried, [seg["gy"] for seg in s["segs"]])
    return [y.detach() for y in ys], (state if isinstance(state, tuple) else (state,)), grads


# ---------------------------------------------------------------------------------------------
# what a pass cannot do without

def work(case):
    """Bytes: the forward pass reads its inputs and writes y and the state once, the backward pass reads
    its inputs (the forward's and the incoming gradient) and writes the gradients once.  Operations:
    v5 / v6 in the chunked form with the chunk length L = min(64, tokens of a call): 4 L N + 4 N^2 per head and
    token forward, 10 L N + 8 N^2 backward."""
    B, T, H, version = case["B"], case["T"], case["H"], case["version"]
    C, size, train = H * N, DTYPES[case["dtype"]].itemsize, case["mode"] == "train"
    nseg = len(_segments(case))
    L = min(64, case["segment"])
    state = B * C * 3 * 4 if version == 4 else B * H * N * N * 4
    tc = B * T * C
    if case["unit"] == "op":
        fwd, bwd = {4: (3, 5), 5: (4, 7), 6: (5, 9)}[version]
        byts = fwd * tc * size + 2 * nseg * state + (bwd * tc * size + 3 * nseg * state if train else 0)
    else:
        params = (4 if version == 4 else 5) * C * C + (C * (5 * 32 * 2 + 64 * 2) if version == 6 else 0)
        byts = 2 * (2 * tc + params * nseg) + 2 * nseg * state
        if train:
            byts += 2 * (3 * tc + params * nseg + params) + 3 * nseg * state
    if version == 4:
        flops = (14 + (40 if train else 0)) * tc
    else:
        flops = (4 * L * N + 4 * N * N + (10 * L * N + 8 * N * N if train else 0)) * B * T * H
    if case["unit"] == "block":
        flops += 2 * params * B * T * (3 if train else 1)
    return {"bytes": byts, "flops": flops}


def tolerance(case):
    # fp32: sums of up to some hundred thousand terms in another order, decays through exp(-exp(.));
    # 16 bit: operands and results are rounded to 8 (11) bits; a block is a chain of such roundings
    if case["dtype"] == "fp32":
        return {"rel": 1e-4}
    return {"rel": 2e-2 if case["unit"] == "block" else 1e-2}
