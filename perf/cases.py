"""The performance cases of this package: what its users have it do, through its public entry points.

Each case is one dict of plain values; ``path`` says which entry point it goes through and the rest are its sizes and
options.  ``listed()`` holds one named case per kind of use, ``draw()`` gives further ones from the same ranges,
``prepare()`` makes what a caller holds before the call, ``run()`` is one pass, ``work()`` the bytes and operations
that no implementation of the pass can avoid and ``tolerance()`` how far two correct ones may lie apart.

Paths:
  causal      ``cos_attn_causal`` forward + backward on ``[B, H, N, D]`` tensors (training and long-context prefill)
  gpt         ``cos_attn_causal_packed`` forward + backward: the attention call of a decoder layer on its QKV projection
  bert        ``cos_attn_bidirectional_packed`` forward + backward: the same of an encoder layer
  dropin      ``CustomAttention`` forward + backward: the operator of the extension this package replaces
  prompt      ``CosAttnDecodeState.prefill``: outputs of a prompt and the recurrent state it leaves
  decode      ``CosAttnDecodeState.step`` with one token per sequence
"""
import math

import torch
import torch.nn.functional as F

from cottention_transformer_b200 import (CosAttnDecodeState, CustomAttention, cos_attn_bidirectional_packed, cos_attn_causal,
                                         cos_attn_causal_packed)

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}


def listed():
    return [
        # the smallest training call: a short sequence of a small model; launches and host work count here
        dict(name="causal_small", path="causal", B=1, H=4, N=200, D=64, dtype="bf16", mask=False),
        # the operator at its benchmark size: a batch of 4k-token sequences, 16 heads of 64
        dict(name="causal_4k", path="causal", B=8, H=16, N=4096, D=64, dtype="bf16", mask=False),
        # a padded batch whose length is no multiple of any tile, in fp16, with a head count that does not fill the GPU
        dict(name="causal_padded", path="causal", B=7, H=12, N=1531, D=64, dtype="fp16", mask=True),
        # one attention layer of a 24 x 1024 decoder in training: batch 8 of 1024 tokens, rotary embedding on q and k
        dict(name="gpt_layer", path="gpt", B=8, H=16, N=1024, D=64, dtype="bf16", mask=False, rotary=64),
        # one attention layer of a base-size encoder in training: batch 32 of 512 tokens, padded
        dict(name="bert_layer", path="bert", B=32, H=12, N=512, D=64, dtype="bf16", mask=True),
        # long-context training of one sequence, both head dims
        dict(name="long_d64", path="causal", B=1, H=16, N=65536, D=64, dtype="bf16", mask=False),
        dict(name="long_d128", path="causal", B=1, H=16, N=16384, D=128, dtype="bf16", mask=False),
        # the replaced extension's own operator in a bf16 training step
        dict(name="dropin_bf16", path="dropin", B=8, H=16, N=1024, D=64, dtype="bf16"),
        # the same module math in fp32, the mode that is used to check a model
        dict(name="causal_fp32", path="causal", B=2, H=8, N=1024, D=64, dtype="fp32", mask=False),
        # serving: a prompt is absorbed, then one token per sequence and step
        dict(name="prompt", path="prompt", B=4, H=16, N=777, D=64, dtype="bf16"),
        dict(name="decode_d64", path="decode", B=64, H=16, N=1, D=64, dtype="bf16"),
        dict(name="decode_d128", path="decode", B=64, H=16, N=1, D=128, dtype="bf16"),
    ]


def _log(rng, lo, hi):
    """An integer between lo and hi, spread over its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case.  The row count B * H * N is kept at or under that of the largest listed case of the path."""
    path = rng.choice(["causal", "causal", "padded", "long", "gpt", "bert", "dropin", "fp32", "prompt", "decode"])
    half = rng.choice(["bf16", "bf16", "fp16"])
    if path in ("causal", "padded"):
        H, N = rng.choice([4, 6, 8, 12, 16]), _log(rng, 64, 4096)
        B = _log(rng, 1, max(1, min(16, 524288 // (H * N))))
        return dict(path="causal", B=B, H=H, N=N, D=64, dtype=half, mask=path == "padded")
    if path == "long":
        D, H = rng.choice([64, 128]), rng.choice([8, 12, 16])
        return dict(path="causal", B=1, H=H, N=_log(rng, 8192, (1048576 if D == 64 else 262144) // H), D=D, dtype=half, mask=False)
    if path == "gpt":
        H, N = rng.choice([8, 12, 16]), _log(rng, 128, 1638)
        # (batches that fill the GPU: below that the rotary embedding works in place on the caller's tensor, which these
        # inputs, kept from pass to pass, do not allow)
        B = _log(rng, -(-75 // H), 262144 // (16 * N))
        return dict(path="gpt", B=B, H=H, N=N, D=64, dtype=half, mask=rng.random() < 0.3, rotary=rng.choice([0, 32, 64]))
    if path == "bert":
        H = rng.choice([8, 12, 16])
        return dict(path="bert", B=_log(rng, 1, 32), H=H, N=_log(rng, 32, 512), D=64, dtype=half, mask=rng.random() < 0.7)
    if path == "dropin":
        D, H, N = rng.choice([64, 64, 128]), rng.choice([8, 12, 16]), _log(rng, 128, 2048)
        B = _log(rng, 1, max(1, min(16, 131072 * 64 // (D * H * N))))
        return dict(path="dropin", B=B, H=H, N=N, D=D, dtype=half)
    if path == "fp32":
        return dict(path="causal", B=rng.choice([1, 2]), H=rng.choice([4, 8]), N=_log(rng, 64, 1024), D=rng.choice([32, 64]), dtype="fp32",
                    mask=rng.random() < 0.5)
    if path == "prompt":
        return dict(path="prompt", B=_log(rng, 1, 8), H=rng.choice([8, 12, 16]), N=_log(rng, 20, 2000), D=rng.choice([64, 64, 128]), dtype=half)
    return dict(path="decode", B=_log(rng, 1, 64), H=rng.choice([8, 12, 16]), N=1, D=rng.choice([64, 128]), dtype=rng.choice(["bf16", "fp16", "fp32"]))


def _keep(B, N, gen):
    """Right padding, as a batch of sentences of different lengths has it: True = a real position (at least one each)."""
    lengths = torch.randint(max(1, N // 2), N + 1, (B, 1), device="cuda", generator=gen)
    return torch.arange(N, device="cuda").unsqueeze(0) < lengths


def prepare(case, seed):
    B, H, N, D, dt = case["B"], case["H"], case["N"], case["D"], DTYPES[case["dtype"]]
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def randn(*shape):
        return torch.randn(*shape, device="cuda", dtype=dt, generator=gen)

    path = case["path"]
    st = dict(path=path)
    # the learned exponent: its initial value 0.5 and what training makes of it
    st["nc"] = 0.5 + 0.2 * torch.randn(1, H, 1, 1, device="cuda", generator=gen)
    st["keep"] = _keep(B, N, gen) if case.get("mask") else None
    if path in ("gpt", "bert"):
        st["qkv"] = randn(B, N, 3, H, D).requires_grad_()
        st["dout"] = randn(B, N, H, D)
        st["rotary"] = None
        if case.get("rotary"):
            half = case["rotary"] // 2
            angle = torch.arange(N, device="cuda").float()[:, None] * 10000.0 ** (-torch.arange(half, device="cuda").float() / half)
            st["rotary"] = (torch.sin(angle), torch.cos(angle))
    elif path in ("prompt", "decode"):
        st["q"], st["k"], st["v"] = randn(B, H, N, D), randn(B, H, N, D), randn(B, H, N, D)
        st["state"] = CosAttnDecodeState(B, H, D)
        if path == "decode":  # in the middle of a generation: some hundred tokens have gone into the state
            st["state"].state.copy_(torch.randn(B, H, D, D, device="cuda", generator=gen) * D ** -0.5)
            st["state"].cur_s = 300
    else:
        q, k, v = randn(B, H, N, D), randn(B, H, N, D), randn(B, H, N, D)
        if path == "dropin":  # the operator sees normalised q and k
            q, k = F.normalize(q, dim=-1), F.normalize(k, dim=-1)
        st["q"], st["k"], st["v"] = q.requires_grad_(), k.requires_grad_(), v.requires_grad_()
        st["dout"] = randn(B, H, N, D)
    if path in ("causal", "gpt", "bert"):
        st["nc"].requires_grad_()
    return st


def run(st):
    path = st["path"]
    if path == "causal":
        out = cos_attn_causal(st["q"], st["k"], st["v"], st["nc"], keep=st["keep"])
        return out, *torch.autograd.grad(out, (st["q"], st["k"], st["v"], st["nc"]), st["dout"])
    if path == "gpt":
        out = cos_attn_causal_packed(st["qkv"], st["nc"], keep=st["keep"], rotary=st["rotary"])
        return out, *torch.autograd.grad(out, (st["qkv"], st["nc"]), st["dout"])
    if path == "bert":
        out = cos_attn_bidirectional_packed(st["qkv"], st["nc"], keep=st["keep"])
        return out, *torch.autograd.grad(out, (st["qkv"], st["nc"]), st["dout"])
    if path == "dropin":
        out = CustomAttention.apply(st["q"], st["k"], st["v"])
        return out, *torch.autograd.grad(out, (st["q"], st["k"], st["v"]), st["dout"])
    state = st["state"]
    if path == "prompt":  # a new request in a slot that is used again
        state.reset()
        return state.prefill(st["q"], st["k"], st["v"], st["nc"]), state.state
    return state.step(st["q"], st["k"], st["v"], st["nc"]), state.state


def work(case):
    B, H, N, D = case["B"], case["H"], case["N"], case["D"]
    tensor = B * H * N * D * DTYPES[case["dtype"]].itemsize
    state = B * H * D * D * 4
    rows = B * H * N
    if case["path"] == "decode":
        # state read and written, q, k, v read, out written; the rank-one update and the product with q
        return {"bytes": 2 * state + 4 * tensor, "flops": 4 * rows * D * D}
    if case["path"] == "prompt":
        return {"bytes": 4 * tensor + state, "flops": 4 * rows * D * D}
    # q, k, v, dout in; out, dq, dk, dv out.  In the recurrent form each position updates a D x D state and multiplies with
    # it: once forward (2 products), and for dq (S again is kept or recomputed: not counted), dk, dv and the second state.
    return {"bytes": 8 * tensor, "flops": (4 + 8) * rows * D * D}


def tolerance(case):
    # Measured against the same math in float64 on the same rounded inputs: the worst output of each path is off by 3.8e-3
    # (bf16), 3.8e-4 (fp16) and 6e-7 (fp32; the gradient of norm_const, a signed sum with much cancellation), four times
    # that is stated.  `max` counts single values over the result's root mean square: the first positions of a causal
    # sequence are many times larger than the rest, and there 0.47, 0.095 and 9e-6 were seen.
    if case["dtype"] == "fp32":
        return {"rel": 5e-6, "max": 5e-5}
    return {"rel": 1.5e-2, "max": 0.95} if case["dtype"] == "bf16" else {"rel": 2e-3, "max": 0.4}
