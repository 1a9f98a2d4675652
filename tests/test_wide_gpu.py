"""The head-dim-128 kernels where their split can go wrong: segment and chunk edges, odd row counts, both widths."""
import pytest
import torch

from oracle import cott_oracle as O

pytestmark = pytest.mark.gpu

REL16 = {torch.bfloat16: 2e-2, torch.float16: 4e-3}  # 16-bit products of scores, state and output rows, several roundings deep


def _rel(a, b):
    return ((a.double().cpu() - b).norm() / b.norm()).item()


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("shape,masked", [((1, 1, 1), False), ((2, 3, 128), False), ((1, 2, 129), True),
                                          ((1, 1, 1001), False),  # segments, and B*H*N odd
                                          ((1, 3, 640), True), ((1, 5, 2500), False), ((2, 40, 300), True)])
def test_fused_128_matches_fp64(shape, masked, dt):
    from cottention_transformer_b200 import cos_attn_causal, _lib
    B, H, N = shape
    g = torch.Generator().manual_seed(N)
    q, k, v, do = (torch.randn(B, H, N, 128, generator=g).to(dt) for _ in range(4))
    nc = 0.5 + 0.2 * torch.randn(1, H, 1, 1, generator=g)
    keep = None
    if masked:
        keep = torch.rand(B, N, generator=g) < 0.7
        keep[:, 0] = True
    leaf = [t.cuda().requires_grad_() for t in (q, k, v, nc)]
    out = cos_attn_causal(*leaf, None if keep is None else keep.cuda())
    got = (out.detach(), *torch.autograd.grad(out, leaf, do.cuda()))
    _lib.check_device_status()
    ref = [t.double().requires_grad_() for t in (q, k, v, nc)]
    o = O.cos_attn_causal(*ref, keep=keep)
    want = (o.detach(), *torch.autograd.grad(o, ref, do.double()))
    for name, a, b in zip(("out", "dq", "dk", "dv"), got, want):
        if b.norm() < 1e-6 * b.numel() ** 0.5:  # (one position: dq and dk vanish, what is left is rounding of O(1) terms)
            assert a.double().cpu().norm() <= 4 * REL16[dt] * b.numel() ** 0.5, name
        else:
            assert _rel(a, b) <= REL16[dt], (name, _rel(a, b))
    # the gradient of norm_const is a sum of terms of both signs: measured against the sum of their magnitudes
    n = (torch.ones(B, N, dtype=torch.bool) if keep is None else keep).cumsum(-1).double()
    sig = torch.sigmoid(nc.double()).view(H)
    terms = (torch.log(n).view(B, 1, N) * (v.double() * want[3]).sum(-1)).abs().sum(dim=(0, 2)) * sig * (1 - sig)
    assert ((got[4].double().cpu() - want[4]).abs().view(H) <= REL16[dt] * terms.clamp(min=1e-3)).all()


@pytest.mark.parametrize("reverse", [False, True])
@pytest.mark.parametrize("H,N,Dv", [(2, 300, 64), (1, 2100, 64), (1, 2100, 128), (2, 700, 256), (1, 1000, 192)])
def test_scan_128_widths_and_segments(H, N, Dv, reverse):
    """Value dims that take one, two or three slices of either width, with and without segments."""
    from cottention_transformer_b200 import kernel, _lib
    g = torch.Generator().manual_seed(Dv + N)
    q, k = (torch.nn.functional.normalize(torch.randn(1, H, N, 128, generator=g), dim=-1).bfloat16() for _ in range(2))
    v = torch.randn(1, H, N, Dv, generator=g).bfloat16()
    got = kernel.bfloat16(q.cuda(), k.cuda(), v.cuda(), 1, False, reverse)
    _lib.check_device_status()
    assert _rel(got, O.scan_recurrent(q.double(), k.double(), v.double(), reverse, "f64")) <= REL16[torch.bfloat16]


@pytest.mark.parametrize("N", [1, 130, 777, 1500])
def test_prefill_state_128(N):
    from cottention_transformer_b200 import CosAttnDecodeState, _lib
    g = torch.Generator().manual_seed(N)
    q, k, v = (torch.randn(2, 3, N, 128, generator=g).bfloat16() for _ in range(3))
    nc = 0.5 + 0.2 * torch.randn(1, 3, 1, 1, generator=g)
    st = CosAttnDecodeState(2, 3, 128)
    st.prefill(q.cuda(), k.cuda(), v.cuda(), nc.cuda())
    _lib.check_device_status()
    n = torch.arange(1, N + 1).double().view(1, 1, N, 1)
    vp = v.double() / n ** torch.sigmoid(nc.double())
    want = torch.einsum("bhnj,bhni->bhji", vp, torch.nn.functional.normalize(k.double(), dim=-1))
    assert st.cur_s == N + 1 and _rel(st.state, want) <= REL16[torch.bfloat16]


@pytest.mark.parametrize("scale", [1e-9, 1e14, 1e18])
def test_fused_128_dq_of_long_and_short_rows(scale):
    """dq through the normalisation for rows whose 1/|q| is far from 1 (bf16 reaches that far): the part of the gradient
    along q cancels whatever |q| is."""
    from cottention_transformer_b200 import cos_attn_causal
    g = torch.Generator().manual_seed(7)
    q, k, v, do = (torch.randn(1, 2, 300, 128, generator=g).bfloat16() for _ in range(4))
    q = (q.float() * scale).bfloat16()
    nc = 0.5 + 0.2 * torch.randn(1, 2, 1, 1, generator=g)
    leaf = [t.cuda().requires_grad_() for t in (q, k, v, nc)]
    (dq,) = torch.autograd.grad(cos_attn_causal(*leaf), leaf[0], do.cuda())
    ref = [t.double().requires_grad_() for t in (q, k, v, nc)]
    (want,) = torch.autograd.grad(O.cos_attn_causal(*ref), ref[0], do.double())
    assert _rel(dq.double() * scale, want * scale) <= REL16[torch.bfloat16]


@pytest.mark.parametrize("reverse", [False, True])
@pytest.mark.parametrize("H,N,Dv", [(80, 300, 128), (74, 130, 128), (16, 4200, 128), (4, 4200, 256), (40, 260, 256)])
def test_scan_128_choice_of_width(H, N, Dv, reverse):
    """Either side of the rule for the columns of a CTA: more CTAs than one wave holds, one wave, and segments."""
    from cottention_transformer_b200 import kernel, _lib
    g = torch.Generator().manual_seed(Dv + N)
    q, k = (torch.nn.functional.normalize(torch.randn(1, H, N, 128, generator=g), dim=-1).bfloat16() for _ in range(2))
    v = torch.randn(1, H, N, Dv, generator=g).bfloat16()
    got = kernel.bfloat16(q.cuda(), k.cuda(), v.cuda(), 1, False, reverse)
    _lib.check_device_status()
    few = [0, H - 1]
    assert _rel(got[:, few], O.scan_recurrent(q[:, few].double(), k[:, few].double(), v[:, few].double(), reverse, "f64")) <= REL16[torch.bfloat16]
