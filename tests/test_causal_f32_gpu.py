"""The fused fp32 causal kernels (head dims 32 and 64) against the fp64 math and against the unfused fp32 path."""
import pytest
import torch

from oracle import cott_oracle as O

pytestmark = pytest.mark.gpu

# fp32 sums of up to D + 64 products per step with random signs: a relative error of a few times 2^-24 * sqrt(128) = 7e-7
REL32 = 4e-6


def _inputs(B, H, N, D, masked, seed):
    g = torch.Generator().manual_seed(seed)
    q, k, v, do = (torch.randn(B, H, N, D, generator=g) for _ in range(4))
    nc = 0.5 + 0.2 * torch.randn(1, H, 1, 1, generator=g)
    keep = None
    if masked:
        keep = torch.rand(B, N, generator=g) < 0.7
        keep[0, : N // 3] = False  # positions before the first kept one: n_s = 0
    return q, k, v, do, nc, keep


def _truth(q, k, v, do, nc, keep):
    q, k, v, nc = (t.double().requires_grad_() for t in (q, k, v, nc))
    out = O.cos_attn_causal(q, k, v, nc, keep=keep)
    return out.detach(), *torch.autograd.grad(out, (q, k, v, nc), do.double())


def _rel(a, b):
    return ((a.double().cpu() - b.double().cpu()).norm() / b.double().norm().clamp(min=1e-30)).item()


def _run(fn, q, k, v, do, nc, keep):
    leaf = [t.detach().requires_grad_() for t in (q, k, v, nc)]
    out = fn(*leaf, keep)
    return out.detach(), *torch.autograd.grad(out, leaf, do)


@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("shape", [(1, 1, 1, 64), (2, 3, 63, 32), (1, 2, 64, 64), (2, 2, 65, 64), (1, 3, 129, 32), (2, 4, 1000, 64),
                                   (1, 2, 64 * 9, 32)])  # (nine chunks: one more than the prefix kernel loads at a time)
def test_fused_f32_matches_fp64(shape, masked):
    from cottention_transformer_b200 import cos_attn_causal
    q, k, v, do, nc, keep = _inputs(*shape, masked, seed=sum(shape))
    if masked and not keep.any():
        keep[0, -1] = True
    truth = _truth(q, k, v, do, nc, keep)
    got = _run(cos_attn_causal, *(t.cuda() for t in (q, k, v, do, nc)), None if keep is None else keep.cuda())
    for name, a, b in zip(("out", "dq", "dk", "dv", "dnorm"), got, truth):
        # the gradient of norm_const is a signed sum that may cancel: measured against the size of its terms
        scale = 20 if name == "dnorm" else 1
        if b.norm() == 0:
            assert a.norm() == 0, name
        else:
            assert _rel(a, b) <= scale * REL32, (name, _rel(a, b))


def test_fused_f32_agrees_with_the_unfused_path_over_the_forms_it_accepts():
    """Strided, offset and expanded inputs, zero and tiny rows, infinities in a masked row, and create_graph."""
    from cottention_transformer_b200 import cos_attn_causal
    from cottention_transformer_b200.cos_attention import _exact_causal, f32_supported
    B, H, N, D = 2, 3, 150, 64
    q, k, v, do, nc, keep = (t.cuda() for t in _inputs(B, H, N, D, True, seed=5))
    q[0, 0, 7] = 0          # normalised to zero
    k[1, 2, 9] = 1e-20      # |k| below the epsilon (1e-20^2 underflows to a zero norm)
    flat = torch.empty(B * H * N * D + 1, device="cuda")
    off = flat[1:].view(B, H, N, D)
    off.copy_(k)            # contiguous, 4 bytes off a 16-byte boundary
    strided = q.transpose(1, 2).contiguous().transpose(1, 2)
    wide = do[:, :1].expand(B, H, N, D)
    for args in ((strided, off, v, wide, nc, keep), (q, k, v, do, nc.reshape(H), None)):
        assert f32_supported(*args[:3], args[4], args[5])
        for name, a, b in zip(("out", "dq", "dk", "dv", "dnorm"), _run(cos_attn_causal, *args), _run(_exact_causal, *args)):
            assert a.shape == b.shape and a.isfinite().all()
            assert _rel(a, b) <= 5 * REL32, name
    # a row that is masked by padding may hold anything finite; an infinity reaches the same outputs on both paths
    q[0, 1, N - 1, 3] = float("inf")
    a, b = cos_attn_causal(q, k, v, nc), _exact_causal(q, k, v, nc, None)
    assert torch.equal(a.isnan(), b.isnan())
    # second derivatives keep going through the module math
    leaf = v.detach().requires_grad_()
    (g,) = torch.autograd.grad(cos_attn_causal(k, k, leaf, nc.requires_grad_()).sum(), nc, create_graph=True)
    assert g.requires_grad


def test_f32_forms_that_stay_with_the_unfused_path():
    from cottention_transformer_b200.cos_attention import f32_supported
    q = torch.randn(1, 2, 5, 64, device="cuda")
    nc = torch.zeros(2, device="cuda")
    assert f32_supported(q, q, q, nc)
    assert not f32_supported(q, q, q.double(), nc)
    assert not f32_supported(q, q, q[..., :32], nc)
    assert not f32_supported(q[..., :16], q[..., :16], q[..., :16], nc)
    assert not f32_supported(q, q, q, nc.double())
    assert not f32_supported(q, q, q, nc, torch.ones(1, 5, device="cuda"))
    assert not f32_supported(q[:, :, :0], q[:, :, :0], q[:, :, :0], nc)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        assert not f32_supported(q, q, q, nc)


@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
@pytest.mark.parametrize("N,pos", [(150, 70), (150, 64), (150, 127), (64, 0), (200, 199), (130, 129)])
@pytest.mark.parametrize("D", [32, 64])
def test_non_finite_rows_reach_what_the_sums_contain(D, N, pos, bad):
    """A non-finite value of v or of the incoming gradient enters the sums it is a term of and no other: the causal mask
    leaves a term out, it does not multiply it by zero."""
    from cottention_transformer_b200 import cos_attn_causal
    q, k, v, do, nc, _ = (None if t is None else t.cuda() for t in _inputs(1, 2, N, D, False, seed=N + pos))
    t = torch.arange(N, device="cuda").view(N, 1)
    col = torch.arange(D, device="cuda").view(1, D) == 5
    vb, dob = v.clone(), do.clone()
    vb[0, 1, pos, 5] = bad
    out, dq, dk, dv, dnc = _run(cos_attn_causal, q, k, vb, do, nc, None)
    assert torch.equal(~out[0, 1].isfinite(), (t >= pos) & col)             # out_t = sum_{s <= t} (q^_t . k^_s) v'_s
    assert torch.equal(~dq[0, 1].isfinite(), (t >= pos).expand(N, D))       # dq^_t = sum_{s <= t} (dO_t . v'_s) k^_s
    assert torch.equal(~dk[0, 1].isfinite(), (t == pos).expand(N, D))       # dk^_s = sum_{t >= s} (v'_s . dO_t) q^_t
    assert dv.isfinite().all()                                              # dv'_s = sum_{t >= s} (q^_t . k^_s) dO_t
    assert not dnc[0, 1].isfinite().any()                                   # (also at position 1, whose ln n is zero)
    assert all(x[0, 0].isfinite().all() for x in (out, dq, dk, dv, dnc))
    dob[0, 1, pos, 5] = bad
    out, dq, dk, dv, dnc = _run(cos_attn_causal, q, k, v, dob, nc, None)
    assert out.isfinite().all()
    assert torch.equal(~dq[0, 1].isfinite(), (t == pos).expand(N, D))
    assert torch.equal(~dk[0, 1].isfinite(), (t <= pos).expand(N, D))
    assert torch.equal(~dv[0, 1].isfinite(), (t <= pos) & col)
    assert all(x[0, 0].isfinite().all() for x in (out, dq, dk, dv, dnc))


@pytest.mark.parametrize("compiled", [True, False])
@pytest.mark.parametrize("masked", [False, True])
def test_second_derivatives(masked, compiled, monkeypatch):
    """create_graph: the gradients' gradients with respect to every input against fp64 autograd of the oracle."""
    from cottention_transformer_b200 import _binding, cos_attn_causal
    if not compiled:
        monkeypatch.setattr(_binding, "autograd", lambda: None)
    q, k, v, do, nc, keep = _inputs(2, 2, 70, 32, masked, seed=11)
    if masked:
        keep[:, 0] = True  # (where n_s = 0 the second derivative of n^sigma is a NaN in the module math itself)
    w = [torch.randn(t.shape, generator=torch.Generator().manual_seed(i)) for i, t in enumerate((q, k, v, nc))]

    def second(fn, dtype, dev):
        x = [t.to(dev, dtype).requires_grad_() for t in (q, k, v, nc, do)]
        out = fn(*x[:4], None if keep is None else keep.to(dev))
        first = torch.autograd.grad(out, x[:4], x[4], create_graph=True)
        return torch.autograd.grad(sum((g * u.to(dev, dtype)).sum() for g, u in zip(first, w)), x)

    want = second(lambda q, k, v, n, kp: O.cos_attn_causal(q, k, v, n, keep=kp), torch.float64, "cpu")
    got = second(lambda q, k, v, n, kp: cos_attn_causal(q.transpose(1, 2).contiguous().transpose(1, 2), k, v, n, kp), torch.float32, "cuda")
    for name, a, b in zip(("q", "k", "v", "norm_const", "dout"), got, want):
        # two passes of fp32 sums one after the other, and for norm_const signed sums over the sequence
        assert _rel(a, b) <= (20 if name == "norm_const" else 5) * REL32, (name, _rel(a, b))


@pytest.mark.parametrize("compiled", [True, False])
def test_the_operator_itself_twice(compiled, monkeypatch):
    from cottention_transformer_b200 import CustomAttention, _binding
    if not compiled:
        monkeypatch.setattr(_binding, "autograd", lambda: None)
    g = torch.Generator().manual_seed(1)
    q, k, v = (torch.randn(1, 2, 5, 32, generator=g, dtype=torch.float64).cuda().requires_grad_() for _ in range(3))
    assert torch.autograd.gradcheck(CustomAttention.apply, (q, k, v), fast_mode=True)
    assert torch.autograd.gradgradcheck(CustomAttention.apply, (q, k.transpose(1, 2).contiguous().transpose(1, 2), v), fast_mode=True)


@pytest.mark.parametrize("D", [32, 64])
@pytest.mark.parametrize("N", [65, 100, 150])
def test_sums_begin_with_a_whole_chunk_in_their_own_direction(N, D):
    """Forward sums are cut from the first position, reversed ones from the last: the 64 rows where either begins are those
    of the 64 positions by themselves, bit for bit.  (With a norm_const of -200 the length factor is 1 everywhere.)"""
    from cottention_transformer_b200 import cos_attn_causal
    q, k, v, do, nc, _ = (None if t is None else t.cuda() for t in _inputs(2, 2, N, D, False, seed=N))
    nc = torch.full_like(nc, -200.0)
    whole = _run(cos_attn_causal, q, k, v, do, nc, None)
    first = _run(cos_attn_causal, *(t[:, :, :64].contiguous() for t in (q, k, v, do)), nc, None)
    last = _run(cos_attn_causal, *(t[:, :, -64:].contiguous() for t in (q, k, v, do)), nc, None)
    for i in (0, 1):
        assert torch.equal(whole[i][:, :, :64], first[i])
    for i in (2, 3):
        assert torch.equal(whole[i][:, :, -64:], last[i])
