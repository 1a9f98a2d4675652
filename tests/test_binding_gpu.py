"""The compiled autograd functions against the Python ones they stand in for: same results bit for bit, and the same
behaviour where a caller does something between the forward and the backward, or transforms the call."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _args(name, dt, seed=3, B=2, H=3, N=150):
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g).to(dt)  # noqa: E731
    nc = 0.5 + 0.2 * torch.randn(1, H, 1, 1, device="cuda", generator=g)
    keep = torch.rand(B, N, device="cuda", generator=g) < 0.7
    keep[:, 0] = True
    D = {"wide": 128, "f32": 32}.get(name, 64)
    if name in ("packed", "rotary", "bidir"):
        x = (r(B, N, 3, H, D),)
        do = r(B, N, H, D)
    else:
        x = tuple(r(B, H, N, D) for _ in range(3))
        do = r(B, H, N, D)
    ang = torch.rand(N, 16, device="cuda", generator=g)
    return x, nc, keep, do, (torch.sin(ang), torch.cos(ang))


def _call(name, x, nc, keep, rot):
    import cottention_transformer_b200 as C
    if name == "dropin":
        return C.CustomAttention.apply(*x)
    if name == "bidir":
        return C.cos_attn_bidirectional_packed(x[0], nc, keep)
    if name in ("packed", "rotary"):
        return C.cos_attn_causal_packed(x[0], nc, keep, rot if name == "rotary" else None)
    return C.cos_attn_causal(*x, nc, keep, one_pass_backward=name == "one_pass")


PATHS = [("causal", torch.bfloat16), ("one_pass", torch.float16), ("packed", torch.bfloat16), ("rotary", torch.float16),
         ("bidir", torch.bfloat16), ("wide", torch.float16), ("f32", torch.float32), ("dropin", torch.bfloat16), ("dropin", torch.float64)]


@pytest.mark.parametrize("name,dt", PATHS)
@pytest.mark.parametrize("masked", [False, True])
def test_same_bits_as_the_python_functions(name, dt, masked, monkeypatch):
    from cottention_transformer_b200 import _binding
    if _binding.module() is None:
        pytest.skip("binding not built")
    x, nc, keep, do, rot = _args(name, dt)
    rot_args = rot
    res = []
    for compiled in (True, False):
        if not compiled:
            monkeypatch.setattr(_binding, "autograd", lambda: None)
        leaf = [t.clone().requires_grad_() for t in x]
        ncl = nc.clone().requires_grad_()
        k = keep.clone() if masked else None
        out = _call(name, leaf, ncl, k, rot_args)
        if masked:
            k.fill_(True)  # what the caller does to its mask afterwards is not the backward's business
        wrt = leaf if name == "dropin" else [*leaf, ncl]
        res.append((out.detach(), *torch.autograd.grad(out, wrt, do)))
    names = ["out", *("dx%d" % i for i in range(len(x))), "dnorm"]
    for n, a, b in zip(names, *res):
        assert a.dtype == b.dtype and a.shape == b.shape
        if n == "dnorm" and dt != torch.float32:  # sums by atomics: the order of the additions is not fixed
            assert torch.allclose(a, b, rtol=1e-3, atol=1e-4)
        else:
            assert torch.equal(a, b), n


def test_saved_tensor_hooks_and_modified_inputs():
    from cottention_transformer_b200 import cos_attn_causal
    x, nc, _, do, _ = _args("causal", torch.bfloat16)
    packed = []
    leaf = [t.clone().requires_grad_() for t in x]
    with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(t.shape) or t.clone(), lambda t: t):
        out = cos_attn_causal(*leaf, nc.requires_grad_())
    assert len(packed) == 4  # q, k, v and norm_const pass through the hooks
    a = torch.autograd.grad(out, leaf, do)
    b = torch.autograd.grad(cos_attn_causal(*leaf, nc), leaf, do)
    assert all(torch.equal(s, t) for s, t in zip(a, b))
    q = x[0].clone().requires_grad_() * 1
    out = cos_attn_causal(q, x[1], x[2], nc)
    q.mul_(2)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        out.backward(do)


def test_transforms_are_refused_as_before():
    from cottention_transformer_b200 import cos_attn_causal
    x, nc, _, _, _ = _args("causal", torch.bfloat16)
    with pytest.raises(RuntimeError):
        torch.func.grad(lambda q: cos_attn_causal(q, x[1], x[2], nc).float().sum())(x[0])
    with pytest.raises(RuntimeError):
        torch.func.vmap(lambda q: cos_attn_causal(q, x[1], x[2], nc))(x[0][None])
    with pytest.raises((RuntimeError, NotImplementedError)):
        torch.func.jvp(lambda q: cos_attn_causal(q, x[1], x[2], nc), (x[0],), (x[0],))


def test_dispatch_modes_see_the_operators():
    from torch.utils._python_dispatch import TorchDispatchMode

    from cottention_transformer_b200 import cos_attn_causal

    class Seen(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            names.append(str(func))
            return func(*args, **(kwargs or {}))

    x, nc, _, do, _ = _args("causal", torch.bfloat16)
    names = []
    leaf = [t.clone().requires_grad_() for t in x]
    with Seen():
        out = cos_attn_causal(*leaf, nc)
    assert any("causal_fwd" in n for n in names)
    assert torch.equal(out, cos_attn_causal(*leaf, nc))
    assert all(torch.equal(a, b) for a, b in zip(torch.autograd.grad(out, leaf, do), torch.autograd.grad(cos_attn_causal(*leaf, nc), leaf, do)))


@pytest.mark.parametrize("D", [64, 128])
def test_transformed_prefill(D):
    """Forward-mode differentiation is refused, not dropped; a trace runs the operator and does not return an empty buffer."""
    import torch.autograd.forward_ad as fw

    from cottention_transformer_b200 import CosAttnDecodeState
    g = torch.Generator(device="cuda").manual_seed(D)
    q, k, v, q2 = (torch.randn(1, 2, 200, D, device="cuda", generator=g).bfloat16() for _ in range(4))
    nc = torch.full((2,), 0.5, device="cuda")
    with fw.dual_level(), pytest.raises((RuntimeError, NotImplementedError)):
        CosAttnDecodeState(1, 2, D).prefill(fw.make_dual(q, q), k, v, nc)
    with fw.dual_level():
        st = CosAttnDecodeState(1, 2, D)
        out = st.prefill(q, k, v, nc)
    ref = CosAttnDecodeState(1, 2, D)
    assert torch.equal(out, ref.prefill(q, k, v, nc))
    # the state: another kernel, the same sums of 16-bit products in fp32
    assert (st.state - ref.state).norm() <= 1e-3 * ref.state.norm() and st.cur_s == ref.cur_s
    traced = torch.jit.trace(lambda a: CosAttnDecodeState(1, 2, D).prefill(a, k, v, nc), (q,), check_trace=False)
    assert torch.equal(traced(q2), CosAttnDecodeState(1, 2, D).prefill(q2, k, v, nc))


def test_other_python_threads_run_while_a_launch_waits():
    """A call that waits for room in the launch queue (behind a kernel of about half a second) does not hold the
    interpreter lock meanwhile."""
    import threading
    import time

    from cottention_transformer_b200 import CosAttnDecodeState
    tok = torch.randn(1, 1, 1, 64, device="cuda").bfloat16()
    nc, st = torch.zeros(1, device="cuda"), CosAttnDecodeState(1, 1, 64)
    st.step(tok, tok, tok, nc)
    torch.cuda.synchronize()
    gaps, stop = [], threading.Event()

    def tick():
        last = time.perf_counter()
        while not stop.is_set():
            time.sleep(0.001)
            now = time.perf_counter()
            gaps.append(now - last)
            last = now

    other = threading.Thread(target=tick)
    other.start()
    t0 = time.perf_counter()
    torch.cuda._sleep(1_000_000_000)
    for _ in range(3000):
        st.step(tok, tok, tok, nc)
    waited = time.perf_counter() - t0
    stop.set()
    other.join()
    torch.cuda.synchronize()
    assert waited > 0.2, "the queue took all launches: nothing was tested"
    assert max(gaps) < 0.5 * waited


def test_short_norm_const_is_refused():
    from cottention_transformer_b200 import CosAttnDecodeState, cos_attn_bidirectional_packed, cos_attn_causal_packed
    x, nc, _, _, _ = _args("packed", torch.bfloat16)
    for fn in (cos_attn_causal_packed, cos_attn_bidirectional_packed):
        with pytest.raises(RuntimeError, match="one entry per head"):
            fn(x[0], nc[:, :2])
    tok = torch.randn(1, 3, 1, 64, device="cuda").bfloat16()
    with pytest.raises(RuntimeError, match="one entry per head"):
        CosAttnDecodeState(1, 3, 64).step(tok, tok, tok, nc[:, :2])


@pytest.mark.parametrize("compiled", [True, False])
@pytest.mark.parametrize("keep_rotated", [True, False])
@pytest.mark.parametrize("B,H,N,rot,segments", [(2, 3, 150, 32, 1), (1, 2, 4100, 64, 2), (1, 3, 5000, 24, 2), (1, 8, 300, 8, 1)])
def test_rotary_leaves_the_projection_alone(B, H, N, rot, segments, keep_rotated, compiled, monkeypatch):
    """Whatever the sizes: cut into segments or not, rotary dims that are no multiple of 16 included."""
    from cottention_transformer_b200 import _binding, _lib, cos_attn_causal_packed, rotary_packed_
    if not compiled:
        monkeypatch.setattr(_binding, "autograd", lambda: None)
    assert (_lib.lib().cott_cos_attn_seg_choice(B, H, N) > 1) == (segments > 1)
    g = torch.Generator(device="cuda").manual_seed(N + rot)
    qkv = torch.randn(B, N, 3, H, 64, device="cuda", generator=g).bfloat16()
    do = torch.randn(B, N, H, 64, device="cuda", generator=g).bfloat16()
    nc = torch.full((H,), 0.5, device="cuda")
    ang = torch.rand(N, rot // 2, device="cuda", generator=g) * 6
    sc = (torch.sin(ang), torch.cos(ang))
    leaf = qkv.clone().requires_grad_()
    out = cos_attn_causal_packed(leaf, nc, rotary=sc, keep_rotated=keep_rotated)
    (dx,) = torch.autograd.grad(out, leaf, do)
    assert torch.equal(leaf, qkv)
    other = qkv.clone().requires_grad_()
    want = cos_attn_causal_packed(rotary_packed_(other * 1, *sc), nc)
    (dw,) = torch.autograd.grad(want, other, do)
    assert torch.equal(out, want) and torch.equal(dx, dw)


@pytest.mark.parametrize("compiled", [True, False])
@pytest.mark.parametrize("D", [64, 128])
def test_shapes_that_do_not_fit_are_refused(D, compiled, monkeypatch):
    """Five dimensions (whose fourth happens to be a head dim), and k, v or a state that would be read past their end."""
    from cottention_transformer_b200 import CosAttnDecodeState, _binding, cos_attn_causal
    if not compiled:
        monkeypatch.setattr(_binding, "autograd", lambda: None)
    nc = torch.zeros(2, device="cuda")
    x = torch.randn(1, 2, 3, D, D, device="cuda").bfloat16()
    with pytest.raises(ValueError):
        cos_attn_causal(x, x, x, nc)
    with pytest.raises(ValueError):
        CosAttnDecodeState(1, 2, D).prefill(x, x, x, nc)
    q = torch.randn(2, 2, 5, D, device="cuda").bfloat16()
    for k, v in ((q[:1], q), (q, q[:, :1]), (q, q[:, :, :3])):
        with pytest.raises(RuntimeError, match="same shape"):
            cos_attn_causal(q, k, v, nc)
        with pytest.raises(RuntimeError, match="same shape"):
            CosAttnDecodeState(2, 2, D).prefill(q, k, v, nc)
        with pytest.raises(RuntimeError, match="do not fit"):
            CosAttnDecodeState(2, 2, D).step(q, k, v, nc)
    with pytest.raises(RuntimeError, match="the state"):
        CosAttnDecodeState(1, 2, D).prefill(q, q, q, nc)
    with pytest.raises(RuntimeError, match="the state"):
        CosAttnDecodeState(1, 2, D).step(q, q, q, nc)


@pytest.mark.parametrize("N,rot", [(1, 64), (130, 16), (300, 48)])
@pytest.mark.parametrize("per_batch", [False, True])
def test_rotation_inside_the_kernels_gives_the_bits_of_the_copying_pass(N, rot, per_batch):
    """``cott_cos_attn_fwd_rotary`` / ``_bwd_rotary`` (C callers without room for the rotated copies) against the op."""
    import ctypes

    from cottention_transformer_b200 import _lib, cos_attn_causal_packed
    B, H, D = 3, 30, 64  # (90 sequences: one segment each)
    g = torch.Generator(device="cuda").manual_seed(N + rot)
    qkv = torch.randn(B, N, 3, H, D, device="cuda", generator=g).bfloat16()
    do = torch.randn(B, N, H, D, device="cuda", generator=g).bfloat16()
    nc = 0.5 + 0.2 * torch.randn(H, device="cuda", generator=g)
    ang = torch.rand(*((B, N, rot // 2) if per_batch else (N, rot // 2)), device="cuda", generator=g) * 6
    sin, cos = torch.sin(ang), torch.cos(ang)
    leaf = qkv.clone().requires_grad_()
    out = cos_attn_causal_packed(leaf, nc, None, (sin, cos))
    (dx,) = torch.autograd.grad(out, leaf, do)
    assert torch.equal(leaf, qkv)
    L, P = _lib.lib(), (lambda t: t.data_ptr())
    o, d, dnc = torch.empty_like(out), torch.empty_like(qkv), torch.empty(H, device="cuda")
    ws = torch.empty(L.cott_cos_attn_seg_workspace_bytes(B, H, N, 1), dtype=torch.uint8, device="cuda")
    lay = _lib.CottLayout(N * 3 * H * D, D, 3 * H * D, N * H * D, D, H * D)
    tab = _lib.CottRotaryTables(P(sin), P(cos), rot, N * rot // 2 if per_batch else 0)
    st = _lib.stream_ptr(qkv.device)
    q, k, v = (P(qkv[:, :, i]) for i in range(3))
    _lib.check(L.cott_cos_attn_fwd_rotary(q, k, v, None, P(nc), P(o), P(ws), ctypes.byref(lay), ctypes.byref(tab), B, H, N, D, D, 3, st), "fwd")
    _lib.check(L.cott_cos_attn_bwd_rotary(q, k, v, None, P(nc), P(do), P(ws), ctypes.byref(lay), ctypes.byref(tab), P(d[:, :, 0]), P(d[:, :, 1]),
                                          P(d[:, :, 2]), P(dnc), B, H, N, D, D, 3, st), "bwd")
    _lib.check_device_status()
    assert torch.equal(o, out) and torch.equal(d, dx)
