"""Prefill: outputs and decode state in one call, at the edges of chunks and segments."""
import pytest
import torch

from oracle import cott_oracle as O

pytestmark = pytest.mark.gpu

REL16 = 2e-2  # 16-bit products, as for the causal operators


def _rel(a, b):
    return ((a.double().cpu() - b).norm() / b.norm()).item()


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,H,N", [(2, 3, 1), (1, 2, 128), (4, 16, 129), (4, 16, 777), (1, 2, 2000), (1, 5, 5000)])
def test_prefill_outputs_and_state(B, H, N, D):
    from cottention_transformer_b200 import CosAttnDecodeState, _lib
    g = torch.Generator().manual_seed(N + D)
    q, k, v = (torch.randn(B, H, N, D, generator=g).bfloat16() for _ in range(3))
    nc = 0.5 + 0.2 * torch.randn(1, H, 1, 1, generator=g)
    st = CosAttnDecodeState(B, H, D)
    st.state.fill_(7.0)  # (a fresh state is at position 1 whatever its buffer holds: the call overwrites it)
    out = st.prefill(q.cuda(), k.cuda(), v.cuda(), nc.cuda())
    _lib.check_device_status()
    kh = torch.nn.functional.normalize(k.double(), dim=-1)
    qh = torch.nn.functional.normalize(q.double(), dim=-1)
    vp = v.double() / torch.arange(1, N + 1).double().view(1, 1, N, 1) ** torch.sigmoid(nc.double())
    assert st.cur_s == N + 1
    assert _rel(st.state, torch.einsum("bhnj,bhni->bhji", vp, kh)) <= REL16
    assert _rel(out, O.scan_recurrent(qh, kh, vp, False, "f64")) <= REL16
    # the state the next token sees
    qn, kn, vn = (torch.randn(B, H, 1, D, generator=g).bfloat16() for _ in range(3))
    nxt = st.step(qn.cuda(), kn.cuda(), vn.cuda(), nc.cuda())
    S = torch.einsum("bhnj,bhni->bhji", vp, kh) + torch.einsum("bhj,bhi->bhji", vn[:, :, 0].double() / (N + 1.0) ** torch.sigmoid(nc.double())[..., 0],
                                                               torch.nn.functional.normalize(kn[:, :, 0].double(), dim=-1))
    want = torch.einsum("bhji,bhi->bhj", S, torch.nn.functional.normalize(qn[:, :, 0].double(), dim=-1))
    assert _rel(nxt[:, :, 0], want) <= REL16


@pytest.mark.parametrize("accumulate", [0, 1])
@pytest.mark.parametrize("D,B,H,N,nseg", [(64, 2, 3, 1, 1), (64, 1, 2, 777, 1), (64, 2, 2, 1300, 3), (64, 1, 3, 5000, 20), (128, 2, 3, 130, 1),
                                          (128, 1, 2, 1, 1), (128, 1, 1, 1001, 0), (128, 1, 3, 5000, 0)])
def test_state_of_a_prompt_by_itself(D, B, H, N, nseg, accumulate):
    """``cott_cos_attn_prefill_state``: one and several segments, the last one ragged, over a state and added to it.  (Head
    dim 128 chooses its segments itself.)"""
    from cottention_transformer_b200 import _lib
    L, P = _lib.lib(), _lib.ptr
    g = torch.Generator().manual_seed(N + D)
    k, v = (torch.randn(B, H, N, D, generator=g).bfloat16() for _ in range(2))
    nc = 0.5 + 0.2 * torch.randn(H, generator=g)
    before = torch.randn(B, H, D, D, generator=g)
    state, kd, vd, ncd = before.cuda(), k.cuda(), v.cuda(), nc.cuda()
    nbytes = L.cott_cos_attn_wide_workspace_bytes(B, H, N) if D == 128 else L.cott_cos_attn_seg_workspace_bytes(B, H, N, nseg)
    ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    _lib.check(L.cott_cos_attn_prefill_state(P(kd), P(vd), P(ncd), P(state), P(ws), nseg, accumulate, B, H, N, D, D, 3,
                                             _lib.stream_ptr(state.device)), "prefill_state")
    _lib.check_device_status()
    n = torch.arange(1, N + 1).double().view(1, 1, N, 1)
    vp = v.double() / n ** torch.sigmoid(nc.double()).view(1, H, 1, 1)
    want = torch.einsum("bhnj,bhni->bhji", vp, torch.nn.functional.normalize(k.double(), dim=-1))
    # (what was there before enters with 1, exactly: the tolerance is that of the products)
    got = state.double().cpu() - (before.double() if accumulate else 0)
    assert ((got - want).norm() / want.norm()).item() <= REL16
