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
