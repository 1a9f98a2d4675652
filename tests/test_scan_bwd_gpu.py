"""cott_scan_bwd: the three scans in one launch against the three calls it stands for."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,H,N", [(1, 1, 1), (2, 3, 127), (1, 2, 128), (2, 2, 129), (3, 50, 700), (1, 2, 6000)])  # (the last one is cut into segments)
def test_one_launch_gives_the_bits_of_three(B, H, N, dt):
    from cottention_transformer_b200 import _lib, kernel
    g = torch.Generator(device="cuda").manual_seed(N)
    q, k, v, do = (torch.nn.functional.normalize(torch.randn(B, H, N, 64, device="cuda", generator=g), dim=-1).to(dt) for _ in range(4))
    want = (kernel.scan(do, v, k, False), kernel.scan(v, do, q, True), kernel.scan(k, q, do, True))
    L, P = _lib.lib(), (lambda t: t.data_ptr())
    got = [torch.full_like(q, float("nan")) for _ in range(3)]
    code, st = _lib.DTYPE_CODE[dt], _lib.stream_ptr(q.device)
    _lib.check(L.cott_scan_bwd(P(q), P(k), P(v), P(do), *(P(t) for t in got), B, H, N, 64, 64, code, st), "cott_scan_bwd")
    _lib.check_device_status()
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    # an output over an input: one scan after the other, as ever (dv may replace v: the last scan does not read it)
    last = v.clone()
    _lib.check(L.cott_scan_bwd(P(q), P(k), P(last), P(do), P(got[0]), P(got[1]), P(last), B, H, N, 64, 64, code, st), "cott_scan_bwd")
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1]) and torch.equal(last, want[2])
