"""The short convolution with channels that go one or two a thread, segments of a few rows and of many, and several activations."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("C, c0, taps", [(257, 0, 4), (256, 3, 2), (300, 8, 8), (2, 2, 1), (510, 4, 7)])
@pytest.mark.parametrize("n", [1, 2, 9, 32, 41, 2400, 9473])
def test_convolution_of_one_segment(dtype, C, c0, taps, n):
    from cbis_b200.kernels import ops
    g = torch.Generator().manual_seed(C + taps + n)
    x = torch.randn(n, c0 + C + 2, generator=g).to(dtype)
    w, b = torch.randn(C, taps, generator=g), torch.randn(C, generator=g)
    before = torch.randn(taps - 1, C, generator=g).to(dtype).float()
    rows = torch.cat([before.double(), x[:, c0:c0 + C].double()])
    sums = sum(rows[j:j + n] * w[:, j].double() for j in range(taps)) + b.double()
    slot, cu = torch.tensor([1], dtype=torch.int32, device="cuda"), torch.tensor([0, n], dtype=torch.int32, device="cuda")
    for act, f in (("silu", torch.nn.functional.silu), (None, lambda v: v), ("sigmoid", torch.sigmoid)):
        state = torch.zeros(2, max(1, (taps - 1) * C), device="cuda")
        if taps > 1:
            state[1] = before.reshape(-1).cuda()
        out = torch.empty(n, C, dtype=dtype, device="cuda")
        ops.causal_conv_act(x.cuda(), c0, C, w.cuda(), b.cuda(), state, slot, cu, 1, n, act, out, update_state=n <= 32 and taps > 1)
        ref = f(sums)
        tol = 1e-5 if dtype == torch.float32 else 1e-2      # eight 32-bit products; one rounding to bfloat16 (2^-9)
        assert (out.double().cpu() - ref).abs().max() < tol * max(1.0, ref.abs().max().item())
        if taps > 1 and n <= 32:
            assert torch.equal(state[1].double().cpu(), rows[n:].reshape(-1))
