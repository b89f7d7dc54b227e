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


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("C, taps", [(300, 8), (255, 1), (6144, 4)])
@pytest.mark.parametrize("segs", [[1, 2, 3, 4, 5, 32, 1], [1, 33, 2, 0, 100, 7], [1] * 20 + [480], [2, 1, 1, 2]])
def test_convolution_of_unlike_segments(dtype, C, taps, segs):
    """Segments of one and two rows, of up to a block's rows and of more side by side (rows one by one, four and eight at a time),
    with 6,144 channels also two channels a thread: every segment from its own state, and its own state afterwards."""
    from cbis_b200.kernels import ops
    g = torch.Generator().manual_seed(C + len(segs))
    T, S = sum(segs), len(segs)
    x = torch.randn(T, C, generator=g).to(dtype)
    w, b = torch.randn(C, taps, generator=g), torch.randn(C, generator=g)
    before = torch.randn(S, taps - 1, C, generator=g).to(dtype).float()
    slot = torch.randperm(S, generator=g).int()
    cu = torch.tensor([0] + segs).cumsum(0).int()
    state = torch.zeros(S, max(1, (taps - 1) * C))
    if taps > 1:
        state[slot.long()] = before.reshape(S, -1)
    state, out = state.cuda(), torch.empty(T, C, dtype=dtype, device="cuda")
    update = max(segs) <= 32 and taps > 1
    ops.causal_conv_act(x.cuda(), 0, C, w.cuda(), b.cuda(), state, slot.cuda(), cu.cuda(), S, max(segs), "silu", out, update_state=update)
    tol = 1e-5 if dtype == torch.float32 else 1e-2      # as above
    for i, n in enumerate(segs):
        rows = torch.cat([before[i].double(), x[cu[i]:cu[i + 1]].double()])
        if n:
            ref = torch.nn.functional.silu(sum(rows[j:j + n] * w[:, j].double() for j in range(taps)) + b.double())
            assert (out[cu[i]:cu[i + 1]].double().cpu() - ref).abs().max() < tol * max(1.0, ref.abs().max().item()), (i, n)
        if taps > 1:
            assert torch.equal(state[slot[i].item()].double().cpu(), (rows[n:] if update else rows[:taps - 1]).reshape(-1))
