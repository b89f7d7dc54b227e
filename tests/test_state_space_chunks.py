"""The state-space recurrence 64 rows at a time, against the walk row by row in 64 bits."""
import pytest
import torch

import plain_vekedra as pv

pytestmark = pytest.mark.gpu


def walk(xbc, raw, a_log, dt_bias, d_skip, H, P, N, G, S=None):
    inner = H * P
    x, B, C = xbc[:, :inner].view(-1, H, P), xbc[:, inner:inner + G * N].view(-1, G, N), xbc[:, inner + G * N:].view(-1, G, N)
    B, C = (t.repeat_interleave(H // G, 1) for t in (B, C))
    dt = pv.softplus(raw + dt_bias)
    S = torch.zeros(H, P, N, dtype=torch.float64) if S is None else S
    out = []
    for t in range(x.shape[0]):
        S = torch.exp(-torch.exp(a_log) * dt[t])[:, None, None] * S + dt[t][:, None, None] * x[t][:, :, None] * B[t][:, None, :]
        out.append((S * C[t][:, None, :]).sum(-1) + d_skip[:, None] * x[t])
    return torch.stack(out).view(-1, inner), S


@pytest.mark.parametrize("H,P,N,G", [(2, 64, 128, 1), (4, 32, 64, 2), (3, 96, 64, 3)])
def test_rows_in_chunks(H, P, N, G):
    """Segments around a chunk's edges (33 rows and more go by chunks, fewer row by row, in one step), continued from their
    states over several steps; one head that hardly decays, one whose decays underflow.  Each result is a sum of up to 700
    32-bit terms around 1: bounded by 2e-6 of the largest, and no further off than the row-by-row kernel's."""
    from cbis_b200.kernels import ops
    g = torch.Generator().manual_seed(H * P)
    inner = H * P
    a_log, dt_bias, d_skip = torch.randn(H, generator=g), torch.randn(H, generator=g) - 1.0, torch.randn(H, generator=g)
    a_log[0], dt_bias[0] = -5.0, -1.0
    a_log[1] = 4.0
    steps = [[64, 33, 1], [63, 200, 32], [129, 65, 700], [2, 34, 128]]
    errs = {}
    data = [[(torch.randn(n, inner + 2 * G * N, generator=g).bfloat16(), torch.randn(n, 3 + H, generator=g).bfloat16())
             for n in s] for s in steps]
    for how in (None, 0):      # by chunks; row by row
        state = torch.zeros(4, inner * N + 5, dtype=torch.float32, device="cuda")
        ref_S, worst = [None] * 3, 0.0
        for sizes, seqs in zip(steps, data):
            xs, ps = (torch.cat([s[i] for s in seqs]).cuda() for i in (0, 1))
            cu = torch.tensor([0] + sizes, dtype=torch.int32).cumsum(0).int().cuda()
            y = torch.full((sum(sizes), inner + 2), float("nan"), device="cuda")
            ops.ssm_scan(xs, ps, 3, dt_bias.cuda(), a_log.cuda(), d_skip.cuda(), state, torch.tensor([2, 0, 1], dtype=torch.int32, device="cuda"),
                         cu, 3, H, P, N, G, y[:, :inner], max_seg_rows=max(sizes), piece_rows=how)
            assert torch.isnan(y[:, inner:]).all()
            at = 0
            for i, n in enumerate(sizes):
                ref, ref_S[i] = walk(seqs[i][0].double(), seqs[i][1][:, 3:].double(), a_log.double(), dt_bias.double(), d_skip.double(), H, P, N, G, ref_S[i])
                worst = max(worst, ((y[at:at + n, :inner].double().cpu() - ref).abs().max() / ref.abs().max()).item())
                at += n
        for slot, i in ((2, 0), (0, 1), (1, 2)):
            got = state[slot, :inner * N].view(H, P, N).double().cpu()
            worst = max(worst, ((got - ref_S[i]).abs().max() / ref_S[i].abs().max()).item())
        assert (state[3] == 0).all() and (state[:, inner * N:] == 0).all()
        errs[how] = worst
    print("largest relative error: chunks %.2e, row by row %.2e" % (errs[None], errs[0]))
    assert errs[None] < 2e-6 and errs[None] <= errs[0], errs


@pytest.mark.parametrize("value", [float("inf"), float("nan"), -float("inf")])
@pytest.mark.parametrize("at", [0, 37, 47, 70])
def test_an_infinite_x_reaches_its_own_column_from_its_own_row_on(value, at):
    """One x that is no finite number, at a tile's edge or inside it: the rows before it and all other columns, of y and of the
    state, are what they are with a 0 in its place (the bound of the test above), its column is not finite from there on."""
    from cbis_b200.kernels import ops
    H, P, N, rows, col = 2, 64, 128, 100, 21
    g = torch.Generator().manual_seed(at)
    xbc, raw = torch.randn(rows, H * P + 2 * N, generator=g).bfloat16(), torch.randn(rows, H, generator=g).bfloat16()
    a_log, dt_bias, d_skip = torch.randn(H, generator=g).cuda(), torch.randn(H, generator=g).cuda(), torch.randn(H, generator=g).cuda()
    out = []
    for v in (0.0, value):
        xbc[at, col] = v
        state, y = torch.zeros(1, H * P * N, device="cuda"), torch.empty(rows, H * P, device="cuda")
        ops.ssm_scan(xbc.cuda(), raw.cuda(), 0, dt_bias, a_log, d_skip, state, torch.zeros(1, dtype=torch.int32, device="cuda"),
                     torch.tensor([0, rows], dtype=torch.int32, device="cuda"), 1, H, P, N, 1, y, max_seg_rows=rows)
        out.append((y.cpu(), state.view(H * P, N).cpu()))
    (y0, s0), (y1, s1) = out
    assert not torch.isfinite(y1[at:, col]).any() and not torch.isfinite(s1[col]).any()
    y1[at:, col], s1[col] = y0[at:, col], s0[col]
    assert (y1 - y0).abs().max() <= 2e-6 * y0.abs().max() and (s1 - s0).abs().max() <= 2e-6 * s0.abs().max()


@pytest.mark.parametrize("H,P,N,rows,launches", [(2, 64, 64, 1100, 3), (2, 64, 64, 640, 1), (4, 32, 128, 1000, 3), (8, 64, 64, 1500, 1)])
def test_long_segments_of_few_states_go_in_pieces(H, P, N, rows, launches):
    """8,192 and 16,384 state elements from some 700 and 960 rows on: three launches side by side; fewer rows or more states: one
    kernel, chunk after chunk.  Sums of up to 1,100 32-bit terms around 1, twice over: 4e-6 of the largest."""
    from cbis_b200.kernels import ops
    g = torch.Generator().manual_seed(rows)
    xbc, raw = torch.randn(rows, H * P + 2 * N, generator=g).bfloat16(), torch.randn(rows, H, generator=g).bfloat16()
    a_log, dt_bias, d_skip = torch.randn(H, generator=g), torch.randn(H, generator=g) - 1.0, torch.randn(H, generator=g)
    state, y = torch.zeros(1, H * P * N, device="cuda"), torch.empty(rows, H * P, device="cuda")
    before = ops.launch_count()
    ops.ssm_scan(xbc.cuda(), raw.cuda(), 0, dt_bias.cuda(), a_log.cuda(), d_skip.cuda(), state, torch.zeros(1, dtype=torch.int32, device="cuda"),
                 torch.tensor([0, rows], dtype=torch.int32, device="cuda"), 1, H, P, N, 1, y, max_seg_rows=rows)
    assert ops.launch_count() - before == launches
    ref, S = walk(xbc.double(), raw.double(), a_log.double(), dt_bias.double(), d_skip.double(), H, P, N, 1)
    assert (y.double().cpu() - ref).abs().max() < 4e-6 * ref.abs().max()
    assert (state.view(H, P, N).double().cpu() - S).abs().max() < 4e-6 * S.abs().max()
