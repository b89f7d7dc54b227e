"""Decode attention whose keys are cut by the rows' own lengths: the plan, and the results against the even cut."""
import pytest
import torch

from test_kernels import dev, ops, paged_case      # noqa: F401  (a fixture)

pytestmark = pytest.mark.gpu


def pieces_of(plan, rows):
    """Per row its (piece, pieces, place of the first); and all entries as (row, piece, pieces, place, request, position)."""
    p = [(w & 4095, (w >> 12) & 31, (w >> 17) + 1, b, s, q) if w >= 0 else (-1, 0, 1, b, s, q) for w, b, s, q in plan.cpu().tolist()]
    return {r: [(e[1], e[2], e[3]) for e in p if e[0] == r] for r in range(rows)}, p


@pytest.mark.parametrize("rows,n_head,hd,longest", [(1, 16, 128, 2048), (8, 16, 128, 2000), (37, 25, 64, 1000), (64, 16, 128, 1400),
                                                    (3, 700, 64, 300), (300, 4, 128, 97), (5, 1, 64, 32768),
                                                    (36, 16, 128, 30000), (2, 16, 128, 200), (24, 25, 64, 300)])
def test_the_plan_covers_every_key_once(ops, rows, n_head, hd, longest):
    g = torch.Generator().manual_seed(rows)
    pos = torch.randint(0, longest, (rows,), generator=g).int()
    pos[0] = longest - 1
    seq = torch.arange(rows, dtype=torch.int32)
    if rows > 2:
        seq[2] = -1
    if rows == 24:                                                        # an even share is one round of keys, the longest row three
        pos[1:] //= 2
    if longest == 30000:                                                  # one place more than rows, and rows of more than half the
        pos[1:] = longest // 2 + 1                                        # longest: hardly any cut is few enough
    plan = ops.decode_plan(dev(seq), dev(pos), rows, n_head, longest, hd)
    by_row, entries = pieces_of(plan, rows)
    used = sum(len(v) for v in by_row.values())
    assert all(e[0] == -1 for e in entries[used:]) and all(e[0] >= 0 for e in entries[:used])
    fit = max(1, 592 // n_head)
    assert used <= (fit if rows <= fit else rows + fit)                  # as many rows as blocks fit side by side: one round of blocks
    if longest <= 200 and rows == 2:
        assert used > rows                                                # ... in several pieces where that saves more than a merge
    if longest == 300 and rows == 24:
        assert used == rows                                               # ... and whole where it does not
    taken = set()
    for r, v in by_row.items():
        n = len(v)
        assert 1 <= n <= 32 and sorted(s for s, _, _ in v) == list(range(n)) and all(of == n and b == v[0][2] for _, of, b in v)
        taken |= set(range(v[0][2], v[0][2] + n))
        assert seq[r] >= 0 or n == 1
    assert taken == set(range(used))                                    # every piece has a place of its own for its result
    assert all(e[4] == int(seq[e[0]]) and e[5] == int(pos[e[0]]) for e in entries[:used])
    keys = [-(-(int(pos[e[0]]) + 1) // e[2]) if e[4] >= 0 else 0 for e in entries[:used]]
    assert keys == sorted(keys, reverse=True)                            # the longest pieces first


@pytest.mark.parametrize("n_head,n_kv_head,hd,window", [(4, 4, 64, 0), (4, 2, 128, 0), (16, 4, 128, 130), (25, 25, 64, -48), (3, 1, 64, 1)])
def test_rows_of_unlike_length_in_pieces(ops, n_head, n_kv_head, hd, window):
    """Contexts around the edges of tiles, rounds and pieces, a padding row, sinks, first keys that stay visible: against the
    plain result, and against the even cut within a rounding of bfloat16 (the same sums in other groups)."""
    ps = 16
    seg_ctx = [1, 15, 16, 17, 64, 65, 127, 128, 129, 700, 2050]
    S = len(seg_ctx)
    c = paged_case(ops, torch.bfloat16, n_head, n_kv_head, hd, ps, window, seg_ctx, [1] * S, seed=hd + n_head)
    q = torch.zeros(S + 1, n_head * hd, dtype=torch.bfloat16, device="cuda")
    q[:S] = c["q"].cuda()
    row_seq = dev(torch.cat([c["row_seq"], torch.tensor([-1], dtype=torch.int32)]))
    positions = dev(torch.cat([c["positions"], torch.tensor([0], dtype=torch.int32)]))
    slots = torch.full((S + 1,), -1, dtype=torch.int32, device="cuda")
    counters = torch.zeros((S + 1) * n_head, dtype=torch.int32, device="cuda")
    sinks = torch.randn(n_head, generator=torch.Generator().manual_seed(1)).cuda()
    for extra in ({}, {"sinks": sinks}, {"cap": 3.0}, {"keep": 20}) if window else ({}, {"sinks": sinks}, {"cap": 3.0}):
        def run(nsplit, plan, floats):
            out = torch.full((S + 1, n_head * hd), float("nan"), dtype=torch.bfloat16, device="cuda")
            ops.paged_decode_bf16(q, -1, -1, c["kc"], c["vc"], dev(c["bt"]), row_seq, positions, slots, out,
                                  torch.full((max(floats, 1),), float("nan"), device="cuda"), counters, n_head, n_kv_head, hd, ps,
                                  c["scale"], window, nsplit, plan=plan, **extra)
            assert int(counters.abs().sum()) == 0
            return out
        plan = ops.decode_plan(row_seq, positions, S + 1, n_head, max(seg_ctx), hd, window, extra.get("keep", 0))
        got, even = run(0, plan, n_head * plan.shape[0] * (hd + 2)), run(1, None, 0)
        if not extra and window >= 0:
            assert (got[:S].double().cpu() - c["ref"]).abs().max() < 1e-2 * max(1.0, c["ref"].abs().max().item())
        assert torch.equal(got[S], torch.zeros_like(got[S]))
        # each of the two is its own sums rounded once to bfloat16 (2^-9 of the value): they differ by two such roundings at most
        assert ((got - even)[:S].abs() <= 2 ** -7 * even[:S].abs().float() + 1e-5).all(), extra
