"""The routed feed-forward's tiles at the sizes where they can go wrong, against 64 bits."""
import pytest
import torch

from test_kernels import dev, ops      # noqa: F401  (a fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,W,F,E,top", [(300, 264, 136, 3, 2), (130, 512, 128, 2, 1), (33, 1032, 264, 5, 3), (700, 256, 520, 1, 1),
                                            (129, 8, 8, 4, 2), (400, 320, 72, 40, 2)])
@pytest.mark.parametrize("weight_on_input", [True, False])
def test_tiles(ops, rows, W, F, E, top, weight_on_input):
    """More and fewer than 128 pairs an expert, experts that nobody chose, columns past a tile of 128 hidden or 256 result
    columns, K past the ring of four stages and in no whole pieces, a strided input.  The hidden values are rounded to bfloat16
    (2^-9 of each, F of them added up) and so are not the sums; the bound is on the result's size."""
    g = torch.Generator().manual_seed(rows + W)
    h = torch.randn(rows, W + 16, generator=g).bfloat16()
    gu, dn = (torch.randn(E, 2 * F, W, generator=g) / W ** 0.5).bfloat16(), (torch.randn(E, W, F, generator=g) / F ** 0.5).bfloat16()
    ids = torch.stack([torch.randperm(E, generator=g)[:top] for _ in range(rows)]).int()
    if E == 40:
        ids[:200, 0] = 7                     # one long run of tiles beside experts with a row or two
        ids[:200, 1] = 8 + torch.arange(200) % 30
    wt = torch.rand(rows, top, generator=g)
    hd = dev(h)[:, 8:8 + W]
    assert ops.routed_tiles_takes(hd, dev(gu), dev(dn))
    out = torch.full((rows, W), float("nan"), device="cuda")
    ops.routed_tiles(hd, dev(gu), dev(dn), dev(ids), dev(wt), "silu", weight_on_input, out)
    x, ref = h[:, 8:8 + W].double(), torch.zeros(rows, W, dtype=torch.float64)
    for k in range(top):
        for e in range(E):
            r = (ids[:, k] == e).nonzero()[:, 0]
            w = wt[r, k].double()[:, None]
            s = (x[r] * (w if weight_on_input else 1)) @ gu[e].double().t()
            a = torch.nn.functional.silu(s[:, :F]) * s[:, F:]
            ref[r] += (a @ dn[e].double().t()) * (1 if weight_on_input else w)
    assert (out.double().cpu() - ref).abs().max() < 2 ** -7 * max(1.0, ref.abs().max())
    ops.raise_if_kernel_errors()


@pytest.mark.parametrize("rows,W,F,E,top", [(300, 264, 136, 3, 2), (33, 1032, 264, 5, 3), (129, 8, 8, 4, 2), (400, 320, 72, 40, 2)])
def test_tiles_without_tcgen05(ops, monkeypatch, rows, W, F, E, top):
    """With tcgen05 switched off the rows still go sorted by expert, on mma.sync tiles (128 rows, 64 columns, K in pieces of 32)."""
    monkeypatch.setattr(ops, "USE_TCGEN05", False)
    test_tiles(ops, rows, W, F, E, top, True)
    test_tiles(ops, rows, W, F, E, top, False)
