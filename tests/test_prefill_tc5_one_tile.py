"""Prompt attention on tcgen05 where a row tile sees one 64-key tile (one block of the cluster works alone) beside some that see more."""
import numpy as np
import pytest
import torch

from test_kernels import dev, ops, paged_case      # noqa: F401  (a fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("how", ["plain", "sinks", "cap", "keep", "bias"])
@pytest.mark.parametrize("hd", [64, 128])
def test_one_tile(ops, hd, how):
    n_head, ps = 3, 16
    window = 40 if how == "keep" else 0
    seg_ctx, seg_rows = [1, 17, 64, 64, 65, 300, 140, 250], [1, 17, 64, 3, 65, 1, 12, 130]
    c = paged_case(ops, torch.bfloat16, n_head, n_head, hd, ps, window, seg_ctx, seg_rows, seed=hd)
    S, T = len(seg_ctx), len(c["positions"])
    g = torch.Generator().manual_seed(1)
    kw = {"plain": {}, "sinks": dict(sinks=dev(torch.randn(n_head, generator=g) * 2)), "cap": dict(cap=2.0), "keep": dict(keep=5),
          "bias": dict(slopes=dev(torch.rand(n_head, generator=g)), rates=dev(torch.rand(n_head, generator=g)))}[how]
    cu = dev(torch.tensor([0] + list(np.cumsum(seg_rows)), dtype=torch.int32))
    start = dev(torch.tensor([cx - n for cx, n in zip(seg_ctx, seg_rows)], dtype=torch.int32))
    q, bt, pos = dev(c["q"]), dev(c["bt"]), dev(c["positions"])
    want = torch.empty_like(q)
    ops.paged_attention_generic(q, c["kc"], c["vc"], bt, dev(c["row_seq"]), pos, want, n_head, n_head, hd, ps, c["scale"], window, **kw)
    for n_chunks, chunk_keys in [(1, 0), (5, 64), (3, 128)]:
        partial = torch.full((T * n_head * n_chunks * (hd + 4),), float("nan"), device="cuda") if n_chunks > 1 else None
        out = torch.full_like(q, float("nan"))
        ops.paged_prefill_tc5(q, c["kc"], c["vc"], bt, cu, start, out, 0, S, max(seg_rows), n_head, n_head, hd, ps, c["scale"], window,
                              (n_chunks, chunk_keys), partial, pos, 0, T, **kw)
        assert ops.tcgen05_error_flag("cuda").item() == 0
        # P is rounded to bfloat16 (2^-9 of each weight), both results once more
        assert (out.float() - want.float()).abs().max() < 1.5e-2 * max(1.0, want.float().abs().max().item()), (n_chunks, chunk_keys)
