"""Routing with eight warps a row and with more."""
import pytest
import torch

from test_kernels import dev, ops      # noqa: F401  (a fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("E", [8, 9, 31, 48, 130])
@pytest.mark.parametrize("rows", [296, 297, 445, 593])
def test_a_rows_choice_is_the_same_among_few_rows_and_many(ops, rows, E, dtype):
    """The number of warps a row gets changes with the rows and the experts; its sums do not: the bits are those of the same rows
    ten at a time, and the choice is the scores' order in 64 bits where neighbouring scores are not too close."""
    W, top = 72, 3
    g = torch.Generator().manual_seed(rows + E)
    h, r = torch.randn(rows, W, generator=g).to(dtype), torch.randn(E + 1, W, generator=g).to(dtype)

    def run(part):
        n = part.shape[0]
        ids, w, side = torch.empty(n, top, dtype=torch.int32, device="cuda"), torch.empty(n, top, device="cuda"), torch.empty(n, device="cuda")
        ops.route_topk(part, dev(r), top, "softmax", True, ids, w, side=side)
        return ids, w, side
    got = run(dev(h))
    few = [torch.cat(t) for t in zip(*(run(p) for p in dev(h).split(10)))]
    assert all(torch.equal(a, b) for a, b in zip(got, few))
    z = (h.double() @ r[:E].double().t()).sort(dim=1, descending=True)
    clear = (z.values[:, :top] - z.values[:, 1:top + 1]).min(1).values > 1e-4      # 72 products of about 1 in 32-bit sums
    assert clear.float().mean() > 0.9 and torch.equal(got[0].cpu()[clear], z.indices[clear, :top].int())
