"""The 32-bit product of up to 16 rows with every length of its ring of pieces."""
import pytest
import torch

from test_kernels import dev, ops      # noqa: F401  (a fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [40, 2400, 7201])      # one block of 16 columns an SM, up to three, more: rings of 4, 2 and 1
@pytest.mark.parametrize("K", [4, 256, 260, 512, 1100, 2052])
def test_few_rows_have_the_bits_of_many(ops, N, K):
    """Every kernel sums along K in one order: 1, 5 and 16 rows give the bits of the same rows among 20 (the tiled kernel)."""
    g = torch.Generator().manual_seed(N + K)
    x, w, b = dev(torch.randn(20, K, generator=g)), dev(torch.randn(N, K, generator=g)), dev(torch.randn(N, generator=g))
    want = torch.empty(20, N, device="cuda")
    ops.linear_f32(x, w, b, "gelu_erf", want, w_is_nk=True)
    for M in (1, 5, 16):
        out = torch.full((M, N), float("nan"), device="cuda")
        ops.linear_f32(x[:M], w, b, "gelu_erf", out, w_is_nk=True)
        assert torch.equal(out, want[:M])
