"""32-bit products of a few rows with 4, 8 and 16 columns a block: at the edges of the rule that chooses among them and at odd
columns, the bits of the tiled kernels (one multiply-add after the other along k)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [1, 5, 256, 296, 297, 592, 593, 1184, 1185, 2500])
@pytest.mark.parametrize("K", [4, 16, 20, 124, 128, 252, 256, 300, 768, 1044])
def test_few_rows_have_the_bits_of_the_tiled_kernel(N, K):
    from cbis_b200.kernels import ops
    g = torch.Generator().manual_seed(N + K)
    x, w, b = torch.randn(16, K, generator=g).cuda(), torch.randn(N, K, generator=g).cuda(), torch.randn(N, generator=g).cuda()
    want = torch.empty(32, N, device="cuda")
    ops.linear_f32(torch.cat([x, x]), w, b, None, want, w_is_nk=True)      # more than 16 rows: tiles
    for rows in (1, 4, 5, 7, 16):
        got = torch.full((rows, N), float("nan"), device="cuda")
        ops.linear_f32(x[:rows], w, b, None, got, w_is_nk=True)
        assert torch.equal(got, want[:rows])
