"""The order of a norm's sum over the four warps of its block."""
import pytest
import torch

from test_kernels import dev, ops      # noqa: F401  (a fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [512, 768, 2048])
def test_the_warps_sums_are_added_as_the_block_wide_sum_adds_them(ops, d):
    """Four warps with the sums 2^30, 1, -2^30 and 1: first with third and second with fourth, as the shuffles of the sum over
    a whole block pair them, the total is 2; in the warps' own order it is 0.  A column that holds 0 shows the mean."""
    x = torch.zeros(2, d)
    x[:, 0], x[:, 128], x[:, 256], x[:, 384] = 2.0 ** 30, 1.0, -2.0 ** 30, 1.0      # a thread has 4 columns, a warp 128
    out = torch.empty(2, d, device="cuda")
    ops.add_layernorm(dev(x), None, None, dev(torch.ones(d)), dev(torch.zeros(d)), 1e-5, out)
    want = -(2.0 / d) / (2.0 ** 61 / d) ** 0.5
    assert ((out[:, 1].cpu() - want).abs() <= 4e-7 * abs(want)).all()      # the mean, the root and two products, each rounded once
