"""The inside of a gated feed-forward for a few rows in one kernel, against 64 bits."""
import pytest
import torch

from test_kernels import dev, ops      # noqa: F401  (a fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 7, 8, 9, 16])
@pytest.mark.parametrize("F,K", [(8, 8), (43, 72), (1408, 2048), (3600, 40), (5440, 264), (200, 4096)])
def test_gated_linear(ops, M, F, K):
    """Both forms the launcher chooses, the 64-register one and the general one;
    columns and K that fill no block; biases, a number per row, the cut and the shift.  The two sums (K terms in 32-bit) are
    rounded to bfloat16, the result is: 2^-9 of each of the two carried through the product, doubled for sums that lie at a
    rounding's edge, and 2^-9 of the result."""
    g = torch.Generator().manual_seed(M * F + K)
    x, w = torch.randn(M, K + 8, generator=g).bfloat16()[:, :K], (torch.randn(2 * F, K, generator=g) / K ** 0.5).bfloat16()
    b, rg = torch.randn(2 * F, generator=g), torch.rand(M, generator=g)
    xd = dev(torch.cat([x, torch.zeros(M, 8).bfloat16()], 1))[:, :K]
    assert ops.gated_linear_takes(xd, dev(w))
    for bias, row_gate, act, kw in ((None, None, "silu", {}), (b, None, "gelu_tanh", {}),
                                    (b, rg, "silu", dict(limit=0.8, beta=1.702, shift=1.0))):
        out = torch.full((M, F + 3), float("nan"), dtype=torch.bfloat16, device="cuda")
        ops.gated_linear(xd, dev(w), None if bias is None else dev(bias), act, out[:, :F],
                         row_gate=None if row_gate is None else dev(row_gate), **kw)
        s = x.double() @ w.double().t() + (0 if bias is None else bias.double())
        gate, up = s[:, :F], s[:, F:]
        if kw:
            gate, up = gate.clamp(max=kw["limit"]), up.clamp(-kw["limit"], kw["limit"]) + kw["shift"]
        a = gate * torch.sigmoid(kw.get("beta", 1.0) * gate) if act == "silu" else torch.nn.functional.gelu(gate, approximate="tanh")
        ref = a * up * (1 if row_gate is None else row_gate.double()[:, None])
        rg_ = 1 if row_gate is None else row_gate.double()[:, None]
        carried = (1.8 * gate.abs() * up.abs() + a.abs() * (up.abs() + kw.get("shift", 0.0))) * rg_      # |a'(g)| <= 1.8 for either activation
        assert ((out[:, :F].double().cpu() - ref).abs() <= 2 ** -8 * carried + 2 ** -8 * ref.abs() + 1e-5 * K ** 0.5).all()
        assert torch.isnan(out[:, F:]).all()


@pytest.mark.parametrize("M", [1, 8, 9, 16])
@pytest.mark.parametrize("F,K", [(43, 72), (704, 1024), (1408, 2048), (2368, 2048), (3600, 40)])
def test_one_kernel_or_two_give_the_same_bits(ops, M, F, K):
    """Wherever one kernel takes the place of the product and the gated product it has their sums and roundings, bit for bit;
    where the product splits K over a cluster (other groups of sums) the two stay."""
    assert ops.gated_linear_pays(M, F, K) == (M > 8 or (F, K) != (1408, 2048))
    if not ops.gated_linear_pays(M, F, K):
        return
    g = torch.Generator().manual_seed(M + F + K)
    x, w = dev(torch.randn(M, K, generator=g).bfloat16()), dev((torch.randn(2 * F, K, generator=g) / K ** 0.5).bfloat16())
    b, rg = dev(torch.randn(2 * F, generator=g)), dev(torch.rand(M, generator=g))
    for kw in ({}, dict(limit=0.8, beta=1.702, shift=1.0, row_gate=rg)):
        one, two = (torch.empty(M, F, dtype=torch.bfloat16, device="cuda") for _ in range(2))
        ops.gated_linear(x, w, b, "silu", one, **kw)
        gu = ops.linear(x, w, b)
        ops.gate_mul(gu[:, :F], gu[:, F:], "silu", two, **kw)
        assert torch.equal(one, two)
