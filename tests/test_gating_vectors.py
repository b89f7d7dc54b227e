"""Unit norms and gated products in 16-byte pieces: sizes around what a block and a thread hold, against 64 bits."""
import pytest
import torch

from test_kernels import dev, ops      # noqa: F401  (a fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("pw,parts", [(8, 3), (40, 1), (256, 2), (4096, 1), (4104, 1), (8192, 1), (8200, 1), (12, 2)])
def test_rms_norm(ops, dtype, pw, parts):
    """Parts within one piece a thread, two, and more than the vector form takes; widths that are no multiple of 8."""
    g = torch.Generator().manual_seed(pw)
    n, rows = pw * parts, 5
    x, z, w = torch.randn(rows, n, generator=g), torch.randn(rows, n + 8, generator=g).to(dtype)[:, :n], torch.rand(n, generator=g) + 0.5
    v = x.double()
    for weight, gate, after, act in ((w, None, False, "silu"), (None, z, False, "silu"), (w, z, True, "sigmoid")):
        a = None if gate is None else (torch.sigmoid(z.double()) if act == "sigmoid" else torch.nn.functional.silu(z.double()))
        u = v if a is None or after else v * a
        u = u.view(rows, parts, pw)
        ref = (u / torch.sqrt((u * u).mean(-1, keepdim=True) + 1e-5)).view(rows, n)
        ref = ref * (1 if weight is None else weight.double()) * (a if after and a is not None else 1)
        out = torch.full((rows, n + 8), float("nan"), dtype=dtype, device="cuda")
        gd = None if gate is None else dev(torch.cat([z, torch.zeros(rows, 8).to(dtype)], 1))[:, :n]
        ops.rms_norm(dev(x), None if weight is None else dev(weight), 1e-5, out[:, :n], parts=parts, gate=gd, gate_act=act, gate_after=after)
        tol = 2e-6 if dtype == torch.float32 else 2 ** -8      # 32-bit sums of pw terms; one rounding
        assert ((out[:, :n].double().cpu() - ref).abs() <= tol * ref.abs() + 2e-6).all() and torch.isnan(out[:, n:]).all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n", [8, 72, 2040, 2048, 2056, 5632, 13])
def test_gate_mul(ops, dtype, n):
    g = torch.Generator().manual_seed(n)
    rows = 7
    both = torch.randn(rows, 2 * n, generator=g).to(dtype)
    table, at, rg = torch.randn(9, n, generator=g).to(dtype), torch.tensor([0, 8, 3, -1, 9, 5, 5], dtype=torch.int32), torch.rand(rows, generator=g)
    d = dev(both)
    a, b = both[:, :n].double(), both[:, n:].double()
    looked = torch.stack([table[t].double() if 0 <= t < 9 else torch.zeros(n).double() for t in at.tolist()])
    for act, bd, br, kw, ref in (("silu", d[:, n:], None, {}, torch.nn.functional.silu(a) * b),
                                 ("silu", d[:, n:], None, dict(limit=0.7, beta=1.702, shift=1.0, row_gate=dev(rg)),
                                  a.clamp(max=0.7) * torch.sigmoid(1.702 * a.clamp(max=0.7)) * (b.clamp(-0.7, 0.7) + 1) * rg.double()[:, None]),
                                 ("gelu_tanh", dev(table), dev(at), {}, torch.nn.functional.gelu(a, approximate="tanh") * looked),
                                 ("relu2", d[:, n:], None, {}, a.clamp(min=0) ** 2 * b)):
        out = torch.empty(rows, n, dtype=dtype, device="cuda")
        ops.gate_mul(d[:, :n], bd, act, out, b_rows=br, **kw)
        tol = 2e-6 if dtype == torch.float32 else 2 ** -8
        assert ((out.double().cpu() - ref).abs() <= tol * ref.abs() + 1e-6).all(), act


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,n", [(313, 256), (304, 264), (41, 2040), (40, 2048), (39, 2056), (17, 5632), (400, 248), (8, 10000)])
def test_gate_mul_of_many_products(ops, dtype, rows, n):
    """80,000 products and more, which go 16 bytes a thread where a row has 256 columns: around a block's 2,048 columns, one row of
    threads that are not all used, and (248) the other form."""
    g = torch.Generator().manual_seed(n)
    both, table = torch.randn(rows, 2 * n, generator=g).to(dtype), torch.randn(9, n, generator=g).to(dtype)
    at, rg = torch.randint(-1, 10, (rows,), generator=g).int(), torch.rand(rows, generator=g)
    d, a, b = dev(both), both[:, :n].double(), both[:, n:].double()
    looked = torch.cat([table.double(), torch.zeros(1, n).double()])[torch.where((at < 0) | (at > 8), 9, at).long()]
    for bd, br, kw, ref in ((d[:, n:], None, dict(limit=0.7, beta=1.702, shift=1.0, row_gate=dev(rg)),
                             a.clamp(max=0.7) * torch.sigmoid(1.702 * a.clamp(max=0.7)) * (b.clamp(-0.7, 0.7) + 1) * rg.double()[:, None]),
                            (dev(table), dev(at), {}, torch.nn.functional.silu(a) * looked)):
        out = torch.full((rows, n + 8), float("nan"), dtype=dtype, device="cuda")
        ops.gate_mul(d[:, :n], bd, "silu", out[:, :n], b_rows=br, **kw)
        tol = 2e-6 if dtype == torch.float32 else 2 ** -8
        assert ((out[:, :n].double().cpu() - ref).abs() <= tol * ref.abs() + 1e-6).all() and torch.isnan(out[:, n:]).all()


def test_rms_norm_of_many_narrow_gated_parts(ops):
    """Parts below 256 columns with a gate go 16 bytes a thread from 350,000 values on; below that, and below 128 columns, not."""
    g = torch.Generator().manual_seed(3)
    for rows, parts, pw in ((330, 8, 136), (300, 8, 136), (700, 8, 72)):
        x, z = torch.randn(rows, parts * pw, generator=g), torch.randn(rows, parts * pw, generator=g).bfloat16()
        u = (x.double() * torch.nn.functional.silu(z.double())).view(rows, parts, pw)
        ref = (u / torch.sqrt((u * u).mean(-1, keepdim=True) + 1e-5)).view(rows, -1)
        out = torch.empty(rows, parts * pw, dtype=torch.bfloat16, device="cuda")
        ops.rms_norm(dev(x), None, 1e-5, out, parts=parts, gate=dev(z))
        assert ((out.double().cpu() - ref).abs() <= 2 ** -8 * ref.abs() + 2e-6).all()
