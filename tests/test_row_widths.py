"""Kernels that keep a row in shared memory, at the widths where the row and what the kernel holds besides pass 48 KB together."""
import pytest
import torch

from test_kernels import dev, ops      # noqa: F401  (a fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("d", [6120, 6127, 6144, 6145, 25568])
def test_add_rmsnorm(ops, d, out_dtype):
    g = torch.Generator().manual_seed(d)
    x, delta, w = torch.randn(2, d, generator=g), torch.randn(2, d, generator=g), torch.randn(d, generator=g)
    xd, out = dev(x), torch.empty(2, d, dtype=out_dtype, device="cuda")
    ops.add_rmsnorm(xd, dev(delta), None, None, dev(w), 1e-6, 1.0, out)
    v = x.double() + delta.double()
    ref = v / (v.pow(2).mean(1, keepdim=True) + 1e-6).sqrt() * (1.0 + w.double())
    tol = 1e-6 if out_dtype == torch.float32 else 2 ** -8      # a few 32-bit roundings; one to bfloat16
    assert ((out.double().cpu() - ref).abs() <= tol * ref.abs() + 1e-6).all()
    assert (xd.double().cpu() - v).abs().max() <= 1e-6


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("width, dims", [(6080, 128), (6080, 60), (6016, 256), (6100, 90), (6110, 2)])
def test_qk_prepare(ops, width, dims, dtype):
    """q and k of one head each, normalised and rotated."""
    g = torch.Generator().manual_seed(width)
    buf = torch.randn(2, 2 * width, generator=g).to(dtype)
    qw, kw = torch.randn(width, generator=g), torch.randn(width, generator=g)
    pos, freqs = torch.tensor([3, 11], dtype=torch.int32), torch.rand(dims // 2, generator=g)
    got = dev(buf)
    ops.qk_prepare(got, 0, 1, width, 1, width, dev(qw), dev(kw), 1e-6, dev(pos), dev(freqs), dims)
    c, s = ((pos[:, None].float() * freqs[None]).double().cos(), (pos[:, None].float() * freqs[None]).double().sin())
    half, tol = dims // 2, 3e-6 if dtype == torch.float32 else 2 ** -8
    for at, w in ((0, qw), (width, kw)):
        v = buf[:, at:at + width].double()
        v = v / (v.pow(2).mean(1, keepdim=True) + 1e-6).sqrt() * w.double()
        a, b = v[:, :half].clone(), v[:, half:dims].clone()
        v[:, :half], v[:, half:dims] = a * c - b * s, b * c + a * s
        assert (got[:, at:at + width].double().cpu() - v).abs().max() <= tol * v.abs().max()
