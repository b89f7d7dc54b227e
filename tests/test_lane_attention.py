"""The general attention kernel's form with a key a lane, against 64 bits."""
import pytest
import torch

from test_kernels import dev, ops      # noqa: F401  (a fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hd,hd_v", [(4, 4), (32, 32), (40, 24), (64, 64), (100, 128), (128, 128)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_a_lane_a_key(ops, hd, hd_v, dtype):
    """The general attention kernel's form with a key a lane: 1..97 keys (below, at and above its groups of 32), widths that
    do not fill the lanes, page sizes that are no power of two, against 64 bits."""
    if dtype == torch.bfloat16 and hd % 8:
        hd, hd_v = 8 * (hd // 8 + 1), hd_v
    g = torch.Generator().manual_seed(hd)
    for ps in (5, 16):
        lens, H = [1, 2, 31, 32, 33, 64, 65, 97], 3
        pages = 64
        kc, vc = torch.randn(pages, H, ps, hd, generator=g).to(dtype), torch.randn(pages, H, ps, hd_v, generator=g).to(dtype)
        bt = torch.stack([torch.randperm(pages, generator=g)[:20] for _ in lens]).int()
        q = torch.randn(len(lens), H * hd, generator=g).to(dtype)
        out = torch.empty(len(lens), H * hd_v, dtype=dtype, device="cuda")
        ops.paged_attention_generic(dev(q), dev(kc), dev(vc), dev(bt), torch.arange(len(lens), dtype=torch.int32, device="cuda"),
                                    torch.tensor([n - 1 for n in lens], dtype=torch.int32, device="cuda"), out, H, H, hd, ps,
                                    hd ** -0.5, v_head_dim=hd_v)
        for r, n in enumerate(lens):
            for h in range(H):
                at = [(int(bt[r, j // ps]), j % ps) for j in range(n)]
                k, v = (torch.stack([t[p, h, o] for p, o in at]).double() for t in (kc, vc))
                w = torch.softmax(k @ q[r, h * hd:(h + 1) * hd].double() * hd ** -0.5, 0)
                tol = 2e-6 if dtype == torch.float32 else 2 ** -8      # 32-bit sums of up to 97 terms of order one; one rounding
                assert (out[r, h * hd_v:(h + 1) * hd_v].double().cpu() - w @ v).abs().max() < tol * 4, (ps, n)
