"""32-bit prompt attention on the tensor cores (head sizes up to 64, 32-bit values in three bfloat16 parts): its error
against 64 bits beside the multiply-add kernel's, and values that cannot be cut into parts."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def run(q, k, v, n_head, hd, ps, window=0, chunks=(1, 0)):
    """The last rows of one sequence (all of it, or a portion behind a context), pages in a mixed order -> (tiled form, general
    form), [rows, heads * hd]."""
    from cbis_b200.kernels import ops
    T, rows = k.shape[0], q.shape[0]
    n_kv_head, n_pages = k.shape[1], -(-T // ps)
    bt = torch.randperm(n_pages, generator=torch.Generator().manual_seed(T)).to(torch.int32)
    kc, vc = (torch.zeros(n_pages, n_kv_head, ps, hd, device="cuda") for _ in range(2))
    pos = torch.arange(T)
    for cache, values in ((kc, k), (vc, v)):
        cache[bt[pos // ps].long().cuda(), :, (pos % ps).cuda()] = values.cuda()
    cu = torch.tensor([0, rows], dtype=torch.int32, device="cuda")
    start = torch.tensor([T - rows], dtype=torch.int32, device="cuda")
    pos = pos[T - rows:].to(torch.int32).cuda()
    bt = bt[None].contiguous().cuda()
    qd = q.reshape(rows, -1).cuda()
    tiled, general = torch.empty_like(qd), torch.empty_like(qd)
    partial = torch.full((rows * n_head * chunks[0] * (hd + 4),), float("nan"), device="cuda") if chunks[0] > 1 else None
    ops.paged_prefill_f32(qd, kc, vc, bt, cu, start, tiled, 0, 1, rows, n_head, n_kv_head, hd, ps, hd ** -0.5, window, chunks, partial,
                          pos, 0, rows)
    ops.paged_attention_generic(qd, kc, vc, bt, torch.zeros(rows, dtype=torch.int32, device="cuda"), pos, general, n_head,
                                n_kv_head, hd, ps, hd ** -0.5, window)
    return tiled.cpu(), general.cpu()


def exact(q, k, v, hd, window=0):
    rows, H = q.shape[:2]
    T, per = k.shape[0], H // k.shape[1]
    k, v = (x.double().repeat_interleave(per, 1).permute(1, 0, 2) for x in (k, v))
    s = torch.matmul(q.double().permute(1, 0, 2), k.transpose(1, 2)) * hd ** -0.5
    back = torch.arange(T - rows, T)[:, None] - torch.arange(T)[None]
    s.masked_fill_((back < 0) | ((back >= window) if window else False), float("-inf"))
    return torch.matmul(torch.softmax(s, -1), v).permute(1, 0, 2).reshape(rows, -1)


@pytest.mark.parametrize("T", [1, 63, 64, 65, 700])
@pytest.mark.parametrize("hd, n_head, n_kv_head, size", [(16, 2, 1, 1.0), (32, 2, 2, 3.0), (48, 1, 1, 0.01), (64, 2, 1, 1.0)])
def test_error_against_64_bits(T, hd, n_head, n_kv_head, size):
    g = torch.Generator().manual_seed(T + hd)
    q, k, v = (torch.randn(T, n, hd, generator=g) * size for n in (n_head, n_kv_head, n_kv_head))
    v = v + 2.0          # sums that do not cancel
    tiled, general = run(q, k, v, n_head, hd, 16)
    ref = exact(q, k, v, hd)
    e_tiled, e_general = ((x.double() - ref).norm() / ref.norm() for x in (tiled, general))
    # the other form sums 32-bit products one by one: no further from 64 bits than that (and than half a unit in the last
    # place of every output, 3e-8 in this norm, where both are that close)
    assert e_tiled <= 1.2 * e_general + 3e-8, (e_tiled, e_general)


@pytest.mark.parametrize("hd, window", [(16, 0), (32, 0), (32, 1000), (48, 0), (64, 300)])
@pytest.mark.parametrize("one_sign", [False, True])
def test_error_behind_a_long_context(hd, window, one_sign):
    """150 rows behind 8,000 keys, the keys whole and cut into chunks that are merged, also with all of q, k and v of one sign, where
    sums that the tensor cores cut off would all be cut the same way: the bound of the test above, which the general form's
    long sums leave far behind, and an absolute one (its rows' 32-bit weights and sums, some 2^-23 of each other)."""
    g = torch.Generator().manual_seed(hd)
    q, k, v = (torch.randn(n, 2, hd, generator=g) for n in (150, 8150, 8150))
    if one_sign:
        q, k, v = q.abs(), k.abs(), v.abs()
    v = v + 2.0
    ref = exact(q, k, v, hd, window)
    for chunks in ((1, 0), (32, 256), (5, 2048)):
        tiled, general = run(q, k, v, 2, hd, 16, window, chunks)
        e_tiled, e_general = ((x.double() - ref).norm() / ref.norm() for x in (tiled, general))
        assert e_tiled <= min(1.2 * e_general + 3e-8, 8e-7), (chunks, e_tiled, e_general)


@pytest.mark.parametrize("T", [64, 150])
@pytest.mark.parametrize("hd", [16, 32, 48, 64])
def test_error_with_large_scores(hd, T):
    """Scores of twenty and more over few keys, where a row's error is that of its largest scores: a sum of head-size products
    whose addends the tensor cores cut off at 2^-24 of the largest one, sixteen at a time, instead of rounding.  Twice the general
    form's error."""
    g = torch.Generator().manual_seed(T + hd)
    q, k, v = (torch.randn(T, 2, hd, generator=g) for _ in range(3))
    q, v = q * 6, v + 2.0
    tiled, general = run(q, k, v, 2, hd, 16)
    ref = exact(q, k, v, hd)
    e_tiled, e_general = ((x.double() - ref).norm() / ref.norm() for x in (tiled, general))
    assert e_tiled <= 2 * e_general + 3e-8, (e_tiled, e_general)


@pytest.mark.parametrize("hd", [16, 32, 48, 64])
@pytest.mark.parametrize("size", [1e-30, 1e-35, 1e-38, 1e-41])
def test_small_values(hd, size):
    """Values down to the smallest that 32 bits hold, whose third parts as they are would be too small for bfloat16: the bound of
    the test above, with half a step of such numbers (7e-46) for every rounding of an output."""
    g = torch.Generator().manual_seed(hd)
    q, k, v = (torch.randn(150, 2, hd, generator=g) for _ in range(3))
    v = (v + 2.0) * size
    tiled, general = run(q, k, v, 2, hd, 16)
    ref = exact(q, k, v, hd)
    e_tiled, e_general = ((x.double() - ref).norm() / ref.norm() for x in (tiled, general))
    assert e_tiled <= 1.2 * e_general + 3e-8 + 7e-46 / size, (e_tiled, e_general)


@pytest.mark.parametrize("window", [0, 40])
@pytest.mark.parametrize("hd", [16, 32, 48, 64])
@pytest.mark.parametrize("what, value", [("k", float("-inf")), ("k", 1e30), ("v", float("inf")), ("v", -3e38), ("v", float("nan")),
                                         ("q", 1e20), ("q", float("inf"))])
def test_values_that_cannot_be_cut(hd, what, value, window):
    """One such value, at position 70, in a tile with rows that see it and rows that do not (those before it, with a window those
    far behind it): all rows are those of the general form, which walks only the keys that a row sees."""
    T, at = 200, 70
    g = torch.Generator().manual_seed(hd)
    q, k, v = (torch.randn(T, 2, hd, generator=g) for _ in range(3))
    q[:, :, 3] = q[:, :, 3].abs() + 0.1
    {"q": q, "k": k, "v": v}[what][at, 1, 3] = value
    tiled, general = run(q, k, v, 2, hd, 16, window)
    assert torch.equal(torch.isfinite(tiled), torch.isfinite(general))
    assert torch.allclose(tiled, general, rtol=3e-6, atol=3e-6, equal_nan=True)
