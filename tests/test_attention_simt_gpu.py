"""The CUDA-core attention with few and many queries a warp: against 64 bits, and the same bits for a
query whichever of them its step takes."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("hd,window", [(64, 0), (48, 21), (128, 0), (20, 0), (288, 0)])
@pytest.mark.parametrize("n,before", [(4, 29), (5, 0), (16, 17), (17, 64), (33, 0), (70, 3)])
def test_attention_simt_queries_a_warp(dtype, hd, window, n, before):
    from scratch_llm_b200.kernels import ops
    ops.prepare_jobs([ops.attention_library(hd)], verbose=False)
    H, G, page = 4, 2, 16
    gen = torch.Generator().manual_seed(n + hd)
    total = before + n
    n_pages = -(-total // page)
    pages = torch.randn(n_pages, 2, G, page, hd, generator=gen).to(dtype).to(DEV)
    q = torch.randn(n, H * hd, generator=gen).to(dtype).to(DEV)
    table = torch.randperm(n_pages, generator=gen).to(torch.int32).view(1, -1).to(DEV)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731

    def attend(first, count):
        out = torch.empty(count, H * hd, dtype=dtype, device=DEV)
        ops.attention_simt(q[first:first + count], pages, table, page, i32([0, count]), i32([before + first]),
                           out, 1, count, H, G, hd, hd ** -0.5, window or None)
        return out

    got = attend(0, n)
    assert torch.equal(got, torch.cat([attend(t, 1) for t in range(n)]))
    kv = pages.double().cpu()[table[0].long().cpu()].permute(1, 2, 0, 3, 4).reshape(2, G, -1, hd)[:, :, :total]
    k, v = kv.repeat_interleave(H // G, 1)
    s = torch.einsum("nhd,hkd->hnk", q.double().cpu().view(n, H, hd), k) * hd ** -0.5
    qpos, kpos = torch.arange(before, total)[:, None], torch.arange(total)[None]
    s.masked_fill_((kpos > qpos) | ((kpos <= qpos - window) if window else False), float("-inf"))
    want = torch.einsum("hnk,hkd->nhd", torch.softmax(s, -1), v).reshape(n, -1)
    # 32-bit sums of hd and of `total` products; bfloat16 rounds the result
    tol = 2e-6 if dtype == torch.float32 else 2 ** -8
    assert ((got.double().cpu() - want).norm() / want.norm()).item() < tol


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
# head sizes of no whole 16-byte words, and pages that start on none: read one element at a time
@pytest.mark.parametrize("hd,odd", [(15, 0), (130, 0), (64, 1), (48, 1), (128, 0)])
@pytest.mark.parametrize("window", [0, 37])
def test_attention_simt_rows_of_all_lengths(dtype, hd, odd, window):
    """Rows of few tokens beside long ones, in launches for as many tokens as they have or more: the same
    bits as alone."""
    from scratch_llm_b200.kernels import ops
    ops.prepare_jobs([ops.attention_library(hd)], verbose=False)
    H, G, page = 4, 2, 16
    rows = [(70, 1), (0, 40), (5, 4), (31, 1), (0, 0), (64, 18), (90, 5), (3, 33)]      # (cached, new)
    gen = torch.Generator().manual_seed(hd)
    need = [-(-(b + n) // page) for b, n in rows]
    flat = torch.randn(sum(need) * 2 * G * page * hd + odd, generator=gen).to(dtype).to(DEV)
    pages = flat[odd:].view(sum(need), 2, G, page, hd)
    n = sum(x for _, x in rows)
    q = torch.randn(n, H * hd, generator=gen).to(dtype).to(DEV)
    table = torch.full((len(rows), max(need)), -1, dtype=torch.int32)
    for r, k in enumerate(need):
        table[r, :k] = torch.arange(sum(need[:r]), sum(need[:r]) + k)
    table = table.to(DEV)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    first = [sum(x for _, x in rows[:r]) for r in range(len(rows) + 1)]

    def attend(which, max_new):
        some = torch.cat([q[first[r]:first[r + 1]] for r in which])
        out = torch.empty_like(some)
        lengths = [rows[r][1] for r in which]
        ops.attention_simt(some, pages, table[which], page, i32([sum(lengths[:i]) for i in range(len(which) + 1)]),
                           i32([rows[r][0] for r in which]), out, len(which), max_new, H, G, hd, hd ** -0.5,
                           window or None)
        return out

    together = attend(list(range(len(rows))), 40)
    assert torch.equal(together, attend(list(range(len(rows))), 100))
    for r, (before, new) in enumerate(rows):
        if new == 0:
            continue
        mine = together[first[r]:first[r + 1]]
        assert torch.equal(mine, attend([r], new))
        kv = pages[table[r, :need[r]].long()].double().permute(1, 2, 0, 3, 4).reshape(2, G, -1, hd)[:, :, :before + new]
        k, v = kv.repeat_interleave(H // G, 1)
        s = torch.einsum("nhd,hkd->hnk", q[first[r]:first[r + 1]].double().view(new, H, hd), k) * hd ** -0.5
        qpos, kpos = torch.arange(before, before + new, device=DEV)[:, None], torch.arange(before + new, device=DEV)[None]
        s.masked_fill_((kpos > qpos) | ((kpos <= qpos - window) if window else False), float("-inf"))
        want = torch.einsum("hnk,hkd->nhd", torch.softmax(s, -1), v).reshape(new, -1)
        tol = 2e-6 if dtype == torch.float32 else 2 ** -8       # (as above)
        assert ((mine.double() - want).norm() / want.norm()).item() < tol


@pytest.mark.parametrize("hd", [64, 48])
@pytest.mark.parametrize("window", [0, 9])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_attention_simt_values_of_unseen_keys(hd, window, bad):
    """A value that is no number reaches the queries that see its key, and no other."""
    from scratch_llm_b200.kernels import ops
    n, H, page, at = 70, 2, 16, 41
    gen = torch.Generator().manual_seed(hd)
    pages = torch.randn(-(-n // page), 2, 1, page, hd, generator=gen).to(DEV)
    q = torch.randn(n, H * hd, generator=gen).to(DEV)
    table = torch.arange(len(pages), dtype=torch.int32, device=DEV).view(1, -1)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    outs = []
    for value in (0.5, bad):
        pages[at // page, 1, 0, at % page] = value
        outs.append(torch.empty_like(q))
        ops.attention_simt(q, pages, table, page, i32([0, n]), i32([0]), outs[-1], 1, n, H, 1, hd, hd ** -0.5, window or None)
    sees = torch.arange(n) >= at
    if window:
        sees &= torch.arange(n) < at + window
    assert torch.equal(outs[0][~sees], outs[1][~sees])
    assert not torch.isfinite(outs[1][sees]).any()
