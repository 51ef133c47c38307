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
