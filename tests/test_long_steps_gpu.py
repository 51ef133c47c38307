"""Kernels for long steps at the edges of their tiles, edges of the nucleus, steps of single tokens in one pass."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _i32(v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("D,V", [(64, 64), (64, 20), (128, 33), (16, 70), (33, 5), (200, 9), (300, 3)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_general_delta_chunks(D, V, dtype):
    """Rows around whole chunks of tokens, in one step and cut in two, against 64 bits."""
    from scratch_llm_b200.kernels import ops
    ops.prepare_jobs([ops.general_delta_library(D)], verbose=False)
    H, lens = 2, [1, 3, 4, 15, 16, 17, 0, 32, 33, 70]
    g = torch.Generator().manual_seed(D + V)
    n, DP = sum(lens), ops.general_delta_padded_dim(D)
    rkv = torch.randn(n, 2 * H * D + H * V, generator=g).to(dtype).to(DEV)
    wa = torch.cat([torch.rand(n, H * D, generator=g) * 0.45 + 0.55, torch.rand(n, H * D, generator=g)], 1).to(DEV)
    first = torch.zeros(len(lens), H, V, DP, device=DEV)
    first[..., :D] = torch.randn(len(lens), H, V, D, generator=g).to(DEV)
    slots = list(reversed(range(len(lens))))

    def step(state, counts, at):
        pick = torch.cat([torch.arange(a, a + c) for a, c in zip(at, counts)]).to(DEV)
        starts = [sum(counts[:i]) for i in range(len(counts) + 1)]
        out = torch.empty(len(pick), H * V, device=DEV)
        ops.general_delta(rkv[pick], (0, H * D, 2 * H * D), wa[pick], state, _i32(starts), _i32(slots), out,
                          len(counts), H, D, V, 1e-6)
        return pick, out

    at = [sum(lens[:i]) for i in range(len(lens))]
    whole, cut, o2 = first.clone(), first.clone(), torch.empty(n, H * V, device=DEV)
    _, o1 = step(whole, lens, at)
    head = [m * 2 // 5 for m in lens]
    for counts, begin in ((head, at), ([m - k for m, k in zip(lens, head)], [a + k for a, k in zip(at, head)])):
        pick, out = step(cut, counts, begin)
        o2[pick] = out

    r, k, v = rkv.double().split([H * D, H * D, H * V], 1)
    r, k, v, (w, a) = r.view(n, H, D), k.view(n, H, D), v.view(n, H, V), wa.double().view(n, 2, H, D).unbind(1)
    u = k / (k.square().sum(-1, keepdim=True) + 1e-6).sqrt()
    want, state = torch.empty(n, H, V, device=DEV, dtype=torch.float64), first.double().clone()
    for i, m in enumerate(lens):
        S = state[slots[i], ..., :D].clone()
        for t in range(at[i], at[i] + m):
            S = S * w[t][:, None] - (S @ u[t][..., None]) * (a[t] * u[t])[:, None] + v[t][..., None] * k[t][:, None]
            want[t] = (S @ r[t][..., None])[..., 0]
        state[slots[i], ..., :D] = S
    # decays of at least 0.55: a few tokens' roundings, each a few of 2^-24
    for got, ref in ((o1, want.flatten(1)), (o2, want.flatten(1)), (whole, state), (cut, state)):
        assert ((got.double() - ref).norm() / ref.norm()).item() < 1e-6


@pytest.mark.parametrize("m,n,k", [(777, 3072, 64), (65, 20480, 20), (640, 1000, 36), (2000, 700, 8), (64, 64 * 300, 12),
                                   (513, 6144, 8), (300, 3072, 24), (256, 3072, 16), (33, 9500, 20)])
def test_32bit_product_widths_of_tiles(m, n, k):
    """Every width of the tiles gives the bits of the plainest kernel (rows that allow no 16-byte requests)."""
    from scratch_llm_b200.kernels import ops
    g = torch.Generator().manual_seed(m + n)
    x, w = torch.randn(m, k, generator=g).to(DEV), torch.randn(n, k, generator=g).to(DEV)
    odd = torch.empty(m, k + 1, device=DEV)[:, :k].copy_(x)
    got = ops.gemm_simt(x, w, torch.full((m, n), float("nan"), device=DEV))
    assert torch.equal(got, ops.gemm_simt(odd, w, torch.empty(m, n, device=DEV)))


@pytest.mark.parametrize("columns,m,n,k", [(64, 513, 6144, 52), (64, 777, 16390, 36), (64, 2050, 5120, 20),
                                            (48, 777, 3070, 52), (48, 129, 4100, 36), (48, 50, 12290, 20),
                                            (32, 129, 6144, 52), (32, 1030, 1020, 36), (32, 33, 16390, 20),
                                            (0, 65, 6144, 52), (0, 33, 3072, 36), (0, 257, 2046, 20)])
def test_32bit_product_over_several_steps(columns, m, n, k):
    """Each width of the wide tiles, and the ring, over more than one step of 16 and a remainder, with rows and columns
    that end inside a tile: the bits of the plainest kernel.  (The rule depends on the SMs: sizes for 148 of them.)"""
    from scratch_llm_b200.kernels import ops
    assert columns == ops._core("sllm_gemm_simt").sllm_gemm_simt_columns(m, n, k, 148)
    g = torch.Generator().manual_seed(m + n)
    x, w = torch.randn(m, k, generator=g).to(DEV), torch.randn(n, k, generator=g).to(DEV)
    odd = torch.empty(m, k + 1, device=DEV)[:, :k].copy_(x)
    got = ops.gemm_simt(x, w, torch.full((m, n), float("nan"), device=DEV))
    assert torch.equal(got, ops.gemm_simt(odd, w, torch.empty(m, n, device=DEV)))


@pytest.mark.parametrize("n,c,r,ld", [(512, 128, 64, 0), (577, 132, 5, 0), (575, 4, 130, 0), (530, 260, 64, 1),
                                       (257, 256, 33, 0), (2113, 900, 64, 1), (2401, 1000, 5, 0), (1900, 1028, 130, 0),
                                       (545, 3076, 64, 0), (300, 4100, 33, 0)])
def test_second_products_of_low_rank_pairs(n, c, r, ld):
    """One chain of multiply-adds over the rank per output: a token's bits are those of a step of few tokens.
    ``ld``: hidden values that allow no reads of 16 bytes.  (Launches of few CTAs keep the kernels of short steps: of the
    sizes up to 577 tokens and 260 channels all but the plain products, at ranks from 64 on; the others take the tiles.)"""
    from scratch_llm_b200.kernels import ops
    g = torch.Generator().manual_seed(n + c + r)
    pre = torch.randn(n, c + r + ld, generator=g).to(DEV)[:, :c + r]
    w2t = (torch.randn(r, c, generator=g) * r ** -0.5).to(DEV)
    w0, ab, rate = (torch.randn(c, generator=g).to(DEV) for _ in range(3))

    def outputs(pre):
        m = len(pre)
        wa, log, gate = (torch.empty(m, w, device=DEV) for w in (2 * c, c, c))
        ops.lowrank_decay(pre, w2t, w0, ab, 0.6, wa)
        ops.lowrank_expand(pre, c, w2t, log, bias=w0, rate_log=rate, per_rate=1, also=(c, w2t, gate))
        half = ops.lowrank_expand(pre, c, w2t, torch.empty(m, c, device=DEV, dtype=torch.bfloat16), tanh_in=True)
        return wa, log, gate, half

    got = outputs(pre)
    for parts in zip(got, *(outputs(pre[t:t + 100]) for t in range(0, n, 100))):
        assert torch.equal(parts[0], torch.cat(parts[1:]))
    x, w = pre.double(), w2t.double()
    z = x[:, c:] @ w
    want = torch.cat([torch.exp(-0.6 * torch.sigmoid(torch.tanh(x[:, c:]) @ w + w0)), torch.sigmoid(x[:, :c] + ab)], 1)
    want = want, -rate.double().exp() * torch.nn.functional.softplus(z + w0), z
    for a, b in zip(got, want):     # 32-bit sums of r products: r / 2 roundings of the largest partial sum at most
        assert ((a.double() - b).norm() / b.norm()).item() < 2 ** -24 * max(8, r / 2)


@pytest.mark.parametrize("V", [8192, 8200, 50001, 190001])
def test_nucleus_of_flat_and_steep_rows(V):
    """The search that starts from a histogram, on rows whose mass lies in one of its buckets, in the last one, or
    on one value: the kept set is the smallest one above top_p that 64 bits give, up to the value at its edge."""
    from scratch_llm_b200.kernels import ops
    g = torch.Generator().manual_seed(V)
    flat, two, steep = torch.zeros(V), torch.zeros(V), torch.arange(V) * -1e-3
    two[::7] = 3.0
    one = torch.full((V,), -60.0)
    one[V // 2] = 0.0
    rows = torch.stack([x for x in (flat, two, steep, one, torch.randn(V, generator=g) * 8) for _ in range(5)])
    tops = torch.tensor([1e-6, 0.37, 0.9, 0.9998, 0.99999] * 5)
    n = len(rows)
    probs, out = torch.empty(n, V, device=DEV), torch.empty(n, dtype=torch.int32, device=DEV)
    seed = torch.arange(n, device=DEV)
    ops.sample(rows.to(DEV), out, torch.ones(n, device=DEV), tops.to(DEV), seed, seed, probs_out=probs)
    kept = probs.cpu() > 0
    assert kept[torch.arange(n), out.cpu().long()].all()
    for r in range(n):
        p = torch.softmax(rows[r].double(), -1)
        k = kept[r]
        # everything above the smallest kept value is kept, and that value is where the mass passes top_p
        edge = p[k].min()
        clear = (p / edge - 1).abs() > 1e-5
        assert (k == (p >= edge))[clear].all()
        slack = 1e-5 + float(edge)               # (32-bit sums; a value on the edge)
        above, upto = float(p[p > edge * (1 + 1e-5)].sum()), float(p[p >= edge * (1 - 1e-5)].sum())
        assert above <= float(tops[r]) + slack and upto >= float(tops[r]) - slack


@pytest.mark.parametrize("V", [8192, 50001])
@pytest.mark.parametrize("more", [0, 1])
def test_nucleus_of_rows_that_one_value_fills(V, more):
    """The largest probability's exponential is not exactly 1 at a temperature (the rounding of its logit over it), so
    it may lie on either side of 1 / Z, and so on either side of an edge of the histogram's buckets.  ``more``: as many
    equal values again, all kept or none but the first."""
    from scratch_llm_b200.kernels import ops
    tops = torch.linspace(8.0, 40.0, 96)
    temps, rows, top_p = (torch.linspace(0.3, 0.8, 96), torch.full((96, V), -200.0),
                          torch.tensor([1e-6, 0.3, 0.9]).repeat(32))
    at = torch.arange(96) * 83 % V
    rows[torch.arange(96), at] = tops
    if more:
        rows[torch.arange(96), (at + V // 2) % V] = tops
    probs, out = torch.empty(96, V, device=DEV), torch.empty(96, dtype=torch.int32, device=DEV)
    seed = torch.arange(96, device=DEV)
    ops.sample(rows.to(DEV), out, temps.to(DEV), top_p.to(DEV), seed, seed, probs_out=probs)
    # (equal values are kept together)
    want = torch.zeros(96, V)
    want[rows == tops[:, None]] = 1.0 / (1 + more)
    assert torch.equal(probs.cpu(), want)
    assert (rows[torch.arange(96), out.cpu().long()] == tops).all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("C,taps", [(1032, 4), (7, 4), (24, 2), (16, 1), (128, 6)])
def test_convolution_and_carried_inputs_in_one_pass(dtype, C, taps):
    """Rows of one token (one of them padding, one row without tokens): the bits of the two passes."""
    from scratch_llm_b200.kernels import ops
    g = torch.Generator().manual_seed(C + taps)
    x = torch.randn(5, C + 8, generator=g).to(dtype).to(DEV)
    w, bias = torch.randn(C, taps, generator=g).to(DEV), torch.randn(C, generator=g).to(DEV)
    state = torch.randn(6, max(taps - 1, 1), C, generator=g).to(dtype).to(DEV)
    token_row, row_start, row_slot = _i32([0, 2, 3, 4, -1]), _i32([0, 1, 1, 2, 3, 4]), _i32([3, 2, 0, 5, 1])
    outs = []
    for update in (False, True):
        st = state.clone()
        out = torch.full((5, C), float("nan"), dtype=dtype, device=DEV)
        ops.conv_silu(x, w, st if taps > 1 else None, token_row, row_start, row_slot, out, w.t().contiguous(),
                      bias, update=update)
        if not update:
            ops.conv_state_update(x, taps, st, row_start, row_slot, 5)
        outs.append((out, st))
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])


@pytest.mark.parametrize("taps", [1, 4])
def test_convolution_step_of_very_many_tokens(taps):
    """More single tokens than a grid's second dimension holds, which the convolution alone has always taken."""
    from scratch_llm_b200.kernels import ops
    n, C, g = 70_000, 8, torch.Generator().manual_seed(taps)
    x, w = torch.randn(n, C, generator=g).to(DEV), torch.randn(C, taps, generator=g).to(DEV)
    state = torch.randn(n, max(taps - 1, 1), C, generator=g).to(DEV)
    rows, starts = torch.arange(n, dtype=torch.int32, device=DEV), torch.arange(n + 1, dtype=torch.int32, device=DEV)
    carried = state if taps > 1 else None
    want = ops.conv_silu(x, w, carried, rows, starts, rows, torch.empty_like(x))
    after = torch.cat([state[:, 1:], x[:, None]], 1)
    assert torch.equal(ops.conv_silu(x, w, carried, rows, starts, rows, torch.empty_like(x), update=True), want)
    assert taps == 1 or torch.equal(state, after)


@pytest.mark.parametrize("hd", [64, 16, 80, 112])
@pytest.mark.parametrize("H,G", [(4, 1), (6, 3), (3, 3)])
@pytest.mark.parametrize("more", [{}, dict(window=37), dict(chunk=48), dict(softcap=5.0), dict(slopes=1, sinks=1)])
def test_attention_simt_tiles(hd, H, G, more):
    """Long 32-bit portions: four, two and one heads of a kv head to a block, each option: a token's bits are those
    it has alone (a kernel of its own)."""
    from scratch_llm_b200.kernels import ops
    ops.prepare_jobs([ops.attention_library(hd)], verbose=False)
    page, before, n = 16, 21, 95
    gen = torch.Generator().manual_seed(hd + H)
    pages = torch.randn(-(-(before + n) // page), 2, G, page, hd, generator=gen).to(DEV)
    q = torch.randn(n, H * hd, generator=gen).to(DEV)
    table = torch.arange(len(pages), dtype=torch.int32, device=DEV).view(1, -1)
    kw = {k: torch.randn(H, generator=gen).to(DEV) if k in ("slopes", "sinks") else v for k, v in more.items()}
    window = kw.pop("window", None)

    def attend(first, count):
        out = torch.empty(count, H * hd, device=DEV)
        ops.attention_simt(q[first:first + count], pages, table, page, _i32([0, count]), _i32([before + first]),
                           out, 1, count, H, G, hd, hd ** -0.5, window, **kw)
        return out

    assert torch.equal(attend(0, n), torch.cat([attend(t, 1) for t in range(n)]))


@pytest.mark.parametrize("hd", [64, 48])
@pytest.mark.parametrize("window", [None, 37])
def test_attention_simt_rows_in_two_launches(hd, window):
    """Rows of all lengths in a launch for long ones (tiles, and the other kernel for rows of up to 16 tokens)."""
    from scratch_llm_b200.kernels import ops
    ops.prepare_jobs([ops.attention_library(hd)], verbose=False)
    H, G, page = 8, 2, 16
    rows = [(70, 1), (0, 40), (5, 4), (31, 16), (0, 0), (64, 17), (90, 5), (3, 33)]      # (cached, new)
    gen = torch.Generator().manual_seed(hd)
    need = [-(-(b + n) // page) for b, n in rows]
    pages = torch.randn(sum(need), 2, G, page, hd, generator=gen).to(DEV)
    first = [sum(x for _, x in rows[:r]) for r in range(len(rows) + 1)]
    q = torch.randn(first[-1], H * hd, generator=gen).to(DEV)
    table = torch.full((len(rows), max(need)), -1, dtype=torch.int32)
    for r, k in enumerate(need):
        table[r, :k] = torch.arange(sum(need[:r]), sum(need[:r]) + k)
    outs = []
    for most in (40, 600):
        outs.append(torch.full_like(q, float("nan")))
        ops.attention_simt(q, pages, table.to(DEV), page, _i32(first), _i32([b for b, _ in rows]), outs[-1], len(rows),
                           most, H, G, hd, hd ** -0.5, window)
    assert torch.equal(outs[0], outs[1])


@pytest.mark.parametrize("D", [64, 128, 16, 33, 200])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("size", [5e2, 1e10, 1e17, 1e25])
def test_general_delta_large_keys(D, dtype, size):
    """Keys whose products with each other or with the state leave the range of 32 bits, though neither the state
    nor the read-outs do, beside ordinary ones, a small one and one of zeros."""
    from scratch_llm_b200.kernels import ops
    ops.prepare_jobs([ops.general_delta_library(D)], verbose=False)
    H, V, lens = 2, 8, [1, 5, 40]
    g = torch.Generator().manual_seed(D)
    n, DP = sum(lens), ops.general_delta_padded_dim(D)
    k = torch.randn(n, H * D, generator=g) * size
    k[::3] /= size
    k[20], k[31] = 1e-3, 0.0
    r, v = torch.randn(n, H * D, generator=g), torch.randn(n, H * V, generator=g) * 1e8
    rkv = torch.cat([r, k, v], 1).to(dtype).to(DEV)
    wa = torch.cat([torch.rand(n, H * D, generator=g) * 0.45 + 0.55, torch.rand(n, H * D, generator=g)], 1).to(DEV)
    state, out = torch.zeros(3, H, V, DP, device=DEV), torch.empty(n, H * V, device=DEV)
    starts = [sum(lens[:i]) for i in range(len(lens) + 1)]
    ops.general_delta(rkv, (0, H * D, 2 * H * D), wa, state, _i32(starts), _i32([0, 1, 2]), out, 3, H, D, V, 1e-6)
    r, k, v = rkv.double().split([H * D, H * D, H * V], 1)
    r, k, v, (w, a) = r.view(n, H, D), k.view(n, H, D), v.view(n, H, V), wa.double().view(n, 2, H, D).unbind(1)
    u = k / (k.square().sum(-1, keepdim=True) + 1e-6).sqrt()
    want = torch.empty(n, H, V, device=DEV, dtype=torch.float64)
    for i in range(len(lens)):
        S = torch.zeros(H, V, D, dtype=torch.float64, device=DEV)
        for t in range(starts[i], starts[i + 1]):
            S = S * w[t][:, None] - (S @ u[t][..., None]) * (a[t] * u[t])[:, None] + v[t][..., None] * k[t][:, None]
            want[t] = (S @ r[t][..., None])[..., 0]
        # (a few tokens' roundings, each a few of 2^-24)
        assert ((state[i, ..., :D].double() - S).norm() / S.norm()).item() < 1e-6
    assert ((out.double() - want.flatten(1)).norm() / want.norm()).item() < 1e-6


@pytest.mark.parametrize("D,V", [(64, 64), (64, 20), (64, 12), (128, 33), (16, 16), (16, 70), (9, 9), (24, 30), (33, 5),
                                 (200, 9), (300, 3)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_general_delta_in_large_launches(D, V, dtype):
    """More CTAs than the SMs hold (four columns a thread, one compute warp where heads have few columns): against 64
    bits, and the bits of a row with three of the heads in a launch of its own (two columns a thread)."""
    from scratch_llm_b200.kernels import ops
    ops.prepare_jobs([ops.general_delta_library(D)], verbose=False)
    lens = [1, 3, 4, 15, 16, 17, 0, 32, 33, 70]
    H = 2 * torch.cuda.get_device_properties(0).multi_processor_count // len(lens) + 1
    g = torch.Generator().manual_seed(D + V)
    n, DP, few = sum(lens), ops.general_delta_padded_dim(D), 3
    rkv = torch.randn(n, 2 * H * D + H * V, generator=g).to(dtype).to(DEV)
    wa = torch.cat([torch.rand(n, H * D, generator=g) * 0.45 + 0.55, torch.rand(n, H * D, generator=g)], 1).to(DEV)
    first = torch.zeros(len(lens), H, V, DP, device=DEV)
    first[..., :D] = torch.randn(len(lens), H, V, D, generator=g).to(DEV)
    cols, starts = (0, H * D, 2 * H * D), [sum(lens[:i]) for i in range(len(lens) + 1)]
    state, out = first.clone(), torch.empty(n, H * V, device=DEV)
    ops.general_delta(rkv, cols, wa, state, _i32(starts), _i32(list(range(len(lens)))), out, len(lens), H, D, V, 1e-6)

    r, k, v = rkv.double().split([H * D, H * D, H * V], 1)
    r, k, v, (w, a) = r.view(n, H, D), k.view(n, H, D), v.view(n, H, V), wa.double().view(n, 2, H, D).unbind(1)
    u = k / (k.square().sum(-1, keepdim=True) + 1e-6).sqrt()
    want, S_all = torch.empty(n, H, V, device=DEV, dtype=torch.float64), first.double().clone()
    for i, m in enumerate(lens):
        at, S = slice(starts[i], starts[i] + m), first[i, ..., :D].double()
        for t in range(starts[i], starts[i] + m):
            S = S * w[t][:, None] - (S @ u[t][..., None]) * (a[t] * u[t])[:, None] + v[t][..., None] * k[t][:, None]
            want[t] = (S @ r[t][..., None])[..., 0]
        S_all[i, ..., :D] = S
        alone, o = first[i:i + 1, :few].contiguous(), torch.empty(m, few * V, device=DEV)
        part = wa[at].view(m, 2, H, D)[:, :, :few].flatten(1).contiguous()
        ops.general_delta(rkv[at].clone(), cols, part, alone, _i32([0, m]), _i32([0]), o, 1, few, D, V, 1e-6)
        assert torch.equal(o, out[at, :few * V]) and torch.equal(alone[0], state[i, :few])
    # decays of at least 0.55: a few tokens' roundings, each a few of 2^-24
    for got, ref in ((out, want.flatten(1)), (state, S_all)):
        assert ((got.double() - ref).norm() / ref.norm()).item() < 1e-6


@pytest.mark.parametrize("hd", [64, 80, 112, 128])
@pytest.mark.parametrize("n", [32, 33, 48, 49, 64, 65])
def test_attention_simt_around_the_tiles_limits(hd, n):
    """A row's portion with a block table of few keys and of many (which kernel takes it depends on that): the same
    bits, those of single tokens."""
    from scratch_llm_b200.kernels import ops
    ops.prepare_jobs([ops.attention_library(hd)], verbose=False)
    H, G, page, before = 6, 3, 16, 5
    gen = torch.Generator().manual_seed(hd + n)
    need = -(-(before + n) // page)
    pages, q = torch.randn(need, 2, G, page, hd, generator=gen).to(DEV), torch.randn(n, H * hd, generator=gen).to(DEV)
    wide = torch.full((1, 40), -1, dtype=torch.int32)
    wide[0, :need] = torch.arange(need)

    def attend(table, first, count):
        out = torch.full((count, H * hd), float("nan"), device=DEV)
        return ops.attention_simt(q[first:first + count], pages, table.to(DEV), page, _i32([0, count]),
                                  _i32([before + first]), out, 1, count, H, G, hd, hd ** -0.5, None)

    single = torch.cat([attend(wide, t, 1) for t in range(n)])
    assert torch.equal(attend(wide, 0, n), single)
    assert torch.equal(attend(wide[:, :need].contiguous(), 0, n), single)


@pytest.mark.parametrize("short", [17, 90])
def test_attention_simt_many_rows_of_own_heads(short):
    """A long row beside many, each head with a kv head of its own: by the tokens a row on average one launch or two,
    the same bits."""
    from scratch_llm_b200.kernels import ops
    ops.prepare_jobs([ops.attention_library(64)], verbose=False)
    H, page, hd, rows = 2, 16, 64, [520] + [short] * 30 + [0, 1]
    gen = torch.Generator().manual_seed(short)
    need = [-(-n // page) for n in rows]
    pages = torch.randn(sum(need), 2, H, page, hd, generator=gen).to(DEV)
    first = [sum(rows[:r]) for r in range(len(rows) + 1)]
    q = torch.randn(first[-1], H * hd, generator=gen).to(DEV)
    table = torch.full((len(rows), max(need)), -1, dtype=torch.int32)
    for r, k in enumerate(need):
        table[r, :k] = torch.arange(sum(need[:r]), sum(need[:r]) + k)
    table = table.to(DEV)
    out = torch.full_like(q, float("nan"))
    ops.attention_simt(q, pages, table, page, _i32(first), _i32([0] * len(rows)), out, len(rows), 520, H, H, hd, 0.125, None)
    for r, n in enumerate(rows):
        if n:
            at = slice(first[r], first[r + 1])
            alone = torch.empty(n, H * hd, device=DEV)
            ops.attention_simt(q[at], pages, table[r:r + 1], page, _i32([0, n]), _i32([0]), alone, 1, n, H, H, hd, 0.125,
                               None)
            assert torch.equal(alone, out[at])
