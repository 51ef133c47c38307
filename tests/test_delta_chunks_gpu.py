"""The delta rule's chunk kernels (long portions) against the rule written out in 64 bits, token by
token, and beside the kernel that walks the tokens in order."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def ops():
    from scratch_llm_b200.kernels import ops as o
    return o


def rand(*shape, seed=0, scale=1.0):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)) * scale


def unit(x):
    return x / torch.sqrt(x.square().sum(-1, keepdim=True) + 1e-6)


def i32(v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


def close(got, want, what):
    # 32-bit sums of up to 64 + D products, and as many roundings from chunk to chunk: a few hundred
    # roundings of 2^-24 that add up like a walk, and a triangular system of unit keys that may grow
    # them a little: 2^-24 * sqrt(512) * 8 = 1.1e-5
    err = ((got.double().cpu() - want).norm() / want.norm()).item()
    assert err < 2e-5, f"{what}: {err}"


# edges of chunks and blocks, rows below the limit beside rows above it, rows without tokens
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("channels", [False, True])
@pytest.mark.parametrize("D,V,H,G,odd", [(128, 128, 2, 1, 0), (64, 72, 3, 3, 0), (32, 37, 2, 2, 1)])
@pytest.mark.parametrize("lengths", [[128], [129, 3, 0, 191, 1], [193, 127, 64], [255, 256]])
def test_delta_rule_in_chunks(dtype, channels, D, V, H, G, odd, lengths):
    n, rows = sum(lengths), len(lengths)
    # (an odd row stride: no reads of several elements)
    act = rand(n, 2 * G * D + H * V + odd, seed=1).to(dtype).to(DEV)
    ab = rand(n, 2 * H, seed=2).to(DEV)
    A_log, dt_bias = rand(H, seed=3), rand(H, seed=4)
    # decays from nearly none to ones that leave nothing
    log_decay = -torch.exp(rand(n, H * D, seed=5, scale=2.0) - 2.0)
    log_decay[:, ::7] = -torch.exp(rand(n, log_decay[:, ::7].shape[1], seed=6) + 3.0)
    start = rand(rows + 1, H, V, D, seed=7)
    slots = list(range(rows, 0, -1))
    q, k, v = act.double().cpu()[:, :2 * G * D + H * V].split([G * D, G * D, H * V], 1)
    q = unit(q.view(n, G, D)).repeat_interleave(H // G, 1) * D ** -0.5
    k = unit(k.view(n, G, D)).repeat_interleave(H // G, 1)
    v = v.view(n, H, V)
    x = ab.double().cpu()
    beta = torch.sigmoid(x[:, H:])
    g = torch.exp(log_decay.double()).view(n, H, D) if channels else torch.exp(
        -torch.exp(A_log.double()) * torch.nn.functional.softplus(x[:, :H] + dt_bias.double()))[..., None]
    want, want_S, t = [], [], 0
    for r, length in enumerate(lengths):
        S = start[slots[r]].double()
        for _ in range(length):
            S = S * g[t][:, None]
            u = beta[t][:, None] * (v[t] - (S @ k[t][..., None])[..., 0])
            S = S + u[..., None] * k[t][:, None]
            want.append((S @ q[t][..., None])[..., 0])
            t += 1
        want_S.append(S)
    want, want_S = torch.stack(want), torch.stack(want_S)
    row_start = i32([sum(lengths[:i]) for i in range(rows + 1)])
    for min_chunked in (None, 0):
        S = start.to(DEV).clone()
        out = torch.full((n, H * V), float("nan"), device=DEV)
        ops().delta_rule(act, ab, None if channels else A_log.to(DEV), None if channels else dt_bias.to(DEV), S,
                         row_start, i32(slots), out, rows, H, G, D, V, longest=max(lengths), shortest=min(lengths),
                         log_decay=log_decay.to(DEV) if channels else None, min_chunked=min_chunked)
        close(out.view(n, H, V), want, f"out, min_chunked {min_chunked}")
        close(S[slots], want_S, f"state, min_chunked {min_chunked}")
        assert torch.equal(S[0].cpu(), start[0])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("channels", [False, True])
@pytest.mark.parametrize("decay", [-6.0, -1.0])
@pytest.mark.parametrize("D,V", [(128, 128), (64, 64), (32, 37)])
def test_chunks_are_as_exact_as_the_order_of_tokens(dtype, channels, decay, D, V):
    """The chunk kernels' error against 64 bits beside that of the kernel that takes the tokens in order, with
    decays that keep hundreds of tokens and with ones that keep a few."""
    n, H, G = 600, 4, 2
    g = torch.Generator(device=DEV).manual_seed(D + int(decay))
    r = lambda *s: torch.randn(*s, device=DEV, generator=g)  # noqa: E731
    act, ab, start = r(n, 2 * G * D + H * V).to(dtype), r(n, 2 * H), r(1, H, V, D)
    A_log, dt_bias, log_decay = r(H) + min(decay, -1) + 1, r(H), -torch.exp(r(n, H * D) + decay)
    q, k, v = act.double().split([G * D, G * D, H * V], 1)
    q = unit(q.view(n, G, D)).repeat_interleave(H // G, 1) * D ** -0.5
    k = unit(k.view(n, G, D)).repeat_interleave(H // G, 1)
    x, v, S, want = ab.double(), v.view(n, H, V), start[0].double(), []
    fade = torch.exp(log_decay.double()).view(n, H, D) if channels else torch.exp(
        -torch.exp(A_log.double()) * torch.nn.functional.softplus(x[:, :H] + dt_bias.double()))[..., None]
    for t in range(n):
        S = S * fade[t][:, None]
        u = torch.sigmoid(x[t, H:])[:, None] * (v[t] - (S @ k[t][..., None])[..., 0])
        S = S + u[..., None] * k[t][:, None]
        want.append((S @ q[t][..., None])[..., 0])
    want, errors = torch.stack(want), []
    for min_chunked in (None, 0):
        state, out = start.clone(), torch.empty(n, H * V, device=DEV)
        ops().delta_rule(act, ab, None if channels else A_log, None if channels else dt_bias, state, i32([0, n]),
                         i32([0]), out, 1, H, G, D, V, longest=n, shortest=n, min_chunked=min_chunked,
                         log_decay=log_decay if channels else None)
        errors.append([((a.double() - b).norm() / b.norm()).item() for a, b in ((out.view(n, H, V), want), (state[0], S))])
    # both are walks of as many roundings in another order: 0.6 to 1.35 measured (4 with sums cut off by mma.sync)
    for what, chunked, in_order in zip(("read-outs", "state"), *errors):
        assert chunked < 1.5 * in_order, f"{what}: {chunked:.2e}, in order {in_order:.2e}"


def rows_case(lengths, H, G, D, V, channels, dtype=torch.bfloat16):
    """A function that runs the given rows of a step (all of them, or some alone); their outputs and states."""
    n, g = sum(lengths), torch.Generator(device=DEV).manual_seed(sum(lengths))
    r = lambda *s: torch.randn(*s, device=DEV, generator=g)  # noqa: E731
    act, ab, start = r(n, 2 * G * D + H * V).to(dtype), r(n, 2 * H), r(len(lengths), H, V, D)
    A_log, dt_bias, log_decay = r(H), r(H), -torch.exp(r(n, H * D) - 2)
    first = [sum(lengths[:i]) for i in range(len(lengths))]

    def run(rows, **more):
        tokens = torch.cat([torch.arange(first[i], first[i] + lengths[i], device=DEV) for i in rows])
        some = [lengths[i] for i in rows]
        S, out = start.clone(), torch.full((sum(some), H * V), float("nan"), device=DEV)
        ops().delta_rule(act[tokens], ab[tokens], None if channels else A_log, None if channels else dt_bias, S,
                         i32([sum(some[:i]) for i in range(len(some) + 1)]), i32(rows), out, len(some), H, G, D, V,
                         max_new=1 if max(some) == 1 else 0, longest=max(some), shortest=min(some),
                         log_decay=log_decay[tokens] if channels else None, **more)
        return list(out.split(some)), S

    return run


@pytest.mark.parametrize("channels", [False, True])
@pytest.mark.parametrize("D,V", [(128, 40), (64, 64)])
@pytest.mark.parametrize("chunks", [1, 3, 7])
def test_groups_of_chunks_and_rows_alone(monkeypatch, channels, D, V, chunks):
    """However many chunks the scratch holds, and whatever rows are beside a row: the same bits."""
    lengths = [129, 3, 0, 500, 1, 193, 64] + [0] * 28 + [128, 1, 300]
    run = rows_case(lengths, 2, 1, D, V, channels)
    rows = list(range(len(lengths)))
    out, S = run(rows)
    floats = (3 * 64 * D + 64 * V + 64 * 64 + V * D + D) * 2
    monkeypatch.setattr(ops(), "DELTA_SCRATCH_BYTES", 4 * floats * chunks)
    again, S_again = run(rows)
    assert torch.equal(torch.cat(out), torch.cat(again)) and torch.equal(S, S_again)
    for i in (0, 1, 3, 4, 5, 36, 37):
        alone, S_alone = run([i])
        assert torch.equal(out[i], alone[0]) and torch.equal(S[i], S_alone[i]), lengths[i]


@pytest.mark.parametrize("lengths,limit", [([130] + [1] * 64, 4), ([200] * 8, 33), ([8192], 78)])
def test_scratch_goes_with_the_chunks(lengths, limit):
    """What a step takes beside its tensors: no more than its chunks (32 heads of 128 x 128), nor than the
    limit that chunks are grouped to."""
    run = rows_case(lengths, 32, 16, 128, 128, False)
    seen, empty = [], torch.empty

    def counting(*a, **k):
        t = empty(*a, **k)
        seen.append(t.numel() * t.element_size())
        return t

    rows = list(range(len(lengths)))
    run(rows)
    with pytest.MonkeyPatch.context() as m:
        m.setattr(torch, "empty", counting)
        run(rows)
    chunk = 32 * 4 * (3 * 64 * 128 + 64 * 128 + 64 * 64 + 128 * 128 + 128)
    assert sum(seen) <= limit * chunk and sum(seen) <= 512 << 20


@pytest.mark.parametrize("channels", [False, True])
def test_captured_step_with_other_rows(channels):
    """A captured step replayed with other rows of the same padded sizes: long rows, none, tokens of padding."""
    D, V, H, G, n, rows = 64, 48, 2, 1, 320, 5
    g = torch.Generator(device=DEV).manual_seed(5)
    r = lambda *s: torch.randn(*s, device=DEV, generator=g)  # noqa: E731
    act, ab, start = r(n, 2 * G * D + H * V).bfloat16(), r(n, 2 * H), r(rows, H, V, D)
    A_log, dt_bias, log_decay = r(H), r(H), -torch.exp(r(n, H * D) - 2)
    S, out, slots = start.clone(), torch.zeros(n, H * V, device=DEV), i32([4, 3, 2, 1, 0])
    row_start = torch.zeros(rows + 1, dtype=torch.int32, device=DEV)

    def step():
        ops().delta_rule(act, ab, None if channels else A_log, None if channels else dt_bias, S, row_start, slots, out,
                         rows, H, G, D, V, longest=n, log_decay=log_decay if channels else None)

    def set_rows(lengths):
        row_start.copy_(i32([sum(lengths[:i]) for i in range(rows + 1)]))
        S.copy_(start)
        out.zero_()

    set_rows([320, 0, 0, 0, 0])
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        step()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        step()
    for lengths in ([320, 0, 0, 0, 0], [1, 150, 7, 128, 1], [60, 70, 80, 1, 1], [127, 0, 1, 192, 0], [2, 1, 1, 1, 1]):
        set_rows(lengths)
        graph.replay()
        got = out.clone(), S.clone()
        set_rows(lengths)
        step()
        assert torch.equal(got[0], out) and torch.equal(got[1], S), lengths


@pytest.mark.parametrize("channels", [False, True])
@pytest.mark.parametrize("cut", [[128, 272], [127, 273], [1, 130, 5, 128, 1, 135], [64, 200, 127, 9]])
def test_portions_above_and_below_the_limit(channels, cut):
    """One row's tokens in one step, and cut into steps that continue from its state."""
    D, V, H, G, n = 128, 40, 2, 1, 400
    g = torch.Generator(device=DEV).manual_seed(6)
    r = lambda *s: torch.randn(*s, device=DEV, generator=g)  # noqa: E731
    act, ab, start = r(n, 2 * G * D + H * V), r(n, 2 * H), r(1, H, V, D)
    A_log, dt_bias, log_decay = r(H), r(H), -torch.exp(r(n, H * D) - 3)
    results = []
    for lengths in ([n], cut):
        S, outs, t = start.clone(), [], 0
        for m in lengths:
            outs.append(torch.empty(m, H * V, device=DEV))
            ops().delta_rule(act[t:t + m], ab[t:t + m], None if channels else A_log, None if channels else dt_bias, S,
                             i32([0, m]), i32([0]), outs[-1], 1, H, G, D, V, max_new=1 if m == 1 else 0, longest=m,
                             shortest=m, log_decay=log_decay[t:t + m] if channels else None)
            t += m
        results.append((torch.cat(outs), S))
    for what, a, b in zip(("out", "state"), *results):
        close(b, a.double().cpu(), f"{what} of the portions")


@pytest.mark.parametrize("channels", [False, True])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_a_row_that_is_no_number(channels, bad):
    """A row with an infinity or a NaN in its tokens or its state leaves the rows beside it alone, and its own
    tokens before the bad one's block of 16."""
    lengths = [130, 200, 20, 1, 300]
    H, G, D, V = 2, 1, 64, 48
    n, rows = sum(lengths), len(lengths)
    g = torch.Generator(device=DEV).manual_seed(7)
    r = lambda *s: torch.randn(*s, device=DEV, generator=g)  # noqa: E731
    act, ab, start = r(n, 2 * G * D + H * V), r(n, 2 * H), r(rows, H, V, D)
    A_log, dt_bias, log_decay = r(H), r(H), -torch.exp(r(n, H * D) - 2)
    results = []
    for spoil in (False, True):
        x, S, out = act.clone(), start.clone(), torch.empty(n, H * V, device=DEV)
        if spoil:
            x[130 + 100, G * D + 3] = bad          # a key of row 1, its token 100
            x[350, :] = bad                        # the single row's token and state
            S[3, 0, 0, 0] = bad
        ops().delta_rule(x, ab, None if channels else A_log, None if channels else dt_bias, S,
                         i32([sum(lengths[:i]) for i in range(rows + 1)]), i32(list(range(rows))), out, rows, H, G, D, V,
                         longest=max(lengths), log_decay=log_decay if channels else None)
        results.append((out, S))
    clean = torch.ones(n, dtype=torch.bool)
    clean[130 + 96:330] = False
    clean[350] = False
    assert torch.equal(results[0][0][clean], results[1][0][clean])
    for row in (0, 2, 4):
        assert torch.equal(results[0][1][row], results[1][1][row])
    assert results[1][0][130 + 101:330].isnan().any(1).all()
