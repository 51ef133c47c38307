"""The delta rule's decode steps (every row one token) against the rule in 64 bits."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("channels", [False, True])
# columns that do not fill a warp's or a CTA's share; key sizes with one and two quads a lane, and odd ones
@pytest.mark.parametrize("D,V,H,G", [(128, 128, 4, 2), (128, 33, 2, 2), (64, 7, 3, 1), (9, 40, 2, 1), (160, 37, 2, 2)])
def test_delta_step(dtype, channels, D, V, H, G):
    from scratch_llm_b200.kernels import ops
    rows = 3
    gen = torch.Generator().manual_seed(D + V)
    r = lambda *s: torch.randn(*s, generator=gen)  # noqa: E731
    act, ab = r(rows, 2 * G * D + H * V).to(dtype).to(DEV), r(rows, 2 * H).to(DEV)
    A_log, dt_bias, start = r(H), r(H), r(rows + 1, H, V, D)
    log_decay = -torch.exp(r(rows, H * D))
    lengths, slots = [1, 0, 1, 1], [2, 0, 3, 1]        # (a row without a token leaves its slot alone)
    q, k, v = act.double().cpu().split([G * D, G * D, H * V], 1)
    unit = lambda x: x / torch.sqrt(x.square().sum(-1, keepdim=True) + 1e-6)  # noqa: E731
    q = unit(q.view(rows, G, D)).repeat_interleave(H // G, 1) * D ** -0.5
    k = unit(k.view(rows, G, D)).repeat_interleave(H // G, 1)
    x = ab.double().cpu()
    g = torch.exp(log_decay.double()).view(rows, H, D) if channels else torch.exp(
        -torch.exp(A_log.double()) * torch.nn.functional.softplus(x[:, :H] + dt_bias.double()))[..., None]
    S0 = start[[2, 3, 1]].double() * g[:, :, None]
    u = torch.sigmoid(x[:, H:])[..., None] * (v.view(rows, H, V) - (S0 @ k[..., None])[..., 0])
    want_S = S0 + u[..., None] * k[:, :, None]
    want = (want_S @ q[..., None])[..., 0]
    S, out = start.to(DEV).clone(), torch.full((rows, H * V), float("nan"), device=DEV)
    i32 = lambda t: torch.tensor(t, dtype=torch.int32, device=DEV)  # noqa: E731
    ops.delta_rule(act, ab, None if channels else A_log.to(DEV), None if channels else dt_bias.to(DEV), S,
                   i32([0, 1, 1, 2, 3]), i32(slots), out, len(lengths), H, G, D, V, max_new=1, longest=1,
                   log_decay=log_decay.to(DEV) if channels else None)
    # sums of D products in 32-bit: 2^-24 * sqrt(160) * 4 = 3e-6
    assert ((out.double().cpu().view(rows, H, V) - want).norm() / want.norm()).item() < 3e-6
    assert ((S[[2, 3, 1]].double().cpu() - want_S).norm() / want_S.norm()).item() < 3e-6
    assert torch.equal(S[0].cpu(), start[0])


@pytest.mark.parametrize("D,V", [(128, 33), (160, 37), (64, 7)])
@pytest.mark.parametrize("lengths", [[1, 1], [1, 5, 1], [1, 130, 20]])
def test_delta_state_on_any_boundary(D, V, lengths):
    """A state that starts on no 16-byte boundary goes element by element: the same bits in steps of single
    tokens, and in mixed ones where no row is long enough for chunks (which need the boundary)."""
    from scratch_llm_b200.kernels import ops
    H, n, rows = 2, sum(lengths), len(lengths)
    gen = torch.Generator(device=DEV).manual_seed(D)
    r = lambda *s: torch.randn(*s, device=DEV, generator=gen)  # noqa: E731
    act, ab, A_log, dt_bias, start = r(n, 4 * D + H * V), r(n, 2 * H), r(H), r(H), r(rows, H, V, D)
    i32 = lambda t: torch.tensor(t, dtype=torch.int32, device=DEV)  # noqa: E731
    row_start, slots = i32([sum(lengths[:i]) for i in range(rows + 1)]), i32(list(range(rows)))
    got = []
    for shift in (0, 1):
        S = torch.empty(start.numel() + 4, device=DEV)[shift:shift + start.numel()].view(start.shape).copy_(start)
        assert S.data_ptr() % 16 == 4 * shift
        out = torch.empty(n, H * V, device=DEV)
        ops.delta_rule(act, ab, A_log, dt_bias, S, row_start, slots, out, rows, H, 2, D, V,
                       max_new=1 if max(lengths) == 1 else 0, longest=max(lengths),
                       min_chunked=0 if shift == 0 else None)
        got.append((out, S.clone()))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
