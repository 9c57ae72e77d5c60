"""Decayed linear attention and the state-space recurrence over prompts in chunks of 128 tokens: lengths at the edges of chunks, sequences
that go on from a state, head sizes that fill tiles and that do not, against 64-bit arithmetic token by token."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(autouse=True, params=["chosen", "larger"])
def chunks(request, monkeypatch):
    """The form that a step's sizes choose, or the chunks of 128 whatever the sizes (their scratch chooses them)."""
    from pace_b200 import _C
    if request.param == "larger":
        for name in ("pace_lightning_scratch_bytes", "pace_ssd_scratch_bytes"):
            monkeypatch.setattr(_C.lib, name, lambda *a, f=getattr(_C.lib, name): max(f(*a), (512 << 20) + 256))
    return request.param
LENS = [[129], [1, 128, 2, 257], [300, 127, 640], [130] * 40]


def _step(lens, starts):
    from pace_b200.llm.step import Step
    return Step(lens, starts, range(len(lens)), torch.zeros(sum(lens), dtype=torch.long), 1, DEV)


def _scan(step, lens, q, k, v, decay, S):
    """q, k [T, H, D], v [T, H, P], decay [T, H], S [B, H, D, P], all fp64; rows in the step's order."""
    at, out, S = 0, torch.empty_like(v), S.clone()
    for row in step.rows:
        for t in range(at, at + lens[row]):
            S[row] = S[row] * decay[t][:, None, None] + k[t][:, :, None] * v[t][:, None]
            out[t] = (S[row] * q[t][:, :, None]).sum(1)
        at += lens[row]
    return out, S


def _close(got, want, tol):
    assert (got.double() - want).norm() <= tol * want.norm()


@pytest.mark.parametrize("lens", LENS)
@pytest.mark.parametrize("H,D,P", [(2, 128, 128), (1, 72, 40), (3, 128, 72), (1, 104, 136)])
def test_lightning(lens, H, D, P):
    from pace_b200.ops import hybrid
    g = torch.Generator(device=DEV).manual_seed(D + P)
    B, T = len(lens), sum(lens)
    starts = [5 if b % 2 else 0 for b in range(B)]
    x = torch.randn(T, H * (2 * D + P), device=DEV, generator=g).bfloat16()
    decay = torch.tensor([1.0, 0.9, 0.999][:H], device=DEV)
    S = torch.randn(B, H, D, P, device=DEV, generator=g)
    q, k, v = (torch.nn.functional.silu(t.double()).bfloat16().double().unflatten(1, (H, -1)) for t in x.split([H * D, H * D, H * P], 1))
    step = _step(lens, starts)
    old = S.double() * torch.tensor([float(s > 0) for s in starts], device=DEV, dtype=torch.float64)[:, None, None, None]
    want, state = _scan(step, lens, q, k, v, decay.double().expand(T, H), old)
    got = hybrid.lightning(step, x, decay, S)
    # outputs: rounded to bf16 (2^-9 at most, and the products of two bf16 terms leave 2^-16); states: 32-bit sums of three-term products, and
    # silu in 32 bits that rounds to the other bf16 now and then
    _close(got, want.flatten(1), 2.0 ** -8)
    _close(S, state, 1e-4)


@pytest.mark.parametrize("lens", LENS)
@pytest.mark.parametrize("H,G,D,P", [(4, 2, 128, 64), (2, 1, 80, 24), (2, 2, 128, 128), (1, 1, 96, 136)])
def test_ssd(lens, H, G, D, P):
    import pace_b200.torch_ops  # noqa: F401
    g = torch.Generator(device=DEV).manual_seed(D + P)
    r = lambda *s: torch.randn(*s, device=DEV, generator=g)      # noqa: E731
    B, T = len(lens), sum(lens)
    starts = [5 if b % 2 else 0 for b in range(B)]
    x, dt_raw = r(T, H * P + 2 * G * D).bfloat16(), r(T, H).bfloat16()
    bias, neg_a, skip, S = r(H) - 3, -r(H).abs() - 0.1, r(H), r(B, H, D, P)
    v, k, q = (t.double().unflatten(1, (-1, n)) for t, n in zip(x.split([H * P, G * D, G * D], 1), (P, D, D)))
    k, q = (t.repeat_interleave(H // G, 1) for t in (k, q))
    dt = torch.nn.functional.softplus(dt_raw.double() + bias.double())
    step = _step(lens, starts)
    old = S.double() * torch.tensor([float(s > 0) for s in starts], device=DEV, dtype=torch.float64)[:, None, None, None]
    want, state = _scan(step, lens, q, k * dt[..., None], v, torch.exp(neg_a.double() * dt), old)
    want = (want + skip.double()[:, None] * v).flatten(1)
    out = torch.empty(T, H * P, device=DEV, dtype=torch.bfloat16)
    torch.ops.pace_b200.ssd_prefill(step.handle, x, dt_raw, bias, neg_a, skip, S, out, G)
    _close(out, want, 2.0 ** -8)
    _close(S, state, 2e-5)        # exponentials of sums of up to 128 log decays: some ulp of 32 bits each


def _lightning_case(lens, H, D, P, seed=3):
    g = torch.Generator(device=DEV).manual_seed(seed)
    x = torch.randn(sum(lens), H * (2 * D + P), device=DEV, generator=g).bfloat16()
    starts = [9 if b % 2 else 0 for b in range(len(lens))]
    S = torch.randn(len(lens), H, D, P, device=DEV, generator=g)
    return x, torch.full((H,), 0.99, device=DEV), S, starts


@pytest.mark.parametrize("lens", [[4000, 1, 129, 3000], [130] * 60 + [700, 5000]])
def test_rounds_of_launches(lens, chunks):
    """Steps whose scratch is more than one round of launches may hold: the same as every sequence by itself."""
    from pace_b200 import _C
    from pace_b200.ops import hybrid
    H, D, P = 64, 128, 128
    x, decay, S, starts = _lightning_case(lens, H, D, P)
    step = _step(lens, starts)
    places = sum(lens) // 128 + len(lens)
    if chunks == "chosen":
        pytest.skip("every sequence by itself may take the other form")
    got_bytes = _C.lib.pace_lightning_scratch_bytes(step.struct, H, D, P, _C.DTYPE_BF16)
    assert got_bytes < places * H * 192 * 1024          # more than one round
    states = S.clone()
    got, at = hybrid.lightning(step, x, decay, states), 0
    for row in step.rows:
        n, one = lens[row], S[row: row + 1].clone()
        want = hybrid.lightning(_step([n], [starts[row]]), x[at: at + n], decay, one)
        # a chunk's products and sums are the same in either; sequences that fit the older chunks alone differ in rounding
        tol = 0 if n > 128 else 2.0 ** -8
        assert (got[at: at + n].double() - want.double()).norm() <= tol * want.double().norm()
        assert (states[row].double() - one[0].double()).norm() <= (0 if n > 128 else 1e-4) * one.double().norm()
        at += n


@pytest.mark.parametrize("room", [0, 1])
def test_less_room_takes_the_smaller_chunks(room, chunks, monkeypatch):
    """Where the scratch of the chunks of 128 cannot be had, those of 64 run in theirs."""
    from pace_b200 import _C
    from pace_b200.ops import hybrid
    lens, H, D, P = [4096], 16, 128, 128
    x, decay, S, starts = _lightning_case(lens, H, D, P)
    step = _step(lens, starts)
    a, b = S.clone(), S.clone()
    want = hybrid.lightning(step, x, decay, a)
    out = torch.empty_like(want)
    need = _C.lib.pace_lightning_scratch_bytes(step.struct, H, D, P, _C.DTYPE_BF16)
    fewer = _C.lib.pace_lightning_workspace_bytes(1, 4096, H, D, P)
    assert fewer < 40 << 20 < need
    real = torch.empty

    def empty(*size, **kw):
        if room and size[0] == need:
            raise torch.OutOfMemoryError("no room for the scratch")
        return real(*size, **kw)
    monkeypatch.setattr(torch, "empty", empty)
    torch.ops.pace_b200.lightning_prefill(step.handle, x, decay, b, out)
    monkeypatch.setattr(torch, "empty", real)
    assert torch.equal(out, want) == (room == 0)         # (the other chunks ran)
    _close(out, want.double(), 2.0 ** -8)
    _close(b, a.double(), 1e-4)


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("bad", [0, 15, 16, 77, 127, 128, 200])
def test_values_of_later_tokens_stay_out(bad, value):
    """A token's infinity or NaN among its values reaches no token in front of its 16."""
    from pace_b200.ops import hybrid
    n, H, D, P, G = 260, 2, 128, 72, 1
    g = torch.Generator(device=DEV).manual_seed(bad)
    step, keep = _step([n], [0]), bad // 16 * 16
    x = torch.randn(n, H * (2 * D + P), device=DEV, generator=g).bfloat16()
    decay = torch.full((H,), 0.9, device=DEV)
    y = x.clone()
    y[bad, 2 * H * D:] = value
    want, got = (hybrid.lightning(step, t, decay, torch.zeros(1, H, D, P, device=DEV)) for t in (x, y))
    assert torch.equal(got[:keep], want[:keep]) and not torch.isfinite(got[bad]).all()
    x = torch.randn(n, H * P + 2 * G * D, device=DEV, generator=g).bfloat16()
    y = x.clone()
    y[bad, : H * P] = value
    dt, bias, neg_a, skip = torch.randn(n, H, device=DEV, generator=g).bfloat16(), *(torch.rand(3, H, device=DEV, generator=g) - 1)
    outs = []
    for t in (x, y):
        outs.append(torch.empty(n, H * P, device=DEV, dtype=torch.bfloat16))
        torch.ops.pace_b200.ssd_prefill(step.handle, t, dt, bias, neg_a, skip, torch.zeros(1, H, D, P, device=DEV), outs[-1], G)
    assert torch.equal(outs[1][:keep], outs[0][:keep]) and not torch.isfinite(outs[1][bad]).all()
