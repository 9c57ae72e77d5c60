"""One token per sequence of gated linear attention: few heads and more than the SMs hold at once, odd sizes, fresh sequences, against
64-bit arithmetic."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("B,H,D,P", [(3, 4, 128, 128), (40, 8, 128, 128), (40, 8, 72, 96), (100, 3, 40, 36), (75, 4, 136, 260), (297, 1, 33, 5)])
def test_step(dtype, B, H, D, P):
    from pace_b200.llm.step import Step
    from pace_b200.ops import hybrid
    g = torch.Generator(device="cuda").manual_seed(B + D + P)
    r = lambda *s, d=dtype: torch.randn(*s, device="cuda", generator=g, dtype=torch.float32).to(d)        # noqa: E731
    starts = [0 if b % 5 == 2 else 3 for b in range(B)]
    step = Step([1] * B, starts, range(B), torch.zeros(B, dtype=torch.long), 1, "cuda")
    qkv, z, gate = r(B, H * (2 * D + P)), r(B, H * D), r(B, H * P)
    S, z_bias, norm = r(B, H, D, P, d=torch.float32), r(H * D, d=torch.float32), 1 + 0.1 * r(P, d=torch.float32)
    q, k, v = (t.double().unflatten(1, (H, -1)) for t in qkv.split([H * D, H * D, H * P], 1))
    decay = torch.sigmoid(z.double() + z_bias.double()).unflatten(1, (H, D)) ** (1 / 16)
    old = S.double() * torch.tensor([float(x > 0) for x in starts], device="cuda", dtype=torch.float64)[:, None, None, None]
    new = old * decay[..., None] + k[..., None] * v[:, :, None]
    o = (new * q[..., None]).sum(2) * D ** -0.5
    want = o / torch.sqrt((o * o).mean(-1, keepdim=True) + 1e-6) * norm.double() * torch.nn.functional.silu(gate.double()).unflatten(1, (H, P))
    got = hybrid.gla(step, qkv, z, z_bias, S, norm, gate, 16.0, D ** -0.5, 1e-6)
    # the state: a product and a sum of 32 bits, decays to some ulp; the output: sums over D in 32 bits, then rounded to the type
    assert (S.double() - new).abs().max() <= 2e-5 * new.abs().max()
    tol = 2.0 ** -8 if dtype == torch.bfloat16 else 5e-5
    assert (got.double() - want.flatten(1)).norm() <= tol * want.norm()
