"""Residual sum and RMS norm in one pass, and projection outputs packed by sequence on their way into the cache."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("rows,width", [(1, 8), (3, 2048), (5, 2056), (33, 4096), (2, 4104), (7, 8192), (300, 136)])
@pytest.mark.parametrize("add", [True, False])
def test_add_norm(rows, width, add):
    import pace_b200.torch_ops  # noqa: F401
    g = torch.Generator(device=DEV).manual_seed(width)
    x, y = (torch.randn(rows, width, device=DEV, generator=g).bfloat16() for _ in range(2))
    w = (1 + torch.randn(width, device=DEV, generator=g) * 0.1).bfloat16()
    s, out = torch.full_like(x, 7.0), torch.empty_like(x)
    torch.ops.pace_b200.add_norm(x, y if add else None, w, s if add else None, out, 1e-5)
    total = x + y if add else x
    assert torch.equal(s, total) if add else bool((s == 7.0).all())
    z = total.double()
    want = z / torch.sqrt((z * z).mean(-1, keepdim=True) + 1e-5) * w.double()
    # one rounding to bf16 of a product with some ulp of 32 bits
    assert ((out.double() - want).abs() <= want.abs() * (2.0 ** -8) * 1.001).all()


@pytest.mark.parametrize("counts", [[5], [1, 0, 70, 3], [64, 65, 1], [0, 9], [1, 700, 30]])
def test_packed_rows_equal_padded_rows(counts):
    from pace_b200.llm.cache import KVCacheManager, KVCacheType
    from pace_b200.ops import RotaryEmbedding
    Hq, H, D, B, n = 4, 2, 128, len(counts), max(counts)
    g = torch.Generator(device=DEV).manual_seed(n)
    rope = RotaryEmbedding(None, D, 1024, 10000.0)
    packed = torch.randn(sum(counts), (Hq + 2 * H) * D, device=DEV, generator=g).bfloat16()
    q, k, v = (t.unflatten(1, (-1, D)) for t in packed.split([Hq * D, H * D, H * D], 1))
    rows = rope.table_rows(torch.arange(n, device=DEV).expand(B, n) + 3)
    at = [sum(counts[:b]) for b in range(B)]
    res = []
    for form in ("packed", "padded"):
        mgr = KVCacheManager(SimpleNamespace(num_hidden_layers=1), n + 8, KVCacheType.BMC)
        out = torch.zeros(B, n, Hq, D, device=DEV, dtype=torch.bfloat16)
        if form == "packed":
            mgr[0].update_cache_rope_packed(q, k, v, torch.tensor(at, dtype=torch.int32, device=DEV), counts,
                                            torch.tensor(counts, dtype=torch.int32, device=DEV), rows, rope, out)
        else:
            pad = [torch.zeros(B, n, x.shape[1], D, device=DEV, dtype=torch.bfloat16) for x in (q, k, v)]
            for b, c in enumerate(counts):
                for p, x in zip(pad, (q, k, v)):
                    p[b, :c] = x[at[b]: at[b] + c]
            mgr[0].update_cache_rope(*pad, rows, rope, n_new_per_seq=counts, query_out=out)
        mgr.pool.check_status()
        assert mgr[0].seq_lens == counts
        res.append((out, mgr[0].read_dense()))
    for b, c in enumerate(counts):
        assert torch.equal(res[0][0][b, :c], res[1][0][b, :c])
        for x, y in zip(res[0][1], res[1][1]):
            assert torch.equal(x[b, :, :c], y[b, :, :c])


def test_weights_side_by_side_give_the_same_layer():
    """One product of adjacent weights or three of separate ones; gradients and hooks keep the separate form."""
    from pace_b200.llm.models.llama import LlamaForCausalLM, _side_by_side
    cfg = SimpleNamespace(hidden_size=512, intermediate_size=1024, num_hidden_layers=1, num_attention_heads=4, num_key_value_heads=2,
                          vocab_size=64, max_position_embeddings=64, rope_theta=1e4, rms_norm_eps=1e-5, rope_scaling=None)
    torch.manual_seed(0)
    model = LlamaForCausalLM(cfg).to(DEV, torch.bfloat16)
    at, mlp = model.model.layers[0].self_attn, model.model.layers[0].mlp
    assert _side_by_side(at.q_proj, at.k_proj, at.v_proj).shape == (1024, 512)
    assert _side_by_side(mlp.gate_proj.linear, mlp.up_proj.linear).shape == (2048, 512)
    x = torch.randn(5, 512, device=DEV, dtype=torch.bfloat16)
    with torch.no_grad():
        fused, proj = mlp(x), at.project(x)
    sep = mlp(x)                                # parameters want gradients: the separate form
    assert sep.grad_fn is not None and fused.grad_fn is None
    assert (fused.float() - sep.float()).norm() <= 0.01 * sep.float().norm()
    for t, m in zip(proj, (at.q_proj, at.k_proj, at.v_proj)):
        want = x.double() @ m.weight.double().T
        assert (t.flatten(1).double() - want).norm() <= 2.0 ** -8 * want.norm()
    seen = []
    hook = at.k_proj.register_forward_hook(lambda *a: seen.append(1))
    with torch.no_grad():
        assert all(torch.equal(a, b) or (a.float() - b.float()).norm() <= 0.01 * b.float().norm() for a, b in zip(at.project(x), proj))
    assert seen == [1]
    hook.remove()


class Doubled(torch.nn.Module):
    """A projection with a forward of its own over a plain linear, as adapters are; fp32 out, rows that lie apart."""

    def __init__(self, base):
        super().__init__()
        self.base, self.weight, self.bias = base, base.weight, None

    def forward(self, x):
        return torch.cat([self.base(x).float() * 2, self.base(x[..., :1].expand_as(x)).float()], -1)[..., : self.weight.shape[0]]


def tiny_llama(layers=2):
    from pace_b200.llm.models.llama import LlamaForCausalLM
    cfg = SimpleNamespace(hidden_size=256, intermediate_size=512, num_hidden_layers=layers, num_attention_heads=4, num_key_value_heads=2,
                          vocab_size=64, max_position_embeddings=128, rope_theta=1e4, rms_norm_eps=1e-5, rope_scaling=None)
    torch.manual_seed(1)
    return LlamaForCausalLM(cfg).to(DEV, torch.bfloat16), cfg


def packed_logits(model, cfg, counts=(7, 3)):
    from pace_b200.llm.cache import KVCacheManager, KVCacheType
    mgr = KVCacheManager(cfg, 32, KVCacheType.BMC)
    ids = torch.arange(sum(counts)) % cfg.vocab_size
    return model.forward_packed(ids, list(counts), mgr, rows=range(len(ids))).logits


def close(a, b):
    return (a.double() - b.double()).norm() <= 0.03 * b.double().norm()


def test_packed_pass_calls_replaced_and_hooked_modules():
    model, cfg = tiny_llama()
    with torch.no_grad():
        want = packed_logits(model, cfg)
        for name in ("q_proj", "k_proj", "v_proj", "o_proj"):
            seen = []
            hooks = [getattr(lay.self_attn, name).register_forward_hook(lambda m, a, y: seen.append(1) or y) for lay in model.model.layers]
            assert close(packed_logits(model, cfg), want) and seen == [1, 1], name
            for h in hooks:
                h.remove()
        for name in ("q_proj", "v_proj"):
            at = model.model.layers[0].self_attn
            base = getattr(at, name)
            setattr(at, name, Doubled(base))
            got = packed_logits(model, cfg)
            setattr(at, name, base)
            base.weight.data.mul_(2)
            assert close(got, packed_logits(model, cfg)) and not close(got, want), name
            base.weight.data.mul_(0.5)
        model.model.layers[1].self_attn.q_proj.bias = torch.nn.Parameter(torch.ones(256, dtype=torch.bfloat16, device=DEV))
        assert not close(packed_logits(model, cfg), want)
        model.model.layers[1].self_attn.q_proj.bias = None
        assert torch.equal(packed_logits(model, cfg), want)


def test_forwards_of_single_objects_are_called():
    """A forward put on one layer, norm or projection, as offloading wrappers do."""
    from pace_b200.llm.cache import KVCacheManager, KVCacheType
    model, cfg = tiny_llama()
    ids = torch.arange(12, device=DEV).view(2, 6)

    def logits():
        return model(ids, kv_cache=KVCacheManager(cfg, 32, KVCacheType.BMC), attention_mask=torch.ones_like(ids)).logits
    with torch.no_grad():
        want = logits()
        lay = model.model.layers[0]
        for m in (lay, lay.input_layernorm, model.model.norm, lay.self_attn.v_proj, lay.mlp.gate_proj.linear):
            seen, own = [], m.forward
            m.forward = lambda *a, **k: seen.append(1) or own(*a, **k)          # noqa: B023
            got = logits()
            del m.forward
            assert seen and close(got, want), type(m)
            with torch.nn.modules.module.register_module_forward_hook(lambda mod, a, y: seen.append(2) if mod is m else None):
                assert close(logits(), want) and 2 in seen, type(m)


def test_transforms_see_the_whole_mlp():
    model, _ = tiny_llama(1)
    mlp = model.model.layers[0].mlp.requires_grad_(False)
    x, dx = torch.randn(4, 256, device=DEV).bfloat16(), torch.randn(4, 256, device=DEV).bfloat16()
    up, gate, down = (m.weight.double() for m in (mlp.up_proj.linear, mlp.gate_proj.linear, mlp.down_proj))
    _, want = torch.func.jvp(lambda t: (t @ up.T * torch.nn.functional.silu(t @ gate.T)) @ down.T, (x.double(),), (dx.double(),))
    _, got = torch.func.jvp(mlp, (x,), (dx,))
    assert close(got, want)
    assert close(torch.func.vmap(mlp)(x), mlp(x))
