"""Attention of 32-bit rows in register tiles (csrc/attn_general.cu) at the edges of its 64-row, 64-key tiles, against the plain
implementation in 64 bits."""
import pytest
import torch

from test_gekupel_gpu import attend, plain_attention, span_case

pytestmark = pytest.mark.gpu

# scores and outputs are sums of at most 128 and 197 products in fp32: (128 + 197) half units of 2^-23 of the values (below 5)
TOL = (128 + 197) * 2.0 ** -24 * 5


@pytest.mark.parametrize("dim,vdim", [(128, 128), (64, 64), (64, 72), (100, 36), (12, 4), (7, 5)])
@pytest.mark.parametrize("counts", [[1, 63, 64, 65, 4], [16, 17, 1, 1, 98], [197]])
@pytest.mark.parametrize("heads,kv,rule", [(8, 2, {}), (3, 3, {"window": 65}), (4, 1, {"chunk": 64}), (4, 2, {"window": 1})])
def test_tiles_against_plain(dim, vdim, counts, heads, kv, rule):
    n = sum(counts)
    qkv, cache = span_case(torch.float32, heads, kv, dim, vdim, n, seed=dim + heads)
    g = torch.Generator().manual_seed(5)
    more = {"slopes": torch.rand(heads, generator=g) * 0.1, "sinks": torch.randn(heads, generator=g)} if heads == 8 else {}
    got = attend(qkv, cache, 1, counts, heads, dim, vdim, dim ** -0.5, **rule, **more)
    want = plain_attention(qkv, heads, kv, dim, vdim, dim ** -0.5, **rule, **{k: v.double() for k, v in more.items()})
    assert (got - want.view(n, heads, vdim)).abs().max() < TOL


@pytest.mark.parametrize("heads,kv,rule", [(8, 2, {}), (3, 3, {"window": 65}), (4, 1, {"chunk": 64}), (2, 2, {"window": 9})])
@pytest.mark.parametrize("dim,vdim", [(128, 128), (64, 36)])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_values_out_of_sight_stay_out(heads, kv, rule, dim, vdim, value):
    """A token's infinity or NaN among its values reaches the rows that see it and no others."""
    n, bad = 197, (5, 63, 64, 130)
    qkv, _ = span_case(torch.float32, heads, kv, dim, vdim, n, seed=3)
    at = heads * dim + kv * dim
    clean = None
    for b in (None,) + bad:
        x = qkv.clone()
        if b is not None:
            x[b, at:] = value
        _, cache = span_case(torch.float32, heads, kv, dim, vdim, n, seed=3)
        got = attend(x, cache, 1, [n], heads, dim, vdim, dim ** -0.5, **rule)
        if b is None:
            clean = got
            continue
        pos = torch.arange(n)
        first = pos - rule["window"] + 1 if "window" in rule else pos // rule["chunk"] * rule["chunk"] if "chunk" in rule else torch.zeros(n)
        free = (pos < b) | (first > b)
        assert free.any() and torch.equal(got[free], clean[free])
        assert not torch.isfinite(got[b]).all()
