"""Decode launches whose units are cut by position (a unit weighs more than its chunks), in chains in which the next launch works its
partition out ahead: lengths at the edges of chunks and shares, empty sequences, few and many thread blocks."""
import pytest
import torch

from test_attn_mma_gpu import DEV, Cfg, _check, _fill, _oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ctas", [0, 1, 7])
@pytest.mark.parametrize("lens", [[1, 6400, 64, 1, 65, 3], [0, 0, 2049, 0], [3000], [97, 0, 128, 1024, 4095, 63, 577] * 3])
def test_cut_units(lens, ctas):
    from pace_b200.llm.cache import KVCacheManager, KVCacheType
    from pace_b200.ops import MultiHeadAttention
    layers, Hq, Hkv, D, B = 3, 8, 2, 128, len(lens)
    g = torch.Generator().manual_seed(sum(lens))
    ks = [torch.randn(Hkv, n, D, generator=g).bfloat16().to(DEV) for n in lens]
    vs = [torch.randn(Hkv, n, D, generator=g).bfloat16().to(DEV) for n in lens]
    mgr = KVCacheManager(Cfg(layers), max(lens) + 8, KVCacheType.BMC)
    kv = [_fill(mgr, i, ks, vs) for i in range(layers)]
    q = torch.randn(layers, B, Hq, 1, D, generator=g).bfloat16().to(DEV)
    got = [MultiHeadAttention()(q[i], *kv[i], max_ctas=ctas, whole_units=False) for i in range(layers)]
    mgr.pool.check_status()
    some = [b for b in range(B) if lens[b]]
    for i in range(layers):
        want = _oracle(q[i][some], [ks[b] for b in some], [vs[b] for b in some])
        for b, w in zip(some, want):
            _check(got[i][b], w)
        assert all(not got[i][b].any() for b in range(B) if not lens[b])


@pytest.mark.parametrize("new,past", [([1, 300, 64, 2, 129, 0, 65], 0), ([1500, 3, 1], 70), ([9] * 5, 1000), ([12, 0, 9, 11], 3000), ([70] * 23, 1),
                                      # 12 to 32 rows of a unit: cut in two, in a few, in many parts (one warp merges them)
                                      ([3], 3000), ([4, 0, 4, 3], 700), ([5] * 12, 300), ([8, 1, 7], 2000), ([6] * 40, 500), ([5], 9000)])
def test_cut_units_of_many_query_rows(new, past):
    """Prompts and verify passes whose units are cut by position: tokens at the edges of tiles, sequences that sit out."""
    from pace_b200.llm.cache import KVCacheManager, KVCacheType
    from pace_b200.ops import MultiHeadAttention
    Hq, Hkv, D, B, S = 8, 2, 128, len(new), max(new)
    g = torch.Generator().manual_seed(sum(new))
    lens = [past + n for n in new]
    ks = [torch.randn(Hkv, n, D, generator=g).bfloat16().to(DEV) for n in lens]
    vs = [torch.randn(Hkv, n, D, generator=g).bfloat16().to(DEV) for n in lens]
    mgr = KVCacheManager(Cfg(1), max(lens) + 8, KVCacheType.BMC)
    kv = _fill(mgr, 0, ks, vs)
    q = torch.randn(B, Hq, S, D, generator=g).bfloat16().to(DEV)
    got = MultiHeadAttention()(q, *kv, q_lens=torch.tensor(new, dtype=torch.int32, device=DEV))
    mgr.pool.check_status()
    some = [b for b in range(B) if new[b]]
    for b, w in zip(some, _oracle(q[some], [ks[b] for b in some], [vs[b] for b in some], q_lens=[new[b] for b in some])):
        _check(got[b][:, : new[b]], w)


@pytest.mark.parametrize("new", [1, 9])
@pytest.mark.parametrize("heads,kv,lens", [(4, 1, [40000, 70]), (8, 2, [70001])])
def test_long_units(heads, kv, lens, new):
    """Units so long that a share's bound cuts them into more than sixteen parts."""
    from pace_b200.llm.cache import KVCacheManager, KVCacheType
    from pace_b200.ops import MultiHeadAttention
    D, B = 128, len(lens)
    g = torch.Generator().manual_seed(lens[0])
    ks = [torch.randn(kv, n, D, generator=g).bfloat16().to(DEV) for n in lens]
    vs = [torch.randn(kv, n, D, generator=g).bfloat16().to(DEV) for n in lens]
    mgr = KVCacheManager(Cfg(2), max(lens) + 8, KVCacheType.BMC)
    cached = [_fill(mgr, i, ks, vs) for i in range(2)]
    q = torch.randn(2, B, heads, new, D, generator=g).bfloat16().to(DEV)
    got = [MultiHeadAttention()(q[i], *cached[i]) for i in range(2)]
    mgr.pool.check_status()
    for i in range(2):
        for b, w in enumerate(_oracle(q[i], ks, vs, q_lens=[new] * B)):
            _check(got[i][b], w)
