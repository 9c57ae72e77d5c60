"""Query rows that span attention is told of: a buffer for the decoding tokens of a mixed step is shorter than the step."""
import ctypes as C
from types import SimpleNamespace

import pytest
import torch


class _Recorder:
    """Stands in for the ops: keeps the calls, launches nothing."""

    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        def call(*args):
            self.calls.append((name, args))
            return True
        return call


@pytest.mark.parametrize("counts,absorbed", [([1, 17, 64], 1), ([40, 1, 1, 64], 2), ([1, 1], 2), ([3, 1, 2], 6)])
def test_rows_of_the_absorbed_queries(monkeypatch, counts, absorbed):
    from pace_b200 import _C, torch_ops
    from pace_b200.llm.step import Step
    from pace_b200.ops import hybrid
    heads, dim, vdim, rank, T = 5, 24, 40, 48, sum(counts)
    step = Step(counts, [7] * len(counts), range(len(counts)), torch.zeros(T, dtype=torch.long), 1, "cpu")
    rec = _Recorder()
    monkeypatch.setattr(hybrid, "_OPS", rec)
    cache = SimpleNamespace(pool=SimpleNamespace(head_dim=rank, handle=0, pages=None), layer=0)
    r = lambda *s: torch.zeros(*s, dtype=torch.bfloat16)      # noqa: E731
    hybrid.latent_attention(step, cache, r(T, rank), None, r(rank), None, r(heads * (dim + vdim), rank), heads, dim, 0, vdim, 1.0, 1e-5,
                            None, q=r(T, heads * dim))
    spans = [a[4:] for name, a in rec.calls if name == "attn_span"]
    assert spans
    for q, out, *rule in spans:
        assert q.shape[0] == absorbed <= T
        a = torch_ops._span_args(_C.AttnSpanArgs(), q, out, *rule)
        assert a.q_rows == q.shape[0]                         # the kernel's copies end there
        last = sum(step.counts[: a.entry_end])                # ... and every entry's tokens lie in front
        assert last <= a.q_rows
        a.q_rows, st = -1, step.struct                        # (refused before anything is launched)
        pool = _C.KVPoolStruct(n_layers=1, n_kv_heads=1, head_dim=rank, page_tokens=64, n_pages=1, max_seqs=4, max_pages_per_seq=4,
                               row_format=_C.ROWS_SHARED, pages=1 << 16, block_table=1 << 20)
        assert _C.lib.pace_attn_span(C.byref(pool), 0, C.byref(st), C.byref(a), None) == _C.PACE_ERR_INVALID
