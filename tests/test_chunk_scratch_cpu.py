"""Scratch of lightning and state-space prompts: bounded, whatever the step, and which steps take the larger chunks."""
import pytest
import torch


@pytest.mark.parametrize("lens", [[129], [4096], [16384], [300] * 64, [100000, 1, 1], [128] * 8])
@pytest.mark.parametrize("heads,vdim", [(1, 64), (16, 128), (64, 64), (64, 128), (128, 256), (5000, 128)])
def test_scratch_is_bounded(lens, heads, vdim):
    from pace_b200 import _C
    from pace_b200.llm.step import Step
    st = Step(lens, [0] * len(lens), range(len(lens)), torch.zeros(sum(lens), dtype=torch.long), 1, "cpu").struct
    for new, old in (("lightning", _C.lib.pace_lightning_workspace_bytes), ("ssd", _C.lib.pace_ssd_workspace_bytes)):
        n = getattr(_C.lib, f"pace_{new}_scratch_bytes")(st, heads, 128, vdim, _C.DTYPE_BF16)
        fewer = old(len(lens), max(lens), heads, 128, vdim)
        assert fewer <= n <= max(fewer, (BUDGET << 20) + 256)
        if max(lens) >= 4096 and heads * vdim <= 64 * 128:
            assert n > fewer                                 # the larger chunks are taken


BUDGET = 512     # MB


# one prompt or several, as calls of either form were timed: few tokens and half empty last chunks stay with the chunks of 64
@pytest.mark.parametrize("op,heads,vdim,lens,larger", [
    ("ssd", 64, 64, [107, 263], False), ("ssd", 64, 64, [77, 144], False), ("ssd", 32, 64, [300], False), ("ssd", 32, 64, [400], True),
    ("ssd", 32, 64, [300] * 4, False), ("ssd", 32, 64, [300] * 8, False), ("ssd", 32, 64, [500] * 8, True), ("ssd", 64, 64, [600] * 4, True),
    ("ssd", 32, 64, [203, 244, 293, 352, 423, 508, 610, 733], True), ("ssd", 32, 128, [300], True), ("ssd", 32, 128, [600] * 4, False),
    ("ssd", 32, 64, [128], False), ("lightning", 16, 128, [130], True), ("lightning", 16, 128, [4096], True),
    ("lightning", 32, 128, [130] * 4, False), ("lightning", 32, 128, [300] * 4, False), ("lightning", 32, 128, [500] * 8, True),
    ("lightning", 16, 128, [300] * 8, False), ("lightning", 16, 128, [1] * 8, False)])
def test_which_chunks(op, heads, vdim, lens, larger):
    from pace_b200 import _C
    from pace_b200.llm.step import Step
    st = Step(lens, [0] * len(lens), range(len(lens)), torch.zeros(sum(lens), dtype=torch.long), 1, "cpu").struct
    n = getattr(_C.lib, f"pace_{op}_scratch_bytes")(st, heads, 128, vdim, _C.DTYPE_BF16)
    assert (n > getattr(_C.lib, f"pace_{op}_workspace_bytes")(len(lens), max(lens), heads, 128, vdim)) == larger
