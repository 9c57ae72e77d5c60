"""Scratch of lightning and state-space prompts: bounded, whatever the step."""
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
        if max(lens) > 128 and heads * vdim <= 64 * 128:
            assert n > fewer                                 # the larger chunks are taken


BUDGET = 512     # MB
