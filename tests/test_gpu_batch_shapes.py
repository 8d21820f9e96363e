"""Configured launch shapes: more blocks per SM than any build of the batch kernel holds
run the 128-register build, 4 blocks, with the consensus of the default shape."""
import pytest

import poa_b200
from poa_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("opts", [[], ["-B"]], ids=["static", "adaptive"])
def test_more_blocks_than_fit(opts):
    ws = synth.windows(81, 2600, (60, 120), (3, 4), 0.08)  # more windows than 4 blocks of 4 warps an SM
    got, slots = {}, {}
    for blocks in (None, 4, 5, 8, 32):
        with poa_b200.Context(poa_b200.Params.from_cli(opts)) as ctx:
            if blocks:
                ctx.batch_config(blocks_per_sm=blocks, smem_per_warp=6144)
            got[blocks], status = ctx.batch_consensus(ws)
            slots[blocks] = ctx.batch_stats()["slots"]
        assert status == [0] * ws.n_windows
    assert got[4] == got[5] == got[8] == got[32] == got[None]
    assert slots[4] == slots[5] == slots[8] == slots[32]
