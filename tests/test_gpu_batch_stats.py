"""Read statistics describe the window, not the launch it ran in: the same windows
alone, among 300 and in a batch that fills the GPU report the same numbers."""
import numpy as np
import pytest

import poa_b200
from poa_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("opts", [[], ["-B"], ["-f", "0"]], ids=["static", "adaptive", "full"])
def test_read_stats_do_not_depend_on_the_batch(opts):
    rng = np.random.default_rng(71)
    few = []
    for length in (640, 620, 300):
        t = synth.random_root(rng, length)
        few.append([synth.to_ascii(r) for r in synth.mutate(rng, t, 6, 0.05, 0.04, 0.04)])
    longest = max(len(r) for w in few for r in w)  # the batch's longest read sets the ring's width
    pad = [r[:longest] for r in [synth.to_ascii(synth.random_root(rng, 200)) for _ in range(2)]]
    got = {}
    for total in (3, 300, 3 * 4 * 148 + 40):
        reads, offs = [], [0]
        for w in few + [pad] * (total - 3):
            reads += w
            offs.append(len(reads))
        ws = synth.pack_windows_from_reads(reads, offs)
        with poa_b200.Context(poa_b200.Params.from_cli(opts)) as ctx:
            ctx.batch_upload(ws)
            ctx.batch_run()
            _, status = ctx.batch_download()
            got[total] = ctx.batch_read_stats()[:offs[3]].tolist()
        assert status == [0] * total
    assert got[3] == got[300] == got[3 * 4 * 148 + 40]
