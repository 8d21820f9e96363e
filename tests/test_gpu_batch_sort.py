"""The batched windows' topological sort: nodes with more out-edges than a warp
has lanes, many nodes that become ready at once, and stretches where none does
(the next node then comes from the stack). A wrong order changes the DP rows, so
every read's graph size and the consensus equal the CPU restatement's.
"""
import numpy as np
import pytest

import poa_b200
from poa_b200 import synth
from tests import oracle_graph

pytestmark = pytest.mark.gpu

BANDS = {"static": [], "adaptive": ["-B"], "full": ["-f", "0"]}


def _bases(rng, n):
    return bytes(rng.choice(list(b"ACGT"), size=n).astype(np.uint8))


def check(reads, opts, smem=0):
    st, steps, cons = oracle_graph.run(reads, opts)
    assert st == 0
    ws = synth.pack_windows_from_reads(reads, [0, len(reads)])
    with poa_b200.Context(poa_b200.Params.from_cli(opts)) as ctx:
        if smem:
            ctx.batch_config(smem_per_warp=smem)
        ctx.batch_upload(ws)
        ctx.batch_run()
        got, status = ctx.batch_download()
        stats = ctx.batch_read_stats()
    assert status == [0]
    assert stats[:, 3].tolist() == [s["nodes"] for s in steps]
    assert stats[:, 6].tolist() == [s["edges"] for s in steps]
    assert got[0] == cons


@pytest.mark.parametrize("smem", [0, 18432])
@pytest.mark.parametrize("band", sorted(BANDS))
def test_fan_out(band, smem, oracle_bin):
    rng = np.random.default_rng(31)
    t = _bases(rng, 400)
    # 45 deletions that start at one node, and 40 insertions after another: with dear
    # mismatches every insertion is a branch of its own, ready when that node is placed
    reads = [t] + [t[:100] + t[100 + k:] for k in range(1, 46)] + [t[:300] + _bases(rng, 5) + t[300:] for _ in range(40)]
    check(reads, ["-M", "2", "-X", "12", "-O", "1", "-E", "1"] + BANDS[band], smem)
