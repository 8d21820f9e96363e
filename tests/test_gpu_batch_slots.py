"""Windows whose rows outgrow the slot sized from the batch's band: with reads of very
different lengths a static row spans the difference of the two, up to the whole
query. The engine re-runs them with larger slots and prints the CPU restatement's
consensus."""
import numpy as np
import pytest

import poa_b200
from poa_b200 import synth
from tests import oracle_graph

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lengths", [(5000, 10000), (10000, 3000), (1500, 6000, 1500, 6000)],
                         ids=["longer", "shorter", "turns"])
def test_reads_of_different_lengths(lengths, oracle_bin):
    rng = np.random.default_rng(sum(lengths))
    t = synth.random_root(rng, max(lengths))
    reads = [synth.to_ascii(synth.mutate(rng, t[:n], 1, 0.02, 0.01, 0.01)[0]) for n in lengths]
    st, steps, cons = oracle_graph.run(reads, [])
    assert st == 0
    ws = synth.pack_windows_from_reads(reads, [0, len(reads)])
    with poa_b200.Context() as ctx:
        ctx.batch_upload(ws)
        ctx.batch_run()
        got, status = ctx.batch_download()
        stats = ctx.batch_read_stats()
    assert status == [0] and got[0] == cons
    assert stats[:, 3].tolist() == [s["nodes"] for s in steps]
