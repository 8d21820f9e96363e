"""Batched windows whose graph has more nodes without in-edges than the source: the
reference's consensus walk starts at the source, so it reaches neither the nodes
behind another start nor the sink, and prints an empty consensus. A negative match
score (match keeps its sign) makes such graphs; zero and free scores make many ties.
The CPU restatement, poa_run and a batch agree on all of them.
"""
import numpy as np
import pytest

import poa_b200
from poa_b200 import synth
from tests import oracle_graph

pytestmark = pytest.mark.gpu

BANDS = {"static": [], "adaptive": ["-B"], "full": ["-f", "0"]}
SCORES = {"m-2": ["-M", "-2", "-X", "1", "-O", "3", "-E", "1"], "m-1": ["-M", "-1", "-X", "4", "-O", "1", "-E", "0"],
          "m-5": ["-M", "-5", "-X", "1", "-O", "1", "-E", "1"], "m0": ["-M", "0", "-X", "1", "-O", "1", "-E", "0"]}


def _windows(score):
    """Windows of 40-300 bp, and one long read: slots and consensus buffers are sized by the
    batch's largest window and read, which leaves room for reads that share no node."""
    rng = np.random.default_rng(len(score))
    wins = [[synth.to_ascii(synth.random_root(rng, 4500))]]
    for length, n in [(40, 6)] * 8 + [(90, 10)] * 4 + [(300, 12)]:
        t = synth.random_root(rng, length)
        wins.append([synth.to_ascii(r) for r in synth.mutate(rng, t, n, 0.06, 0.045, 0.045)])
    return wins


@pytest.mark.parametrize("smem", [0, 18432])
@pytest.mark.parametrize("band", sorted(BANDS))
@pytest.mark.parametrize("score", sorted(SCORES))
def test_second_source(score, band, smem, oracle_bin):
    opts = SCORES[score] + BANDS[band]
    wins = _windows(score)
    want = [oracle_graph.run(w, opts) for w in wins]
    assert all(st == 0 for st, _, _ in want)
    if score != "m0":
        assert sum(steps[-1]["sources"] > 1 for _, steps, _ in want) >= 8
    ws = synth.pack_windows_from_reads(sum(wins, []), np.concatenate([[0], np.cumsum([len(w) for w in wins])]).tolist())
    with poa_b200.Context(poa_b200.Params.from_cli(opts)) as ctx:
        if smem:
            ctx.batch_config(smem_per_warp=smem)
        ctx.batch_upload(ws)
        ctx.batch_run()
        cons, status = ctx.batch_download()
        stats = ctx.batch_read_stats()
        text = [ctx.run(w, None)[0] for w in wins[:4]]
    assert status == [0] * len(wins)
    assert stats[:, 3].tolist() == [s["nodes"] for _, steps, _ in want for s in steps]
    assert stats[:, 6].tolist() == [s["edges"] for _, steps, _ in want for s in steps]
    assert cons == [c for _, _, c in want]
    assert text == [b">consensus sequence\n" + c + b"\n" for _, _, c in want[:4]]
