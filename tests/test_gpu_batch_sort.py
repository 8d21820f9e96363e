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


def _noisy(seed, length, n, err=0.15):
    rng = np.random.default_rng(seed)
    return [synth.to_ascii(r) for r in synth.mutate(rng, synth.random_root(rng, length), n, .4 * err, .3 * err, .3 * err)]


# 3,136 bytes a warp: lists in shared memory up to about 390 nodes, in-degrees up to 2,624
@pytest.mark.parametrize("band", sorted(BANDS))
@pytest.mark.parametrize("length,n", [(250, 8), (600, 10), (900, 24), (1200, 30)])
def test_lists_beyond_shared_memory(length, n, band, oracle_bin):
    check(_noisy(length, length, n), BANDS[band], 3136)


@pytest.mark.parametrize("band", sorted(BANDS))
def test_fan_out_beyond_shared_memory(band, oracle_bin):
    rng = np.random.default_rng(33)
    t = _bases(rng, 500)
    reads = [t] + [t[:100] + t[100 + k:] for k in range(1, 70)] + _noisy(3, 500, 6)
    check(reads, ["-M", "2", "-X", "12", "-O", "1", "-E", "1", "-b", "200"] + BANDS[band], 3136)


@pytest.mark.parametrize("n", [280, 320, 420])
def test_stack_beyond_shared_memory(n, oracle_bin):
    # a negative match score: every read is a chain with a start of its own, so the sort begins with n entries
    rng = np.random.default_rng(n)
    reads = [_bases(rng, 7) for _ in range(n)]
    opts = ["-M", "-1", "-X", "4", "-O", "1", "-E", "0", "-B"]
    st, steps, cons = oracle_graph.run(reads, opts)
    assert st == 0 and steps[-1]["sources"] >= n - 1
    room = [_bases(rng, 5000)]  # slots are sized by the batch's largest window
    ws = synth.pack_windows_from_reads(room + reads, [0, 1, 1 + n])
    with poa_b200.Context(poa_b200.Params.from_cli(opts)) as ctx:
        ctx.batch_config(smem_per_warp=3136)
        ctx.batch_upload(ws)
        ctx.batch_run()
        got, status = ctx.batch_download()
        stats = ctx.batch_read_stats()
    assert status == [0, 0] and got == [room[0], cons]
    assert stats[1:, 3].tolist() == [s["nodes"] for s in steps]
    assert stats[1:, 6].tolist() == [s["edges"] for s in steps]


def test_in_degree_beyond_a_byte(oracle_bin):
    rng = np.random.default_rng(35)
    t = _bases(rng, 420)
    check([t] + [t[:350 - k] + t[350:] for k in range(1, 290)], ["-b", "400"], 18432)


def test_cost_beyond_shared_memory(oracle_bin):
    """The sort of a graph of 3,000-5,000 nodes costs about the same a node whether its
    in-degrees and order fit the shared memory (20 KB) or only its in-degrees do (10 KB)."""
    reads = _noisy(36, 2000, 26)
    ws = synth.pack_windows_from_reads(reads, [0, len(reads)])
    cycles = {}
    for smem in (20480, 10240):
        with poa_b200.Context(poa_b200.Params(ab_band=True)) as ctx:
            ctx.batch_config(smem_per_warp=smem)
            ctx.batch_upload(ws)
            ctx.batch_run()
            ctx.batch_run()
            cycles[smem] = ctx.batch_stats()["phase_cycles"]["topsort"]
            assert 4000 < ctx.batch_read_stats()[-1, 3] < 6000
    assert cycles[10240] < 1.6 * cycles[20480], cycles
