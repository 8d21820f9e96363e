"""Batched windows where the row fill and the backtrack change their path: scores
at the limit of the byte tables and beyond it, more predecessors than the staged
records, predecessors and successors beyond the rows whose state is kept in
shared memory, and gaps whose origin lies further than one search step to the
left. Warps and teams both print the CPU restatement's consensus.
"""
import subprocess

import numpy as np
import pytest

import poa_b200
from poa_b200 import synth

pytestmark = pytest.mark.gpu

BANDS = {"static": [], "adaptive": ["-B"], "full": ["-f", "0"]}


def _bases(rng, n):
    return bytes(rng.choice(list(b"ACGT"), size=n).astype(np.uint8))


def _check(reads, opts, oracle_bin, tmp_path):
    fa = tmp_path / "w.fa"
    synth.write_fasta(str(fa), reads)
    want = subprocess.run([oracle_bin, str(fa)] + opts, capture_output=True, check=True, timeout=300).stdout.split(b"\n")[1]
    ws = synth.pack_windows_from_reads(reads, [0, len(reads)])
    for smem in (0, 18432):  # a configured shared-memory size: one warp per window
        with poa_b200.Context(poa_b200.Params.from_cli(opts)) as ctx:
            if smem:
                ctx.batch_config(smem_per_warp=smem)
            cons, st = ctx.batch_consensus(ws)
        assert st == [0] and cons[0] == want, smem


@pytest.mark.parametrize("band", sorted(BANDS))
@pytest.mark.parametrize("match,mismatch", [(127, 127), (128, 4), (5, 128), (127, 128), (128, 129)])
def test_score_table_limits(match, mismatch, band, oracle_bin, tmp_path):
    rng = np.random.default_rng(match * 1000 + mismatch)
    t = _bases(rng, 260)
    reads = [t] + [t[:40 + 7 * k] + _bases(rng, 2) + t[44 + 7 * k + k % 3:] for k in range(7)]
    _check(reads, ["-M", str(match), "-X", str(mismatch), "-O", "20", "-E", "9"] + BANDS[band], oracle_bin, tmp_path)


@pytest.mark.parametrize("band", sorted(BANDS))
def test_many_and_far_predecessors(band, oracle_bin, tmp_path):
    rng = np.random.default_rng(9)
    t = _bases(rng, 640)
    P = 420
    dels = list(range(1, 41)) + [62, 63, 64, 65, 126, 127, 128, 129, 200, 300]
    reads = [t] + [t[:P - k] + t[P:] for k in dels] + [t[:200] + _bases(rng, 9) + t[330:]]
    _check(reads, ["-b", "600"] + BANDS[band], oracle_bin, tmp_path)


@pytest.mark.parametrize("band", sorted(BANDS))
@pytest.mark.parametrize("ins", [126, 127, 128, 129, 254, 257, 511, 514, 700])
def test_long_insertions(ins, band, oracle_bin, tmp_path):
    rng = np.random.default_rng(ins)
    t = _bases(rng, 300)
    reads = [t, t[:150] + _bases(rng, ins) + t[150:], t, t[:150] + _bases(rng, ins + 3) + t[150:]]
    _check(reads, ["-b", "900", "-O", "6", "-E", "1"] + BANDS[band], oracle_bin, tmp_path)
