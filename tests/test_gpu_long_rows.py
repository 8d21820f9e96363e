"""Static bands about as wide as the team's columns (16 strips of 128; 8 with wide
cells): as the band moves, rows that fit the team are followed by rows that do
not, which read every predecessor from the row store, and the other way round.
Every output equals the CPU restatement's.
"""
import subprocess

import numpy as np
import pytest

import poa_b200
from poa_b200 import synth
from tests import fasta

pytestmark = pytest.mark.gpu

BIG = ["-M", "400", "-X", "800", "-O", "900", "-E", "300"]  # 3,000 columns of these do not fit the packed cell


def _strips(length, b, f=40):
    """Strips of the rows of a graph that is one read, length bases long."""
    m = length + 1
    w = b + m // f
    bands = [(max(0, h - w) // 8, min(m, h + w) // 8 + 2) for h in range(m + 1)]
    return [((be - 2) >> 4) - (bs >> 4) + 1 for bs, be in bands]


@pytest.mark.parametrize("b", [905, 925, 948])
@pytest.mark.parametrize("scores,warps", [([], 16), (BIG, 8)], ids=["packed", "wide"])
def test_rows_around_the_teams_columns(scores, warps, b, oracle_bin, tmp_path):
    b = b if warps == 16 else b - 512
    rng = np.random.default_rng(b)
    t = synth.random_root(rng, 3000)
    reads = [synth.to_ascii(r) for r in synth.mutate(rng, t, 4, 0.03, 0.01, 0.01)]
    s = _strips(3000, b)
    assert sum(x <= warps < y for x, y in zip(s, s[1:])) >= 5  # a wider row after one that fits
    fa = tmp_path / "in.fa"
    synth.write_fasta(str(fa), reads)
    opts = ["-b", str(b), "-r", "1"] + scores
    want = subprocess.run([oracle_bin, str(fa)] + opts, capture_output=True, check=True, timeout=600).stdout
    with poa_b200.Context(poa_b200.Params.from_cli(opts)) as ctx:
        got, _ = ctx.run(reads, fasta.headers(str(fa)))
    assert got == want
