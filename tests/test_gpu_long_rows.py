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


def _check(reads, opts, oracle_bin, tmp_path):
    fa = tmp_path / "in.fa"
    synth.write_fasta(str(fa), reads)
    want = subprocess.run([oracle_bin, str(fa)] + opts, capture_output=True, check=True, timeout=600).stdout
    with poa_b200.Context(poa_b200.Params.from_cli(opts)) as ctx:
        got, _ = ctx.run(reads, fasta.headers(str(fa)))
    assert got == want


# wide cells: teams of 8, 12 and 16 warps, and rows of two laps
@pytest.mark.parametrize("band", [["-f", "0"], ["-b", "2000"], ["-B", "-b", "60"], ["-B", "-b", "400"]],
                         ids=["full", "whole", "adaptive", "adaptive_b400"])
@pytest.mark.parametrize("length", [1016, 1030, 1528, 1540, 2040, 2056, 2600])
def test_wide_team_widths(length, band, oracle_bin, tmp_path):
    rng = np.random.default_rng(length)
    t = synth.random_root(rng, length)
    reads = [synth.to_ascii(r) for r in synth.mutate(rng, t, 3, 0.04, 0.02, 0.02)]
    # predecessors up to 40 rows back, beyond the rows kept in shared memory
    reads += [reads[0][:400] + reads[0][400 + k:] for k in (6, 7, 8, 9, 15, 16, 17, 40)]
    _check(reads, band + ["-r", "1"] + BIG, oracle_bin, tmp_path)


def test_wide_rows_around_sixteen_strips(oracle_bin, tmp_path):
    rng = np.random.default_rng(16)
    t = synth.random_root(rng, 3000)
    reads = [synth.to_ascii(r) for r in synth.mutate(rng, t, 4, 0.03, 0.01, 0.01)]
    s = _strips(3000, 925)
    assert sum(x <= 16 < y for x, y in zip(s, s[1:])) >= 5
    _check(reads, ["-b", "925", "-r", "1"] + BIG, oracle_bin, tmp_path)
