"""The single-alignment kernel (one team of warps per poa() call) at the sizes
and scorings where its paths change: the packed cell's limits and the wide
cell beyond them, gap openings of 0 and at the packed cell's 8 bits, rows at
the edges of strips, rows wider than the team's columns (laps), more than 32
predecessors of a node, and predecessors further back than the rows kept in
shared memory. Every output equals the CPU restatement's.
"""
import subprocess

import numpy as np
import pytest

import poa_b200
from tests import fasta

pytestmark = pytest.mark.gpu

BANDS = {"static": [], "adaptive": ["-B"], "full": ["-f", "0"]}
SCORES = {
    "linear": ["-O", "0"], "free_extend": ["-E", "0"], "free_gaps": ["-O", "0", "-E", "0"],
    "open_255": ["-O", "255", "-E", "1"], "open_256": ["-O", "256", "-E", "1"],
    "wide": ["-M", "4000", "-X", "9000", "-O", "12000", "-E", "6000"],
    "at_limit": ["-M", "1100", "-X", "1100", "-O", "200", "-E", "900"],
}


def _bases(rng, n):
    return bytes(rng.choice(list(b"ACGT"), size=n).astype(np.uint8))


def _noisy(rng, t, rate):
    out = bytearray()
    for c in t:
        u = rng.random()
        if u < 0.4 * rate:
            out += _bases(rng, 1)
        elif u < 0.7 * rate:
            out += bytes([c]) + _bases(rng, 1)
        elif u >= rate:
            out.append(c)
    return bytes(out)


def _check(reads, opts, oracle_bin, tmp_path):
    fa = tmp_path / "in.fa"
    with open(fa, "wb") as fh:
        for k, r in enumerate(reads):
            fh.write(b">r%d\n%s\n" % (k + 1, r))
    want = subprocess.run([oracle_bin, str(fa)] + opts, capture_output=True, timeout=300)
    _, seqs = fasta.read(str(fa))
    with poa_b200.Context(poa_b200.Params.from_cli(opts)) as ctx:
        if want.returncode != 0:  # the backtrack has no move there (free gaps): the same refusal
            with pytest.raises(poa_b200.PoaError) as err:
                ctx.run(seqs, fasta.headers(str(fa)))
            assert err.value.status in (1, 2)
            return
        got, _ = ctx.run(seqs, fasta.headers(str(fa)))
    assert got == want.stdout


@pytest.mark.parametrize("band", sorted(BANDS))
@pytest.mark.parametrize("score", sorted(SCORES))
def test_scorings(score, band, oracle_bin, tmp_path):
    rng = np.random.default_rng(11)
    t = _bases(rng, 420)
    _check([_noisy(rng, t, 0.1) for _ in range(7)], SCORES[score] + BANDS[band] + ["-r", "1"], oracle_bin, tmp_path)


@pytest.mark.parametrize("band", sorted(BANDS))
@pytest.mark.parametrize("length", [1, 7, 8, 9, 119, 126, 127, 128, 129, 255, 256, 257, 511, 513])
def test_strip_edges(length, band, oracle_bin, tmp_path):
    rng = np.random.default_rng(length)
    t = _bases(rng, length)
    _check([t, t, _noisy(rng, t, 0.05) or b"A", _bases(rng, 3) + t, t[1:] + b"C"], BANDS[band] + ["-b", "24", "-r", "1"],
           oracle_bin, tmp_path)


@pytest.mark.parametrize("opts", [["-f", "0"], ["-B", "-b", "1300"], ["-b", "1300"],
                                  ["-B", "-b", "1300", "-M", "400", "-X", "800", "-O", "900", "-E", "300"],
                                  ["-f", "0", "-M", "400", "-X", "800", "-O", "900", "-E", "300"]],
                         ids=["full", "adaptive", "static", "adaptive_wide", "full_wide"])
def test_laps(opts, oracle_bin, tmp_path):
    rng = np.random.default_rng(5)
    t = _bases(rng, 2600)
    _check([_noisy(rng, t, 0.06) for _ in range(4)], opts, oracle_bin, tmp_path)


@pytest.mark.parametrize("band", sorted(BANDS))
def test_many_predecessors_and_long_gaps(band, oracle_bin, tmp_path):
    rng = np.random.default_rng(9)
    a, b, c = _bases(rng, 90), _bases(rng, 160), _bases(rng, 70)
    reads = [a + b + c, a + c, a + _bases(rng, 150) + c, a + b + c]
    reads += [a + b[:k] + c for k in range(3, 153, 3)]  # each joins c from another node of b
    _check(reads, BANDS[band] + ["-r", "1"], oracle_bin, tmp_path)
