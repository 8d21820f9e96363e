"""Small adaptive batches run a team of warps per window, larger ones (or a
configured shared-memory size) one warp per window: the same windows give the
same consensus either way, at every team width and with rows wider than the
team's columns, and equal the CPU restatement's.
"""
import subprocess

import pytest

import poa_b200
from poa_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("length,opts", [(60, ["-B"]), (250, ["-B"]), (440, ["-B"]), (700, ["-B"]), (1300, ["-B"]),
                                         (1300, ["-B", "-b", "900"]),
                                         (300, ["-B", "-M", "5", "-X", "4", "-O", "8", "-E", "6"])])
def test_team_and_warp_agree(length, opts, oracle_bin, tmp_path):
    ws = synth.windows(length, 6, (max(30, length - 40), length), (2, 9), 0.13, chimeric=0.05)
    with poa_b200.Context(poa_b200.Params.from_cli(opts)) as ctx:
        ctx.batch_upload(ws)
        ctx.batch_run()
        team, st = ctx.batch_download()
        stats = ctx.batch_read_stats()
    with poa_b200.Context(poa_b200.Params.from_cli(opts)) as ctx:
        ctx.batch_config(smem_per_warp=18432)
        ctx.batch_upload(ws)
        ctx.batch_run()
        warp, st_w = ctx.batch_download()
        stats_w = ctx.batch_read_stats()
    assert st == st_w == [0] * ws.n_windows
    assert team == warp
    assert (stats == stats_w).all()
    for w in range(ws.n_windows):
        fa = tmp_path / f"w{w}.fa"
        synth.write_fasta(str(fa), ws.window_reads(w))
        out = subprocess.run([oracle_bin, str(fa)] + opts, capture_output=True, check=True, timeout=300).stdout
        assert team[w] == out.split(b"\n")[1], w
