"""The work a program has this library do, as timed cases over its public entry points.

Three groups, each through the calls a caller makes:

* ``run``: one read set, one graph (``Context.run``): consensus, row-column MSA
  and GFA output; static band, adaptive band (``-B``), seeding (``-S``).
* ``windows``: many independent windows (``Context.batch_consensus``), host
  buffers in, consensus strings out; static band, adaptive band, adaptive band
  planned by the proposer.
* ``predict`` / ``gradient``: the proposer's network, inference and one
  training step's loss and gradient.

Everything is synthetic and made from the seed: uniform random templates, reads
with substitutions, insertions and deletions 4:3:3, as in poa_b200/synth.py.
The windows are mutated on the GPU, because a large set takes the host minutes.
"""
import math

import numpy as np
import torch

import poa_b200 as pb
from poa_b200 import synth

BINS, CIN, CH, KW, OUT = 32, 8, 64, 3, 4  # the proposer's network (include/poa_b200.h)


def listed():
    return [
        # a handful of short reads, the smallest call there is: barcode or UMI family consensus
        _run("umi_family", reads=4, length=90, err=0.03),
        # one amplicon as rows of an alignment, ragged small reads
        _run("amplicon_msa", reads=24, length=443, err=0.05, result=1),
        # a set of whole mitochondrial-size sequences, consensus (the benchmark's first configuration)
        _run("genome_consensus", reads=10, length=16569, err=0.015),
        # related sequences of one phylogeny, seeded, MSA (the benchmark's second configuration, a third of its reads)
        _run("phylogeny_seeded_msa", reads=36, length=16500, err=0.002, seeding=True, tree=True, result=1),
        # noisy long reads with the adaptive band (the benchmark's third configuration, fewer and shorter reads), the graph written out
        _run("noisy_adaptive_graph", reads=10, length=5000, err=0.10, adaptive=True, result=2),
        # one deep polishing window on its own: a correction done on demand
        _win("polish_one", windows=1, lo=600, hi=600, rlo=64, rhi=64, err=0.08),
        # a small batch of polishing windows, fewer than the GPU has SMs
        _win("polish_small", windows=96, lo=400, hi=600, rlo=4, rhi=64, err=0.08),
        # a full batch of polishing windows (the benchmark's polishing configuration, fewer windows)
        _win("polish_batch", windows=8000, lo=400, hi=600, rlo=4, rhi=64, err=0.08),
        # an ordinary batch of ragged windows with the adaptive band
        _win("adaptive_ragged", windows=240, lo=150, hi=900, rlo=3, rhi=20, err=0.12, adaptive=True),
        # long noisy windows with chimeric reads, planned by the proposer (the benchmark's default workload, fewer reads)
        _win("planned_batch", windows=1024, lo=2000, hi=2000, rlo=6, rhi=18, err=0.15, chimeric=0.01, adaptive=True,
             planned=True),
        # the proposer's prediction for the reads of such a batch
        {"name": "proposer_predict", "kind": "predict", "reads": 20000},
        # the loss and gradient of one training step at the trainer's batch size
        {"name": "proposer_gradient", "kind": "gradient", "reads": 256},
    ]


def _run(name, **kw):
    c = dict(kind="run", reads=4, length=100, err=0.05, adaptive=False, seeding=False, tree=False, result=0, scoring="default")
    c.update(kw)
    if name:
        c["name"] = name
    return c


def _win(name, **kw):
    c = dict(kind="windows", windows=1, lo=100, hi=100, rlo=2, rhi=2, err=0.08, chimeric=0.0, adaptive=False, planned=False,
             scoring="default")
    c.update(kw)
    if name:
        c["name"] = name
    return c


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["run", "run", "run", "windows", "windows", "windows", "windows", "predict", "gradient"])
    if what == "predict":
        return {"kind": "predict", "reads": _log_int(rng, 1, 20000)}
    if what == "gradient":
        return {"kind": "gradient", "reads": _log_int(rng, 1, 4096)}
    scoring = rng.choice(["default", "default", "steep"])
    most = max(_ops(c) for c in listed() if c["kind"] in ("run", "windows"))
    while True:
        if what == "run":
            seeded = rng.random() < 0.15
            if seeded:
                c = _run(None, reads=_log_int(rng, 4, 36), length=_log_int(rng, 6000, 16500), err=0.002, seeding=True,
                         tree=True, result=1)
            else:
                c = _run(None, reads=_log_int(rng, 2, 40), length=_log_int(rng, 60, 16600),
                         err=round(rng.uniform(0.005, 0.12), 3), adaptive=rng.random() < 0.35,
                         result=rng.choice([0, 0, 1, 2]), scoring=scoring)
        else:
            adaptive = rng.random() < 0.45
            hi = _log_int(rng, 120, 2000 if adaptive else 1200)
            rhi = _log_int(rng, 3, 24 if adaptive else 64)
            c = _win(None, windows=_log_int(rng, 1, 8000), lo=max(100, int(hi * rng.uniform(0.4, 1.0))), hi=hi,
                     rlo=max(2, int(rhi * rng.uniform(0.2, 1.0))), rhi=rhi, err=round(rng.uniform(0.02, 0.15), 3),
                     chimeric=rng.choice([0.0, 0.0, 0.01]), adaptive=adaptive, planned=adaptive and rng.random() < 0.5,
                     scoring=scoring)
        rows = _rows(c) / c.get("windows", 1)
        # no dearer than the largest listed case: in all, and along the chain of rows of one graph
        if _ops(c) <= 0.5 * most and rows <= (180000 if what == "run" and not c["adaptive"] else 60000):
            return c


# ---- inputs -----------------------------------------------------------------
SCORING = {"default": (2, -4, -4, -2), "steep": (5, -4, -8, -6)}


def _params(c):
    m, x, o, e = SCORING[c["scoring"]]
    return pb.Params(match=m, mismatch=x, gap_open=o, gap_ext=e, ab_band=c["adaptive"],
                     seeding=c.get("seeding", False), result=c.get("result", 0))


def _mutated_windows(c, seed):
    """A synth.WindowSet of the case's shape, mutated on the GPU in groups of windows."""
    rng = np.random.default_rng(seed)
    n = c["windows"]
    L = rng.integers(c["lo"], c["hi"] + 1, size=n)
    R = rng.integers(c["rlo"], c["rhi"] + 1, size=n)
    gen = torch.Generator(device="cuda").manual_seed(int(seed) * 1000003 + 17)
    acgt = torch.tensor(list(b"ACGT"), dtype=torch.uint8, device="cuda")
    t_off = np.concatenate([[0], np.cumsum(L)])
    tmpl = torch.randint(0, 4, (int(t_off[-1]),), generator=gen, device="cuda", dtype=torch.uint8)
    seqs, lens = [], []
    group = max(1, int(2e7 / max(1.0, float((L * R).mean()))))
    for w0 in range(0, n, group):
        w1 = min(n, w0 + group)
        read_win = np.repeat(np.arange(w0, w1), R[w0:w1])
        read_len = L[read_win]
        nr, total = len(read_win), int(read_len.sum())
        src = t_off[:-1][read_win]  # where each read's template starts
        # a chimeric read's second half comes from another window's template
        other = np.where(rng.random(nr) < c["chimeric"], rng.integers(0, n, size=nr), read_win)
        first = np.concatenate([[0], np.cumsum(read_len)[:-1]])
        tot = torch.as_tensor(read_len, device="cuda")
        rid = torch.repeat_interleave(torch.arange(nr, device="cuda"), tot, output_size=total)
        pos = torch.arange(total, device="cuda") - torch.as_tensor(first, device="cuda")[rid]
        half = pos >= (tot // 2)[rid]
        a = torch.as_tensor(src, device="cuda")[rid] + pos
        b = torch.as_tensor(t_off[:-1][other], device="cuda")[rid] + pos % torch.as_tensor(L[other], device="cuda")[rid]
        base = tmpl[torch.where(half, b, a)]
        u = torch.rand(total, generator=gen, device="cuda")
        e = c["err"]
        turn = torch.randint(1, 4, (total,), generator=gen, device="cuda", dtype=torch.uint8)
        base = torch.where(u < 0.4 * e, (base + turn) & 3, base)
        ins = (u >= 0.4 * e) & (u < 0.7 * e)
        keep = ~((u >= 0.7 * e) & (u < e))
        count = keep.to(torch.int64) + ins.to(torch.int64)
        at = torch.cumsum(count, 0) - count
        out = torch.empty(int(count.sum()), dtype=torch.uint8, device="cuda")
        out[at[keep]] = acgt[base[keep].long()]
        extra = torch.randint(0, 4, (total,), generator=gen, device="cuda", dtype=torch.uint8)
        out[at[ins] + 1] = acgt[extra[ins].long()]
        got = torch.zeros(nr, dtype=torch.int64, device="cuda").index_add_(0, rid, count)
        seqs.append(out.cpu().numpy())
        lens.append(got.cpu().numpy())
    torch.cuda.empty_cache()
    read_len = np.concatenate(lens).astype(np.int32)
    off = np.concatenate([[0], np.cumsum(read_len, dtype=np.int64)[:-1]]).astype(np.int64)
    return synth.WindowSet(seq=np.concatenate(seqs), read_off=off, read_len=read_len,
                           win_off=np.concatenate([[0], np.cumsum(R)]).astype(np.int32))


def _reads(c, seed):
    if c["tree"]:
        return synth.single_graph_msa(seed=seed, nseq=c["reads"], length=c["length"], branch_div=c["err"])
    rng = np.random.default_rng(seed)
    root = synth.random_root(rng, c["length"])
    e = c["err"]
    return [synth.to_ascii(r) for r in synth.mutate(rng, root, c["reads"], 0.4 * e, 0.3 * e, 0.3 * e)]


def _features(n, seed):
    """Features and targets with the ranges that poa_batch_features and the band statistics have."""
    rng = np.random.default_rng(seed)
    X = np.empty((n, BINS, CIN), dtype=np.float32)
    X[:, :, 0] = rng.gamma(4.0, 0.2, (n, BINS))
    X[:, :, 1] = rng.beta(0.6, 1.2, (n, BINS))
    X[:, :, 2] = X[:, :, 1] * rng.gamma(2.0, 0.3, (n, BINS))
    X[:, :, 3] = rng.uniform(0.9, 1.05, (n, 1))
    X[:, :, 4] = rng.uniform(0.9, 1.05, (n, 1))
    X[:, :, 5] = rng.integers(0, 100, (n, 1)) / 100.0
    X[:, :, 6] = rng.integers(20, 101, (n, 1)) / 100.0
    X[:, :, 7] = (np.arange(BINS) + 0.5) / BINS
    Y = np.stack([rng.gamma(2.0, 0.03, n), rng.uniform(0.1, 0.4, n), rng.uniform(1.5, 3.0, n), rng.normal(0.5, 0.02, n)],
                 axis=1).astype(np.float32)
    return X, Y


def prepare(case, seed):
    c = case
    if c["kind"] in ("predict", "gradient"):
        X, Y = _features(c["reads"], seed)
        return {"case": c, "prop": pb.Proposer(weights=pb.PROP_WEIGHTS), "X": X, "Y": Y}
    ctx = pb.Context(_params(c))
    if c["kind"] == "run":
        return {"case": c, "ctx": ctx, "reads": _reads(c, seed), "room": _room(c)}
    if c["planned"]:
        ctx.batch_use_proposer(pb.Proposer(weights=pb.PROP_WEIGHTS))
    return {"case": c, "ctx": ctx, "windows": _mutated_windows(c, seed), "room": _room(c)}


def _room(c):
    """Bytes that hold the longest text of the case's shape (per window for a batch): outputs of every seed have one shape."""
    if c["kind"] == "windows":
        return 2 * c["hi"] + 64
    n, length = c["reads"], c["length"]
    return [2 * length + 64, n * (4 * length + 64), 60 * n * length + 4096][c["result"]]


def _padded(text, room):
    out = np.zeros(room, dtype=np.uint8)
    out[:len(text)] = np.frombuffer(text, dtype=np.uint8)
    return out


def run(state):
    kind = state["case"]["kind"]
    if kind == "run":
        text, scores = state["ctx"].run(state["reads"])
        return {"text": _padded(text, state["room"]), "scores": np.array(scores, dtype=np.int64)}
    if kind == "windows":
        cons, status = state["ctx"].batch_consensus(state["windows"])
        rows = np.frombuffer(b"".join([x.ljust(state["room"], b"\0") for x in cons]), dtype=np.uint8)
        return {"consensus": rows.reshape(len(cons), state["room"]),
                "lengths": np.array([len(x) for x in cons], dtype=np.int64), "status": np.array(status, dtype=np.int64)}
    if kind == "predict":
        return {"targets": state["prop"].predict(state["X"])}
    loss, grad = state["prop"].gradient(state["X"], state["Y"])
    return {"loss": loss, "grad": grad}


# ---- what a pass cannot do without ------------------------------------------
def _shape(c):
    """(windows, reads per window, mean length)."""
    if c["kind"] == "run":
        return 1, c["reads"], c["length"]
    return c["windows"], 0.5 * (c["rlo"] + c["rhi"]), 0.5 * (c["lo"] + c["hi"])


def _rows(c):
    """DP rows of a pass: every read after the first meets a graph that has grown by a share of each read's errors."""
    n, reads, length = _shape(c)
    k = max(0.0, reads - 1)
    return n * k * length * (1.0 + 0.4 * c["err"] * 0.5 * k)


def _ops(c):
    """Integer operations: 5 a band cell and 7 for each of its (about 1.3) predecessors, 1 more for the adaptive argmax."""
    _, _, length = _shape(c)
    width = min(length + 1.0, 2.0 * (100 + length / 40.0) + 1.0)
    if c.get("seeding"):
        width = min(width, 230.0)
    return _rows(c) * width * (5 + 7 * 1.3 + (1 if c["adaptive"] else 0))


def work(case):
    c = case
    if c["kind"] in ("predict", "gradient"):
        macs = BINS * CH * KW * (CIN + 2 * CH) + CH * CH + CH * OUT
        nparam = CH * KW * (CIN + 2 * CH) + 3 * CH + CH * CH + CH + CH * OUT + OUT
        n, back = c["reads"], c["kind"] == "gradient"
        return {"bytes": 4 * n * (BINS * CIN + OUT) + 2 * nparam + (4 * nparam if back else 0),
                "flops": 2 * macs * n * (3 if back else 1)}
    n, reads, length = _shape(c)
    out = n * length * (reads if c.get("result") else 1)
    return {"bytes": n * reads * length + out, "flops": _ops(c)}


# ---- the network in 64 bits -------------------------------------------------
def _network(w, X):
    """poa_prop_predict's standardised outputs from a flat parameter vector (float64, differentiable)."""
    at = 0

    def take(*shape):
        nonlocal at
        n = int(np.prod(shape))
        r = w[at:at + n].reshape(shape)
        at += n
        return r

    x = X
    for cin in (CIN, CH, CH):
        W, b = take(CH, KW, cin), take(CH)
        x = torch.relu(torch.nn.functional.conv1d(x.transpose(1, 2), W.permute(0, 2, 1), b, padding=1).transpose(1, 2))
    h = x.mean(dim=1)
    z = torch.relu(h @ take(CH, CH).T + take(CH))
    return z @ take(OUT, CH).T + take(OUT)


def exact(case, seed):
    if case["kind"] not in ("predict", "gradient"):
        return None  # text, consensus and whole numbers: compared as they are
    X, Y = _features(case["reads"], seed)
    flat = torch.from_numpy(np.fromfile(pb.PROP_WEIGHTS, dtype="<f4").astype(np.float64))
    w, mean, std = flat[:-12].clone(), flat[-12:-8], flat[-8:-4]
    X = torch.from_numpy(X.astype(np.float64))
    if case["kind"] == "predict":
        with torch.no_grad():
            y = torch.cat([_network(w, x) for x in X.split(1024)]) * std + mean
        return {"targets": y.numpy()}
    w.requires_grad_(True)
    o = _network(w, X)
    loss = ((o - (torch.from_numpy(Y.astype(np.float64)) - mean) / std) ** 2).mean()
    loss.backward()
    return {"loss": float(loss.detach()), "grad": w.grad.numpy()}
