"""The CPU restatement's graph after every read (test infrastructure): what the
batched engine reports per read, and the consensus."""
import ctypes
import os

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LIB = os.path.join(ROOT, "oracle", "build", "libpoa_oracle.so")

P32 = ctypes.POINTER(ctypes.c_int)
PU8 = ctypes.POINTER(ctypes.c_uint8)


class OParams(ctypes.Structure):
    _fields_ = [(n, ctypes.c_int) for n in ("match", "mismatch", "gap_open1", "gap_ext1", "b", "f", "ab_band",
                                            "verbose")]


def _lib():
    o = ctypes.CDLL(LIB)
    vp = ctypes.c_void_p
    o.po_graph_new.restype = vp
    o.po_graph_free.argtypes = [vp]
    o.po_alignment.argtypes = [vp, ctypes.POINTER(OParams), PU8, ctypes.c_int, ctypes.POINTER(vp), P32, P32]
    o.po_add_path.argtypes = [vp, ctypes.c_int, vp, ctypes.c_int, ctypes.c_int]
    o.po_topsort.argtypes = [vp, ctypes.POINTER(OParams), ctypes.c_int]
    o.po_graph_sizes.argtypes = [vp] + [P32] * 5
    o.po_graph_export.argtypes = [vp, PU8] + [P32] * 12
    o.po_consensus.argtypes = [vp, P32]
    o.po_consensus.restype = vp
    o.po_params_default.argtypes = o.po_params_normalize.argtypes = [ctypes.POINTER(OParams)]
    return o


def params(opts):
    o, p = _lib(), OParams()
    o.po_params_default(ctypes.byref(p))
    field = {"-M": "match", "-X": "mismatch", "-O": "gap_open1", "-E": "gap_ext1", "-b": "b", "-f": "f"}
    it = iter(opts)
    for x in it:
        if x == "-B":
            p.ab_band = 1
        else:
            setattr(p, field[x], int(next(it)))
    o.po_params_normalize(ctypes.byref(p))
    return p


def run(reads, opts):
    """(status, per read {nodes, edges, sources, hlen, tlen}, consensus): hlen and tlen by
    rank; sources: nodes without in-edges, the source included. status != 0 ends the list at that read."""
    o, p = _lib(), params(opts)
    libc = ctypes.CDLL(None)
    libc.free.argtypes = [ctypes.c_void_p]
    g = o.po_graph_new()
    steps = []
    try:
        for i, r in enumerate(reads):
            q = np.array([("ACGT".find(chr(c)) if chr(c) in "ACGT" else 4) for c in r] or [4], dtype=np.uint8)
            path, plen, score = ctypes.c_void_p(), ctypes.c_int(), ctypes.c_int()
            st = o.po_alignment(g, ctypes.byref(p), q.ctypes.data_as(PU8), len(r), ctypes.byref(path),
                                ctypes.byref(plen), ctypes.byref(score))
            if st != 0:
                return st, steps, b""
            o.po_add_path(g, i, path, plen.value, 1)
            libc.free(path)
            o.po_topsort(g, ctypes.byref(p), 0)
            sz = [ctypes.c_int() for _ in range(5)]
            o.po_graph_sizes(g, *[ctypes.byref(x) for x in sz])
            nn, ni, no, nr, nl = [x.value for x in sz]
            base = np.zeros(nn, np.uint8)
            a = {k: np.zeros(max(n, 1), np.int32) for k, n in (
                ("rank", nn), ("par", nn), ("ind", nn), ("aligned", 5 * nn), ("in_ptr", nn + 1), ("in_id", ni),
                ("in_w", ni), ("out_ptr", nn + 1), ("out_id", no), ("rank_to_id", nr), ("hlen", nl), ("tlen", nl))}
            o.po_graph_export(g, base.ctypes.data_as(PU8), *[x.ctypes.data_as(P32) for x in a.values()])
            steps.append(dict(nodes=nn, edges=ni, sources=int((np.diff(a["in_ptr"][:nn + 1]) == 0).sum()),
                              hlen=a["hlen"], tlen=a["tlen"]))
        n = ctypes.c_int()
        c = o.po_consensus(g, ctypes.byref(n))
        cons = ctypes.string_at(c, n.value)
        libc.free(c)
        return 0, steps, cons
    finally:
        o.po_graph_free(g)
