"""The work that users of this package have it do, as measurable cases.

Every case is one call (or the two calls of the pipeline) of the public entry
points: `pairwise.run` and `phylogeny.run` on a host `Database`, the C ABI on
sequences and matrices that stay on the device, and the serving loop. The
sizes are those of the seeded workloads of `msa_b200.workloads` and of the
usual inputs of a guide-tree step: protein families, short DNA reads, viral
genomes, aligned (gapped) files, and distance matrices of up to some thousand
taxa.

A case is a dict:

    kind    "pipeline"  Database on the host -> scores and tree on the host
            "pairwise"  Database on the host -> scores on the host
            "store"     uploaded store -> scores on the device
            "nj"        matrix on the device or the host -> tree
            "serve"     jobs submitted together to a running server -> scores
    family  how the sequences are made (see `sequences`)
    n, lo, hi, table    number of sequences, their lengths, scoring table
    order   removal order of a tree: "symmetric" or "linear"
    where   an "nj" case's matrix: "device" (int32) or "host" (float32)
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from msa_b200 import _lib, pairwise, phylogeny, runtime
from msa_b200 import workloads as W
from msa_b200.database import Database
from msa_b200.pairwise import DistanceMatrix, ScoringTable
from msa_b200.serve import Server

U8P = ctypes.POINTER(ctypes.c_uint8)
U64P = ctypes.POINTER(ctypes.c_uint64)
TABLES = ("blosum62", "blosum45", "blosum50", "blosum80", "blosum90", "pam250")


def listed() -> list:
    return [
        # The smallest useful run: sixteen proteins from a file to a guide tree.
        dict(name="pipeline protein 16", kind="pipeline", family="iid", n=16, lo=100, hi=300, table="blosum62",
             order="symmetric"),
        # An ordinary protein family with ragged lengths, to a guide tree.
        dict(name="pipeline protein 120", kind="pipeline", family="clades", n=120, lo=80, hi=600, table="blosum62",
             order="symmetric"),
        # A large family of one ancestor, about 500 residues each, kept on the device.
        dict(name="family 1000x500", kind="store", family="clades", n=1000, lo=480, hi=520, table="blosum62"),
        # Many short DNA reads.
        dict(name="reads 3000x150", kind="store", family="dna", n=3000, lo=100, hi=250, table="default"),
        # DNA of very uneven length (log-normal, 200 to 16,000 bases).
        dict(name="uneven dna 1200", kind="store", family="uneven", n=1200, lo=200, hi=16000, table="default"),
        # A set of viral genomes from the host, as in a first look at an outbreak.
        dict(name="viral genomes 50", kind="pairwise", family="dna", n=50, lo=2000, hi=10000, table="default"),
        # A few long genomes of about 30,000 bases.
        dict(name="long genomes 24", kind="store", family="dna", n=24, lo=29000, hi=30500, table="default"),
        # An aligned protein file scored again: '-' in most sequences.
        dict(name="gapped protein 400", kind="store", family="gapped", n=400, lo=450, hi=750, table="blosum62"),
        # The guide tree of 2,000 proteins in clades, its matrix already on the device.
        dict(name="nj 2000", kind="nj", family="clades", n=2000, lo=200, hi=600, table="blosum62",
             order="symmetric", where="device"),
        # A guide tree in the linear removal order from a matrix in host memory.
        dict(name="nj 257 linear host", kind="nj", family="clades", n=257, lo=150, hi=400, table="blosum62",
             order="linear", where="host"),
        # A large guide tree.
        dict(name="nj 5000", kind="nj", family="clades", n=5000, lo=100, hi=250, table="blosum62",
             order="symmetric", where="device"),
        # A burst of all-pairs jobs of mixed sizes at a running server.
        dict(name="serve 24 jobs", kind="serve", family="jobs", n=24, lo=50, hi=2000, table="blosum62"),
    ]


def _log(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    """Another case of the same ranges; its cells stay within the largest listed case's."""
    kind = rng.choice(("pipeline", "family", "reads", "uneven", "genomes", "long", "gapped", "nj", "nj", "serve"))
    order = rng.choice(("symmetric", "symmetric", "linear"))
    if kind == "pipeline":
        lo = _log(rng, 40, 300)
        return dict(kind="pipeline", family=rng.choice(("iid", "clades")), n=_log(rng, 6, 200), lo=lo,
                    hi=lo + _log(rng, 10, 500), table=rng.choice(TABLES), order=order)
    if kind == "family":
        lo = _log(rng, 100, 1000)
        n = min(_log(rng, 100, 1200), int(math.sqrt(5e11) / lo))
        return dict(kind="store", family="clades", n=n, lo=lo, hi=int(lo * rng.uniform(1.02, 1.6)),
                    table=rng.choice(TABLES))
    if kind == "reads":
        lo = _log(rng, 40, 180)
        return dict(kind="store", family="dna", n=_log(rng, 300, 3000), lo=lo, hi=lo + _log(rng, 10, 120),
                    table="default")
    if kind == "uneven":
        return dict(kind="store", family="uneven", n=_log(rng, 100, 1100), lo=200, hi=16000, table="default")
    if kind == "genomes":
        lo = _log(rng, 2000, 6000)
        return dict(kind="pairwise", family="dna", n=_log(rng, 8, 64), lo=lo, hi=lo + _log(rng, 100, 5000),
                    table="default")
    if kind == "long":
        lo = _log(rng, 10000, 30000)
        return dict(kind="store", family="dna", n=_log(rng, 4, 24), lo=lo, hi=lo + _log(rng, 50, 2000),
                    table="default")
    if kind == "gapped":
        lo = _log(rng, 100, 500)
        return dict(kind="store", family="gapped", n=_log(rng, 20, 400), lo=lo, hi=lo + _log(rng, 20, 300),
                    table=rng.choice(("blosum62", "blosum45", "blosum80")))
    if kind == "nj":
        lo = _log(rng, 60, 150)
        return dict(kind="nj", family="clades", n=_log(rng, 5, 4500), lo=lo, hi=lo + _log(rng, 10, 150),
                    table=rng.choice(TABLES), order=order, where=rng.choice(("device", "host")))
    return dict(kind="serve", family="jobs", n=_log(rng, 2, 24), lo=_log(rng, 40, 200), hi=_log(rng, 400, 2000),
                table="blosum62")


# ------------------------------------------------------------------- inputs

def _substituted(rng, seq, rate):
    out = seq.copy()
    m = rng.random(out.shape) < rate
    out[m] = W.AMINO[rng.integers(0, 20, int(m.sum()))]
    return out


def _clades(rng, n, lo, hi):
    """Proteins in clades of 40 under one root: clade ancestors diverge by 40%
    and have a length of their own in [lo, hi]; members diverge by 10 to 30%,
    lose up to 8 residues at either end and hold one insertion or deletion."""
    root = W.AMINO[rng.integers(0, 20, hi + 16)]
    seqs = []
    while len(seqs) < n:
        m = min(40, n - len(seqs))
        anc = _substituted(rng, root, 0.4)[: int(rng.integers(lo, hi + 1)) + 16]
        block = _substituted(rng, np.broadcast_to(anc, (m, len(anc))), rng.uniform(0.1, 0.3, (m, 1)))
        for row in block:
            a, b, at, k = (int(v) for v in rng.integers(0, (8, 8, len(row) - 16, 7)))
            if k & 1:
                row = np.concatenate([row[:at], row[at + k:]])
            elif k:
                row = np.concatenate([row[:at], W.AMINO[rng.integers(0, 20, k)], row[at:]])
            seqs.append(row[a: len(row) - b])
    return seqs


def sequences(family: str, rng, n: int, lo: int, hi: int) -> list:
    """`n` sequences of letters: "iid" (independent proteins), "clades" (related
    proteins), "dna" (bases with 1% N, uniform lengths), "uneven" (the same
    with log-normal lengths), "gapped" (related proteins with '-' runs, as rows
    of an alignment)."""
    if family == "iid":
        return [W.AMINO[rng.integers(0, 20, int(L))] for L in rng.integers(lo, hi + 1, n)]
    if family == "clades":
        return _clades(rng, n, lo, hi)
    if family == "gapped":
        seqs = _clades(rng, n, lo, hi)
        for s in seqs:
            for _ in range(int(rng.integers(0, 6))):
                at = int(rng.integers(0, len(s) - 1))
                s[at: at + int(rng.integers(1, 12))] = ord("-")
        return seqs
    if family == "uneven":
        lens = np.clip(W.c3_lengths(rng, n), lo, hi)
    else:
        lens = rng.integers(lo, hi + 1, n)
    seqs = []
    for L in lens:
        s = W.DNA[rng.integers(0, 4, int(L))]
        s[rng.random(int(L)) < 0.01] = ord("N")
        seqs.append(s)
    return seqs


def _rng(seed):
    return np.random.Generator(np.random.PCG64(seed))


def _sequences_of(case, seed):
    return sequences(case["family"], _rng(seed), case["n"], case["lo"], case["hi"])


class Store:
    """An uploaded sequence store and a device triangle for its scores."""

    def __init__(self, seqs, table: str):
        self.ctx = runtime.context(0)
        flat, offs, lens = W.Workload("case", seqs, table, 0).flat_units()
        self.n = len(lens)
        self.table = ScoringTable(table)
        self.handle = ctypes.c_uint64()
        _lib.check(_lib.lib().msa_seqs_upload(self.ctx.handle, flat.ctypes.data_as(U8P), offs.ctypes.data_as(U64P),
                                              lens.ctypes.data_as(U64P), self.n, ctypes.byref(self.handle)),
                   self.ctx.handle)
        self.out = torch.empty(self.n * (self.n - 1) // 2, dtype=torch.int32, device="cuda")

    def score(self):
        _lib.check(_lib.lib().msa_nw_all_pairs(self.ctx.handle, self.handle.value, ctypes.byref(self.table._t),
                                               _lib.MSA_NW_AUTO, ctypes.c_void_p(self.out.data_ptr()), 1),
                   self.ctx.handle)
        return self.out

    def __del__(self):
        if getattr(self, "handle", None):
            _lib.lib().msa_seqs_release(self.ctx.handle, self.handle.value)


_server = None


def _running_server() -> Server:
    """The program's one server on the device."""
    global _server
    if _server is None:
        _server = Server(device=0)
    return _server


def _job_size(k: int) -> int:
    """Sequences of a burst's k-th job: 8 to 319, spread evenly and out of order."""
    return 8 + k * 197 % 312


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("pipeline", "pairwise"):
        db = Database()
        db.add([(f"seq{k}", bytes(s)) for k, s in enumerate(_sequences_of(case, seed))])
        return kind, db, ScoringTable(case["table"]), case.get("order")
    if kind == "store":
        return kind, Store(_sequences_of(case, seed), case["table"])
    if kind == "nj":
        store = Store(_sequences_of(case, seed), case["table"])
        tri = store.score()
        order = _lib.MSA_NJ_LINEAR if case["order"] == "linear" else _lib.MSA_NJ_SYMMETRIC
        if case["where"] == "host":
            return kind, DistanceMatrix(tri.cpu().numpy(), store.n), case["order"], None
        return kind, tri, order, store.n
    rng = _rng(seed)
    jobs = []
    for k in range(case["n"]):
        protein, n = k % 2 == 0, _job_size(k)
        seqs = sequences("iid" if protein else "dna", rng, n, case["lo"], case["hi"])
        table = case["table"] if protein else "default"
        jobs.append((W.Workload("job", seqs, table, 0).flat_units(), ScoringTable(table)))
    return kind, _running_server(), jobs


# ------------------------------------------------------------------ one pass

def _tree(t):
    return {"parent": t.parent, "child0": t.child0, "child1": t.child1, "distance": t.distance, "level": t.level}


NODE = np.dtype([("parent", "<u4"), ("c0", "<u4"), ("c1", "<u4"), ("distance", "<f4"), ("level", "<u4")])


def run(state):
    kind = state[0]
    if kind == "pipeline":
        _, db, table, order = state
        m = pairwise.run(db, table)
        tree = phylogeny.run(m, db.count, "linear" if order == "linear" else "default")
        return {"scores": m.int_scores, "tree": _tree(tree)}
    if kind == "pairwise":
        _, db, table, _ = state
        return {"scores": pairwise.run(db, table).int_scores}
    if kind == "store":
        return {"scores": state[1].score()}
    if kind == "nj":
        _, tri, order, n = state
        if n is None:
            return {"tree": _tree(phylogeny.run(tri, algorithm="linear" if order == "linear" else "default"))}
        ctx = runtime.context(0)
        nodes = (_lib.MsaOtu * (2 * n - 1))()
        _lib.check(_lib.lib().msa_nj_order(ctx.handle, ctypes.c_void_p(tri.data_ptr()), _lib.MSA_TRI_I32_DEVICE, n,
                                           order, nodes), ctx.handle)
        a = np.frombuffer(nodes, dtype=NODE)
        return {"tree": {"parent": a["parent"], "child0": a["c0"], "child1": a["c1"], "distance": a["distance"],
                         "level": a["level"]}}
    _, server, jobs = state
    ids = [server.submit(*units, table) for units, table in jobs]
    return {"scores": [server.wait(i)[0] for i in ids]}


# ------------------------------------------------- what a pass cannot do without

def _mean_cells(case) -> float:
    """Expected cells of all pairs: sum over pairs of L_i * L_j."""
    n, lo, hi = case["n"], case["lo"], case["hi"]
    if case["family"] == "uneven":
        mean = 1500.0 * math.exp(0.75 ** 2 / 2)
    else:
        mean = (lo + hi) / 2
    return n * (n - 1) / 2 * mean * mean


def work(case) -> dict:
    """One addition and two maxima per cell; sequences read and scores written
    once. A tree: its matrix read once; one Q (a multiplication and two
    subtractions) per pair for the first join, and six operations for every
    distance and row sum that a join replaces."""
    n = case["n"]
    pairs = n * (n - 1) / 2
    tree = {"bytes": 4 * pairs + 20 * (2 * n - 1), "flops": 3 * pairs + 6 * pairs}
    if case["kind"] == "nj":
        return tree
    if case["kind"] == "serve":
        sizes, mean = [_job_size(k) for k in range(n)], (case["lo"] + case["hi"]) / 2
        pairs = sum(m * (m - 1) / 2 for m in sizes)
        return {"bytes": sum(sizes) * mean + 4 * pairs, "flops": 3 * pairs * mean * mean}
    mean = math.sqrt(_mean_cells(case) / max(pairs, 1))
    got = {"bytes": n * mean + 4 * pairs, "flops": 3 * _mean_cells(case)}
    if case["kind"] == "pipeline":
        got = {k: got[k] + tree[k] for k in got}
    return got


# --------------------------------------------------------------- in 64 bits

def _exact_scores(seqs, name):
    """Needleman-Wunsch scores of all pairs, row-major lower triangle. One row
    of every pair's matrix at a time: max(diagonal + s, up - g), then the
    left-to-right maximum with a linear gap as a running maximum of v + g*j."""
    table = ScoringTable(name)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    t = torch.tensor(table.matrix(), dtype=torch.int64, device=dev)
    g = int(table.penalty)
    n, L = len(seqs), max(len(s) for s in seqs)
    units = torch.zeros(n, L, dtype=torch.int64)
    for k, s in enumerate(seqs):
        units[k, : len(s)] = torch.from_numpy(W.letters_to_units(s).astype(np.int64))
    units = units.to(dev)
    lens = torch.tensor([len(s) for s in seqs], device=dev)
    ii, jj = torch.tril_indices(n, n, -1, device=dev)
    out = torch.empty(len(ii), dtype=torch.int64, device=dev)
    gj = g * torch.arange(L + 1, device=dev)
    for p in range(0, len(ii), 4096):
        a, b = ii[p: p + 4096], jj[p: p + 4096]
        h = (-gj).expand(len(a), -1).clone()
        got = torch.empty(len(a), dtype=torch.int64, device=dev)
        for i in range(int(lens[a].max())):
            s = t[units[a, i]].gather(1, units[b])
            v = h - g
            v[:, 1:] = torch.maximum(v[:, 1:], h[:, :-1] + s)
            h = torch.cummax(v + gj, 1).values - gj
            done = lens[a] == i + 1
            got[done] = h[done].gather(1, lens[b][done, None])[:, 0]
        out[p: p + 4096] = got
    return out.cpu().numpy()


def exact(case, seed):
    """Scores in 64-bit integers where that is quick. Trees have no such value:
    which pair a join takes and the lengths that follow are defined by the
    order of the reference's 32-bit operations (the last join divides by zero),
    so every field of theirs is given as None. GAP units are scored through the
    reference's table storage, which plain code does not have."""
    if case["kind"] not in ("pipeline", "store", "pairwise") or case["family"] == "gapped" or _mean_cells(case) > 1e10:
        return None
    got = {"scores": _exact_scores(_sequences_of(case, seed), case["table"])}
    if case["kind"] == "pipeline":
        got["tree"] = {"parent": None, "child0": None, "child1": None, "distance": None, "level": None}
    return got
