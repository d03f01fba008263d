"""Performance cases of the all-pairs TN93 engine: what is timed when a change to it is judged.

Every case goes through the package's public entry points, as a user's program calls them:

  run       an alignment in host memory -> Engine.upload, Engine.run (text to a sink, in order), Engine.free
  resident  an alignment already in HBM -> Engine.run_to_device (the distance file stays in HBM)
  fasta     a FASTA file's bytes        -> Engine.upload_fasta, Engine.run, Engine.free
  batch     many alignments in one call -> Engine.batch_run
  serve     a batch of queries against a resident reference -> ResidentReference.batch

Alignments have the shapes of swifttn93_b200/synth.py's workloads, drawn here on the GPU so that making them is quick:
"hiv" (a background of about 6% divergence with transmission clusters, 1% two-fold codes with 4% of the sequences at
3-5%, a few N, gap runs, ragged ends), "real" (the code frequencies of the HIV-1 pol set in tests/golden: 0.5% two-fold
codes, 0.1% N, a trace of three-fold codes, and some copy numbers), "long" (0.1% star-like divergence, long N runs).
"""
from __future__ import annotations

import math

import numpy as np
import torch

from swifttn93_b200 import Engine, Fasta, HostAlignment, Options, ResidentReference

ALPHABET = np.frombuffer(b"ACGTURYSWKMBDHVN?-", dtype=np.uint8)
TWOFOLD = (5, 9, 10, 6, 7, 8)  # R K M Y S W
N, GAP = 15, 17
ALL = 1000.0  # a threshold that reports every pair


def listed():
    hiv = dict(data="hiv", g=0.05, l=500, format="csv")
    return [
        # one small outbreak: latency and launches are all there is to it
        dict(name="tiny_run_50x900", path="run", n=50, L=900, mode="resolve", t=0.015, data="hiv", g=0.05, l=100, format="csv"),
        # a study of the size that also runs on a laptop (the plain 500 x 1,300 workload's flags)
        dict(name="small_run_500x1300", path="run", n=500, L=1300, mode="resolve", t=0.015, **hiv),
        # HIV-TRACE's call on a national set: few links reported, so the text is small
        dict(name="network_run_6700x1500", path="run", n=6700, L=1500, mode="resolve", t=0.015, **hiv),
        # every distance delivered to the host, odd sizes, column numbers instead of names
        dict(name="alltext_run_1801x1203", path="run", n=1801, L=1203, mode="average", t=ALL, data="hiv", g=1.0, l=100, format="csvn"),
        # the benchmark set in HBM, every pair written, in its three ambiguity modes
        dict(name="all_resolve_6700x1500", path="resident", n=6700, L=1500, mode="resolve", t=ALL, **hiv),
        dict(name="all_average_6700x1500", path="resident", n=6700, L=1500, mode="average", t=ALL, **hiv),
        dict(name="all_gapmm_6700x1500", path="resident", n=6700, L=1500, mode="gapmm", t=ALL, **hiv),
        # genome-length alignments with N runs (SARS-CoV-2-like), close pairs only
        dict(name="long_run_2000x29900", path="run", n=2000, L=29900, mode="resolve", t=0.0001, data="long", g=0.05, l=5000, format="csvn"),
        # a cohort's many alignments of uneven size in one call, modes mixed
        dict(name="batch_24", path="batch", k=24, n=2000, L=3000, data="hiv", g=0.05, l=500, format="csv"),
        # one request against a resident reference (latency), and a saturated service's batch (throughput)
        dict(name="serve_one_30000", path="serve", k=1, q=32, n=30000, L=1500, mode="resolve", t=0.015, **hiv),
        dict(name="serve_batch_30000", path="serve", k=40, q=32, n=30000, L=1500, mode="resolve", t=0.015, **hiv),
        # a file straight from disk, 60-column lines, real code frequencies with copy numbers
        dict(name="fasta_3001x1065", path="fasta", n=3001, L=1065, mode="resolve", t=0.02, data="real", g=0.05, l=500, format="csv"),
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    path = rng.choice(("run", "run", "resident", "resident", "fasta", "batch", "serve"))
    mode = rng.choice(("resolve", "resolve", "average", "gapmm", "skip", "RY"))
    opts = dict(mode=mode, g=rng.choice((0.05, 0.015, 1.0)), l=rng.choice((100, 500)), format=rng.choice(("csv", "csv", "csvn")))
    if path == "serve":
        return dict(path=path, k=_log(rng, 1, 40), q=_log(rng, 4, 32), n=_log(rng, 2000, 30000), L=rng.randint(700, 1500),
                    data="hiv", t=rng.uniform(0.005, 0.02), **opts)
    if path == "batch":
        return dict(path=path, k=rng.randint(4, 24), n=_log(rng, 200, 2000), L=rng.randint(1000, 3000), data="hiv",
                    g=opts["g"], l=opts["l"], format=opts["format"])
    if path == "run" and rng.random() < 0.3:
        opts["l"] = 5000
        return dict(path=path, n=_log(rng, 60, 1400), L=rng.randint(9000, 29900), data="long",
                    t=rng.choice((0.0001, 0.0005)), **opts)
    data = "real" if path == "fasta" else rng.choice(("hiv", "real"))
    L = rng.randint(500, 3000)
    if path == "resident":
        n = min(_log(rng, 300, 6700), int(math.sqrt(2 * 22.4e6 * 1500 / max(L, 1500))))
        return dict(path=path, n=n, L=L, t=rng.choice((0.015, ALL, ALL)), data=data, **opts)
    t = rng.choice((0.015, 0.03, ALL))
    return dict(path=path, n=_log(rng, 40, 2000 if t == ALL else 4000), L=L, t=t, data=data, **opts)


# ---- inputs -----------------------------------------------------------------------------------------------------
class _Random:
    """Draws on the GPU (on the CPU where there is none), from the seed alone."""

    def __init__(self, seed):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.g = torch.Generator(device=self.dev)
        self.g.manual_seed(seed)

    def rand(self, *shape):
        return torch.rand(shape, generator=self.g, device=self.dev)

    def randint(self, lo, hi, *shape):
        return torch.randint(lo, hi, shape, generator=self.g, device=self.dev)


def _mutate(R, seqs, rate):
    """Substitutions at `rate` per site (a number or one per sequence): 85% transitions (A<->G, C<->T)."""
    u = R.rand(*seqs.shape)
    rate = torch.as_tensor(rate, device=R.dev, dtype=torch.float32).reshape(-1, 1)
    v = R.rand(*seqs.shape)
    to = torch.where(v < 0.85, 2, torch.where(v < 0.925, 1, 3)).to(torch.uint8)
    return torch.where(u < rate, seqs ^ to, seqs)


def _runs(R, seqs, mean, lo, hi, code):
    """Runs of `code`, a Poisson(mean) number per sequence, of length lo..hi."""
    n, L = seqs.shape
    num = torch.poisson(torch.full((n,), mean, device=R.dev), generator=R.g).to(torch.int64)
    col = torch.arange(L, device=R.dev)
    for k in range(int(num.max()) if n else 0):
        st = (R.rand(n, 1) * L).long()
        ln = R.randint(lo, hi + 1, n, 1)
        on = (col >= st) & (col < st + ln) & (num > k)[:, None]
        seqs = torch.where(on, code, seqs)
    return seqs


def _ends(R, seqs, most, code):
    n, L = seqs.shape
    col = torch.arange(L, device=R.dev)
    a, b = R.randint(0, most + 1, n, 1), R.randint(0, most + 1, n, 1)
    return torch.where((col < a) | (col >= L - b), code, seqs).to(torch.uint8)


def _codes(R, n, L, data):
    """An alignment's codes on the device, uint8 [n, L]."""
    pi = torch.tensor((0.30, 0.18, 0.20, 0.32) if data == "long" else (0.39, 0.17, 0.23, 0.21), device=R.dev)
    root = torch.multinomial(pi, L, replacement=True, generator=R.g).to(torch.uint8)[None]
    two = torch.tensor(TWOFOLD, dtype=torch.uint8, device=R.dev)
    if data == "long":
        s = _mutate(R, root.expand(n, L), -0.0005 * torch.log(R.rand(n) + 1e-9))
        s = torch.where(R.rand(n, L) < 0.0002, two[R.randint(0, 6, n, L)], s)
        return _ends(R, _runs(R, s, 3.0, 50, 400, N), 300, N)
    # a shallow tree: 6 clades, 60 lineages, then one branch per background sequence; clusters hang on some of them
    clade = _mutate(R, root.expand(6, L), 0.009)
    line = _mutate(R, clade[R.randint(0, 6, 60)], 0.008)
    s = _mutate(R, line[R.randint(0, 60, n)], 0.015)
    at = 0
    for k in range(min(40, n // 12)):
        size = min(5 + (k * 37) % 56, n // 2 - at)
        if size < 5:
            break
        s[at:at + size] = _mutate(R, s[at:at + 1].expand(size, L), 0.001 + 0.005 * ((k * 13) % 40) / 40)
        at += size
    s = s[torch.randperm(n, generator=R.g, device=R.dev)]
    if data == "real":
        rate, three, nn = torch.full((n, 1), 0.005, device=R.dev), 3e-5, 0.001
    else:
        rate = torch.where(R.rand(n, 1) < 0.04, 0.03 + 0.02 * R.rand(n, 1), torch.full((n, 1), 0.01, device=R.dev))
        three, nn = 0.0, 0.0005
    pick = R.randint(0, 6, n, L)
    if data == "real":  # transitions' codes (R, Y) are most of them
        pick = torch.where(R.rand(n, L) < 0.7, 3 * R.randint(0, 2, n, L), pick)
    s = torch.where(R.rand(n, L) < rate, two[pick], s)
    if three:
        s = torch.where(R.rand(n, L) < three, (11 + R.randint(0, 4, n, L)).to(torch.uint8), s)
    s = torch.where(R.rand(n, L) < nn, N, s)
    return _ends(R, _runs(R, s, 0.3, 1, 30, GAP), min(80, L // 8), GAP)


def _names(n, data, seed):
    if data == "real":  # accession-like, of uneven length; some carry a copy number
        return [f"{'ABCFG'[i % 5]}.{i * 7919 % 1000}.PZ{seed % 97}{i}.1" + (f":{2 + i % 3}" if i % 50 == 7 else "") for i in range(n)]
    return [f"{data}_{seed % 97}_{i:06d}" for i in range(n)]


def _copies(n, data):
    return np.array([2 + i % 3 if data == "real" and i % 50 == 7 else 1 for i in range(n)], dtype=np.int64)


def _fasta(names, codes, wrap):
    text = ALPHABET[codes]
    out = []
    for name, row in zip(names, text):
        out.append(b">" + name.encode() + b"\n")
        s = row.tobytes()
        out.extend(s[k:k + wrap] + b"\n" for k in range(0, len(s), wrap))
    return b"".join(out)


def _options(c, **more):
    return Options(**{**dict(threshold=c.get("t", 0.015), mode=c.get("mode", "resolve"), resolve_fraction=c["g"],
                             min_overlap=c["l"], format=c["format"]), **more})


def _batch(c, seed):
    """The batch's alignments: (codes on the device, Options) each; lengths, sizes, modes and thresholds uneven."""
    R, rng, out = _Random(seed), np.random.default_rng(seed), []
    sizes = np.exp(np.linspace(math.log(50), math.log(c["n"]), c["k"])).round().astype(int)
    for k in rng.permutation(c["k"]):
        L = int(c["L"] * (0.3 + 0.7 * ((k * 11) % c["k"]) / c["k"]))
        out.append((_codes(R, int(sizes[k]), L, c["data"]),
                    _options(c, mode=("resolve", "average", "gapmm")[k % 3], threshold=float(rng.uniform(0.005, 0.02)))))
    return out


def _serve(c, seed):
    """The reference's codes and each query's, on the device: queries derive from reference sequences at 0.5-3%."""
    R, rng = _Random(seed), np.random.default_rng(seed)
    ref = _codes(R, c["n"], c["L"], c["data"])
    # sizes around the mean c["q"] with a long tail, the same total for every seed
    w = np.linspace(0.2, 1.8, c["k"]) if c["k"] > 1 else np.ones(1)
    sizes = np.maximum(1, (w / w.mean() * c["q"]).round().astype(int))
    rng.shuffle(sizes)
    total = int(sizes.sum())
    src = ref[R.randint(0, c["n"], total)]
    s = torch.where(src < 4, _mutate(R, src & 3, 0.005 + 0.025 * R.rand(total)), src)
    two = torch.tensor(TWOFOLD, dtype=torch.uint8, device=R.dev)
    s = torch.where((R.rand(total, c["L"]) < 0.01) & (s < 4), two[R.randint(0, 6, total, c["L"])], s)
    return ref, list(torch.split(s, sizes.tolist()))


_engine = None


def _the_engine():
    """The program's one engine context, kept from job to job."""
    global _engine
    if _engine is None:
        _engine = Engine()
    return _engine


class _Resident:
    """A set in HBM, given back when the program lets go of it."""

    def __init__(self, engine, alignment):
        self.engine, self.set = engine, engine.upload(alignment)

    def __del__(self):
        if self.engine.ctx:
            self.engine.free(self.set)


def _room(pairs, n, c):
    """Bytes that hold the program's copy of the text: every pair where all (or many) are reported, else 100 links a
    sequence; 52 bytes a line with names, 26 with column numbers."""
    lines = pairs if c.get("t", 0.0) >= ALL or c["data"] == "long" else min(pairs, 100 * n + 1000)
    return int(lines * (52 if c["format"] == "csv" else 26)) + 64


class _File:
    """Where the program collects the text: a buffer of its own, filled in order."""

    def __init__(self, size):
        self.buf, self.at = np.zeros(size, dtype=np.uint8), 0

    def write(self, text):
        self.buf[self.at:self.at + len(text)] = np.frombuffer(text, dtype=np.uint8)
        self.at += len(text)


def prepare(case, seed):
    c, eng = case, _the_engine()
    if c["path"] == "batch":
        work = _batch(c, seed)
        sizes = [len(a) for a, _ in work]
        alns = [HostAlignment(a.cpu().numpy(), _names(len(a), "b%d" % k, seed)) for k, (a, _) in enumerate(work)]
        return dict(c=c, eng=eng, alns=alns, opts=[o for _, o in work],
                    file=_File(sum(_room(n * (n - 1) // 2, n, c) for n in sizes)))
    if c["path"] == "serve":
        ref, queries = _serve(c, seed)
        total = sum(len(q) for q in queries)
        ref = Fasta(_fasta(_names(c["n"], "ref", seed), ref.cpu().numpy(), c["L"]))
        server = ResidentReference(eng, ref, _options(c), max_batch_sequences=(total + 63) // 64 * 64, max_batch_queries=c["k"])
        return dict(c=c, eng=eng, server=server, file=_File(_room(c["n"] * total, 20 * total, c)),
                    queries=[Fasta(_fasta(_names(len(q), "q%d" % k, seed), q.cpu().numpy(), c["L"])) for k, q in enumerate(queries)])
    codes = _codes(_Random(seed), c["n"], c["L"], c["data"]).cpu().numpy()
    names = _names(c["n"], c["data"], seed)
    room = _room(c["n"] * (c["n"] - 1) // 2, c["n"], c)
    if c["path"] == "fasta":
        return dict(c=c, eng=eng, fasta=_fasta(names, codes, 60), opts=_options(c), file=_File(room))
    aln = HostAlignment(codes, names, _copies(c["n"], c["data"]))
    if c["path"] == "resident":
        return dict(c=c, eng=eng, set=_Resident(eng, aln), opts=_options(c), stream=torch.cuda.ExternalStream(eng.stream),
                    text=torch.zeros(room, dtype=torch.uint8, device="cuda"))
    return dict(c=c, eng=eng, aln=aln, opts=_options(c), file=_File(room))


# ---- one pass ---------------------------------------------------------------------------------------------------
def _one(text, s):
    return dict(text=text, links=s.links, skipped=s.skipped, hist=s.hist[0].astype(np.int64), max=s.max[0], mean=s.mean[0],
                weighted=s.weighted[0])


def _many(file, results):
    file.at = 0
    for body, _ in results:
        file.write(body)
    ss = [s for _, s in results]
    return dict(text=file.buf, length=np.array([len(b) for b, _ in results]), links=np.array([s.links for s in ss]),
                skipped=np.array([s.skipped for s in ss]), hist=np.stack([s.hist[0] for s in ss]).astype(np.int64),
                max=np.array([s.max[0] for s in ss]), mean=np.array([s.mean[0] for s in ss]),
                weighted=np.array([s.weighted[0] for s in ss]))


class _DeviceBytes:
    def __init__(self, ptr, n):
        self.__cuda_array_interface__ = dict(shape=(n,), typestr="|u1", data=(ptr, False), version=3)


def run(state):
    c, eng = state["c"], state["eng"]
    if c["path"] == "resident":
        ptr, n, s = eng.run_to_device(state["set"].set, state["opts"])
        if n:  # the engine's next run reuses its buffer: the program copies the text to its own, in the engine's stream
            with torch.cuda.stream(state["stream"]):
                state["text"][:n].copy_(torch.as_tensor(_DeviceBytes(ptr, n), device="cuda"))
        return _one(state["text"], s)
    if c["path"] == "batch":
        return _many(state["file"], eng.batch_run(state["alns"], state["opts"]))
    if c["path"] == "serve":
        return _many(state["file"], state["server"].batch(state["queries"]))
    file = state["file"]
    file.at = 0
    s = eng.upload_fasta(state["fasta"]) if c["path"] == "fasta" else eng.upload(state["aln"])
    _, summary = eng.run(s, state["opts"], sink=file.write)
    eng.free(s)
    return _one(file.buf, summary)


def work(case):
    """Codes and names read once; the text of a run that reports every pair (about 36 bytes a line with names, 20 with
    column numbers) written once; per pair the 4 x 4 table of base combinations over the columns (16 multiply-adds each)."""
    c = case
    if c["path"] == "batch":
        sizes = np.exp(np.linspace(math.log(50), math.log(c["n"]), c["k"])).round()
        lens = [int(c["L"] * (0.3 + 0.7 * ((k * 11) % c["k"]) / c["k"])) for k in range(c["k"])]
        return dict(bytes=float(sum(n * (L + 15) for n, L in zip(sizes, lens))),
                    flops=float(sum(16 * n * (n - 1) * L for n, L in zip(sizes, lens))))
    if c["path"] == "serve":
        q = c["k"] * c["q"]
        return dict(bytes=float((c["n"] + q) * (c["L"] + 15)), flops=32.0 * c["n"] * q * c["L"])
    pairs = c["n"] * (c["n"] - 1) / 2
    line = (36 if c["format"] == "csv" else 20) if c["t"] >= ALL else 0
    return dict(bytes=c["n"] * (c["L"] + 15.0) + pairs * line, flops=32.0 * pairs * c["L"])


# ---- the same in 64 bits ----------------------------------------------------------------------------------------
BASES = [{0}, {1}, {2}, {3}, {3}, {0, 2}, {1, 3}, {1, 2}, {0, 3}, {2, 3}, {0, 1}, {1, 2, 3}, {0, 2, 3}, {0, 1, 3}, {0, 1, 2},
         {0, 1, 2, 3}, {0, 1, 2, 3}, set()]


def _site(a, b, mode):
    """tn93's contribution of one site with codes a and b: {(x, y): weight}, and whether it resolved an ambiguity."""
    if GAP in (a, b):
        if mode != "gapmm" or a == b:
            return {}, 0
        a, b = (N if a == GAP else a), (N if b == GAP else b)
    A, B = BASES[a], BASES[b]
    if a < 4 and b < 4:
        return {(a, b): 1.0}, 0
    if mode == "skip":
        return {}, 0
    resolves = mode == "resolve" or mode == "RY"
    listed_ = [x < 4 or mode == "resolve" or (mode == "RY" and x in (5, 6)) for x in (a, b)]
    if resolves and all(listed_):
        if (a < 4 or b < 4) and A & B:
            x = min(A & B)
            return {(x, x): 1.0}, 1
        if a >= 4 and b >= 4:
            both = A & B
            if both:
                return {(x, x): 1.0 / len(both) for x in both}, 1
            return {(x, y): 1.0 / len(A) / len(B) for x in A for y in B}, 1
    return {(x, y): 1.0 / len(A) / len(B) for x in A for y in B}, 0


def _distances(F, tot):
    """The TN93 distance from the 4 x 4 tables F (16 arrays of doubles), K2P where a base is absent."""
    nf = [sum(F[4 * x + y] + F[4 * y + x] for y in range(4)) for x in range(4)]
    s = nf[0] + nf[1] + nf[2] + nf[3]
    f = [x / s for x in nf]
    ag, ct = (F[2] + F[8]) / tot, (F[7] + F[13]) / tot
    tv = 1 - (F[0] + F[5] + F[10] + F[15]) / tot - ag - ct
    r, y = f[0] + f[2], f[1] + f[3]
    k1, k2 = 2 * f[0] * f[2] / r, 2 * f[1] * f[3] / y
    k3 = 2 * (r * y - f[0] * f[2] * y / r - f[1] * f[3] * r / y)
    a1, a2, a3 = 1 - ag / k1 - tv / (2 * r), 1 - ct / k2 - tv / (2 * y), 1 - tv / (2 * r * y)
    d = -k1 * torch.log(a1) - k2 * torch.log(a2) - k3 * torch.log(a3)
    d = torch.where((a1 > 0) & (a2 > 0) & (a3 > 0), d, 1000.0)
    b1, b2 = 1 - 2 * (ag + ct) - tv, 1 - 2 * tv
    k2p = torch.where((b1 > 0) & (b2 > 0), -0.5 * torch.log(b1) - 0.25 * torch.log(b2), 1000.0)
    absent = (nf[0] == 0) | (nf[1] == 0) | (nf[2] == 0) | (nf[3] == 0)
    return torch.where(absent, k2p, d).clamp(min=0)


def _sums(rows, cols, w_rows, w_cols, opts, triangle):
    """Per column: the largest distance, the sum of distance x weight and the sum of weights over its counted pairs."""
    mode, g, dev = opts.mode, opts.resolve_fraction, rows.device
    present = sorted(set(torch.unique(rows).tolist()) | set(torch.unique(cols).tolist()))
    X = {c: (cols == c).float() for c in present}
    mx, mean, wsum = (torch.zeros(len(cols), dtype=torch.float64, device=dev) for _ in range(3))
    step = max(1, int(12e6 // max(1, len(cols))))
    for r0 in range(0, len(rows), step):
        blk = rows[r0:r0 + step]
        shape = (len(blk), len(cols))
        fall = mode in ("resolve", "RY") and g < 1.0
        F = [torch.zeros(shape, dtype=torch.float64, device=dev) for _ in range(16)]
        V = [torch.zeros(shape, dtype=torch.float64, device=dev) for _ in range(16)] if fall else None
        amb = torch.zeros(shape, dtype=torch.float64, device=dev)
        for a in present:
            Y = (blk == a).float()
            if not bool(Y.any()):
                continue
            for b in present:
                cells, resolved = _site(a, b, mode)
                averaged = _site(a, b, "average")[0] if fall else {}
                if not cells and not averaged:
                    continue
                num = (Y @ X[b].T).double()  # whole numbers below 2^24: exact
                for (x, y), v in cells.items():
                    F[4 * x + y].add_(num, alpha=v)
                for (x, y), v in averaged.items():
                    V[4 * x + y].add_(num, alpha=v)
                if resolved:
                    amb += num
        tot = sum(F)
        counted = tot > opts.min_overlap
        if fall:
            over = counted & (tot * g <= amb)
            F = [torch.where(over, v, f) for v, f in zip(V, F)]
            tot = sum(F)
            counted &= tot > opts.min_overlap
        if triangle:
            counted &= torch.arange(len(cols), device=dev)[None] > (r0 + torch.arange(len(blk), device=dev))[:, None]
        w = w_rows[r0:r0 + step, None] * w_cols[None] * counted
        d = torch.where(counted, _distances(F, tot), 0.0)
        mx = torch.maximum(mx, d.max(dim=0).values)
        mean += (d * w).sum(dim=0)
        wsum += w.sum(dim=0)
    return mx, mean, wsum


def exact(case, seed):
    c = case
    whole = dict(text=None, length=None, links=None, skipped=None, hist=None)
    if c["path"] == "batch":
        got = []
        for a, o in _batch(c, seed):
            w = torch.ones(len(a), dtype=torch.float64, device=a.device)
            m, s, t = _sums(a, a, w, w, o, True)
            got.append((float(m.max()), float(s.sum()), float(t.sum())))
        got = np.array(got)
        return dict(whole, max=got[:, 0], mean=got[:, 1], weighted=got[:, 2])
    if c["path"] == "serve":
        ref, queries = _serve(c, seed)
        q = torch.cat(queries)
        one = torch.ones(len(ref), dtype=torch.float64, device=ref.device)
        m, s, t = _sums(ref, q, one, one.new_ones(len(q)), _options(c), False)
        parts = [x.split([len(k) for k in queries]) for x in (m, s, t)]
        return dict(whole, max=np.array([float(x.max()) for x in parts[0]]), mean=np.array([float(x.sum()) for x in parts[1]]),
                    weighted=np.array([float(x.sum()) for x in parts[2]]))
    codes = _codes(_Random(seed), c["n"], c["L"], c["data"])
    w = torch.as_tensor(_copies(c["n"], c["data"]), dtype=torch.float64, device=codes.device)
    m, s, t = _sums(codes, codes, w, w, _options(c), True)
    own = float((w * (w - 1) / 2).sum())  # copies of one sequence: pairs at distance 0
    return dict(whole, max=float(m.max()), mean=float(s.sum()), weighted=float(t.sum()) + own)
