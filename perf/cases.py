"""The work a user of this framework has it do, as cases that can be timed and checked.

Every case is one call of a public entry point on reads drawn like the benchmark's (uniform random
references, about 1.6 events per k-mer, an anchor every 50 positions):

* "single"    getAlignedPairsUsingAnchors: one read per call, in FP64
* "align"     align_batch from host data: planning, upload, kernels, download
* "resident"  run + download of a batch planned and uploaded before, as a program does that keeps
              several batches in flight and overlaps those steps with another batch's kernels
* "noalloc"   align_batch_noalloc: a batch without device allocations
* "em"        getExpectationsBatch: the expectations of an EM iteration

Machines: "acgt" (6-mer ACGT, Gaussian), "acegt" (6-mer ACEGT, Gaussian), "hdp" (6-mer ACEGT with
2000-point HDP densities).  With "sites" the reference has an X (C or E) at its CCWGG motifs.

`exact` gives the same outputs in 64 bits from numpy alone.
"""
import ctypes
import math
import os
import tempfile

import numpy as np

from signalalign_b200 import api, synth

_PAIR_FIELDS = 4   # score, x, y, k-mer: 64-bit integers


def listed():
    return [
        # the smallest call: one short read, as signalMachine aligns one strand (1,000 bp: the
        # benchmark's first configuration)
        dict(name="single_1kb", kind="single", machine="acgt", reads=1, shortest=1000, longest=1000, expansion=50),
        # a methylation call on one read: C or E at every CCWGG site, two paths over the sites
        dict(name="single_sites_3kb", kind="single", machine="acegt", sites=True, reads=1, shortest=3000,
             longest=3000, expansion=50),
        # one read handed to the batched form: latency of a whole call
        dict(name="align_1_read", kind="align", machine="acgt", reads=1, shortest=700, longest=700, expansion=50),
        # an ordinary small batch, whole call, the band of the library's default parameters
        dict(name="align_16_reads", kind="align", machine="acgt", reads=16, shortest=1000, longest=4000,
             expansion=20),
        # a batch that fills the GPU, the headline benchmark's machine and band with long reads
        dict(name="batch_30_long", kind="resident", machine="acgt", reads=30, shortest=8000, longest=30000,
             expansion=50),
        # a batch of middling reads as the serving loop forms them
        dict(name="batch_8_served", kind="resident", machine="acgt", reads=8, shortest=8000, longest=12000,
             expansion=50),
        # methylation with the HDP machine (5 to 15 kb, as in the benchmark's second configuration)
        dict(name="batch_12_hdp", kind="resident", machine="hdp", reads=12, shortest=5000, longest=15000,
             expansion=50),
        # a wide band, for reads whose anchors are doubtful
        dict(name="batch_6_wide", kind="resident", machine="acgt", reads=6, shortest=3000, longest=8000,
             expansion=200),
        # a batch of methylation calls: every read has two-path cells
        dict(name="batch_10_sites", kind="resident", machine="acegt", sites=True, reads=10, shortest=1000,
             longest=10000, expansion=50),
        # a caller whose memory another framework holds: a few reads, no allocation
        dict(name="noalloc_5", kind="noalloc", machine="acgt", reads=5, shortest=300, longest=1500, expansion=50),
        # one EM iteration's expectations over a few training reads
        dict(name="em_6_reads", kind="em", machine="acgt", reads=6, shortest=1000, longest=5000, expansion=50),
        # the HDP machine's expectations: transitions and k-mer assignments
        dict(name="em_2_hdp", kind="em", machine="hdp", reads=2, shortest=1500, longest=3000, expansion=50),
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["single", "single", "align", "align", "resident", "resident", "resident", "noalloc", "em"])
    sites = kind in ("single", "align", "resident") and rng.random() < 0.25
    machine = "acegt" if sites else rng.choice(["acgt", "acgt", "hdp"]) if kind != "single" else "acgt"
    most, top = dict(single=(1, 6000), align=(24, 6000), resident=(24, 24000), noalloc=(4, 1500),
                     em=(6, 4000))[kind]
    if sites:
        most, top = min(most, 8), min(top, 8000)
    reads = _spread(rng, 1, most)
    expansion = rng.choice([20, 50, 50, 50] if sites or kind in ("em", "noalloc") else [20, 50, 50, 50, 100, 200])
    if expansion > 50:
        reads, top = min(reads, 8), min(top, 8000)
    longest = _spread(rng, 300, top)
    shortest = max(200, int(longest * rng.uniform(0.3, 1.0)))
    case = dict(kind=kind, machine=machine, reads=reads, shortest=min(shortest, longest), longest=longest,
                expansion=expansion)
    if sites:
        case["sites"] = True
    return case


def work(case):
    """Bytes: sequences, events' means and noises, anchors and the machine's tables in, pairs (about
    three for four events) out.  Operations: 74 a band cell (emissions, both sweeps, posterior)."""
    kmers = case["reads"] * 0.5 * (case["shortest"] + case["longest"])
    events = 1.6 * kmers
    cells = (kmers + events) * (2 * case["expansion"] + 1) * (1.0 if case["expansion"] > 20 else 1.1)
    n = 4 ** 6 if case["machine"] == "acgt" else 5 ** 6
    tables = n * 5 * 8 + (min(n, kmers) * 2000 * 16 if case["machine"] == "hdp" else 0)
    out = 32 * 0.75 * events if case["kind"] != "em" else case["reads"] * n * 25
    return {"bytes": float(kmers + 16 * events + 16 * kmers / 50 + tables + out),
            "flops": float((74 if case["kind"] != "em" else 100) * cells)}


# ------------------------------------------------------------------------------------------------
# machines and reads
# ------------------------------------------------------------------------------------------------
_machines = {}


def _hdp_tables(alphabet, k, seed, start=30.0, stop=150.0, length=2000):
    """Mixture densities on a grid with the knot slopes of the natural cubic spline, as
    synth.hdp_tables makes them; the mixtures two normals wide at most, the densities from one
    product per component."""
    r = np.random.Generator(np.random.PCG64(seed))
    n = len(alphabet) ** k
    base = r.uniform(60.0, 120.0, n)
    means = base[:, None] + r.uniform(-3.0, 3.0, (n, 2))
    sds = r.uniform(1.0, 3.0, (n, 2))
    w = r.uniform(0.0, 1.0, (n, 1))
    w = np.concatenate([w, 1.0 - w], axis=1)
    dx = (stop - start) / float(length - 1)
    grid = np.empty(length)
    grid[:-1] = start + np.arange(length - 1) * dx
    grid[-1] = stop
    dens = np.zeros((n, length))
    for c in range(2):
        z = (grid[None, :] - means[:, c:c + 1]) / sds[:, c:c + 1]
        dens += w[:, c:c + 1] * np.exp(-0.5 * z * z) / (sds[:, c:c + 1] * math.sqrt(2 * math.pi))
    slope = np.ascontiguousarray(synth.spline_knot_slopes_batch(grid, np.asfortranarray(dens)))
    mean = (w * means).sum(axis=1)
    var = (w * (sds ** 2 + means ** 2)).sum(axis=1) - mean ** 2
    return dict(start=start, stop=stop, length=length, grid=grid, density=dens, slope=slope, mean=mean,
                sd=np.sqrt(var), comp_means=means, comp_sds=sds, weights=w)


def _loaded(alphabet, table, emission):
    f = tempfile.NamedTemporaryFile("w", suffix=".model", delete=False)
    try:
        f.write(synth.model_text(alphabet, 6, table))
        f.close()
        return api.StateMachine.load(f.name, api.THREE_STATE, emission)
    finally:
        os.unlink(f.name)


def _machine(name):
    """The machine a program loads once and keeps, with what its reads are drawn from."""
    if name not in _machines:
        alphabet = "ACGT" if name == "acgt" else "ACEGT"
        hdp, drawer = None, None
        if name == "hdp":
            hdp = _hdp_tables(alphabet, 6, 502)
            r = np.random.Generator(np.random.PCG64(2))
            table = np.zeros((len(alphabet) ** 6, 5))
            table[:, 0], table[:, 1] = hdp["mean"], hdp["sd"]
            table[:, 2] = r.uniform(0.5, 2.0, len(table))
            table[:, 3] = 0.3 * table[:, 2]
            table[:, 4] = table[:, 2] ** 3 / table[:, 3] ** 2
            t = _loaded(alphabet, table, api.EMIT_DESCALED).tables()
            sm = api.StateMachine.from_tables(alphabet, 6, t["t"], t["match"], t["gapy"], t["gapx"],
                                              emission=api.EMIT_HDP)
            sm.set_hdp(hdp["start"], hdp["stop"], hdp["length"], hdp["density"], hdp["slope"],
                       np.arange(len(table), dtype=np.int64))

            def drawer(kmers, rr):
                c = (rr.random(len(kmers)) > hdp["weights"][kmers, 0]).astype(np.int64)
                return rr.normal(hdp["comp_means"][kmers, c], hdp["comp_sds"][kmers, c])
        else:
            table = synth.gaussian_table(alphabet, 6, 1000 if name == "acgt" else 103)
            sm = _loaded(alphabet, table, api.EMIT_DESCALED)
        _machines[name] = dict(sm=sm, alphabet=alphabet, table=table, hdp=hdp, drawer=drawer, tables=sm.tables())
    return _machines[name]


def _lengths(case):
    """the reads' reference lengths: the case's own, whatever the seed"""
    r = np.random.Generator(np.random.PCG64(case["reads"]))
    return [int(v) for v in r.integers(case["shortest"], case["longest"] + 1, case["reads"])]


def _capacity(length):
    """pairs a read's output buffer holds (reads of these shapes give 1.0 to 1.3 pairs a reference base)"""
    return 2 * length + 256


def _reads(case, seed):
    M = _machine(case["machine"])
    t = M["table"]
    r = np.random.Generator(np.random.PCG64(seed))
    out = []
    for length in _lengths(case):
        seq = list(synth.random_reference(length, r))
        sites = []
        if case.get("sites"):
            for pos in range(int(r.integers(0, 256)), length - 5, 256):
                seq[pos:pos + 5] = list(("CCAGG", "CCTGG")[int(r.integers(0, 2))])
                sites.append(pos + 1)
        if case["machine"] != "acgt":
            for i in (sites if case.get("sites") else range(length - 1)):
                if seq[i] == "C" and (case.get("sites") or seq[i + 1] == "G") and r.random() < 0.5:
                    seq[i] = "E"
        rd = synth.make_read("".join(seq), M["alphabet"], 6, t[:, 0], t[:, 1], t[:, 2], t[:, 3], r,
                             drawer=M["drawer"])
        for i in sites:
            seq[i] = "X"
        rd["reference"] = "".join(seq)
        out.append(rd)
    return out


def prepare(case, seed):
    M = _machine(case["machine"])
    p = api.pairwiseAlignmentBandingParameters_construct(diagonal_expansion=case["expansion"], threshold=0.01)
    reads = _reads(case, seed)
    degenerate = api.CYTOSINE_METHYLATION2 if case.get("sites") else api.CYTOSINE_METHYLATION3
    state = dict(kind=case["kind"], p=p, degenerate=degenerate)
    # where the program keeps a read's pairs: posteriors in parts per ten million, and x, y, k-mer
    state["out"] = [{"posterior": np.zeros(_capacity(n), np.float32), "where": np.zeros((_capacity(n), 3), np.int32)}
                    for n in _lengths(case)]
    if case["kind"] == "single":
        # a machine per read, scaled to it (getStateMachine3_descaled)
        rd = reads[0]
        sm = _loaded(M["alphabet"], M["table"], api.EMIT_DESCALED)
        sm.set_scaling(rd["scale"], rd["shift"], 1.0)
        state.update(sm=sm, read=rd)
        return state
    state["inputs"] = [api.ReadInput(sm=M["sm"], reference=rd["reference"], events=rd["events"],
                                     anchors=rd["anchors"], scale=rd["scale"], shift=rd["shift"],
                                     degenerate=degenerate) for rd in reads]
    if case["kind"] == "resident":
        state["batch"] = api.Batch(state["inputs"], p)
        state["batch"].upload()
    if case["kind"] == "noalloc" and case["machine"] not in _resident:
        # the entry wants the machine's tables on the device: any allocating call puts them there
        _resident.add(case["machine"])
        api.align_batch(state["inputs"][:1], p)
    return state


_resident = set()


def _keep(out, a):
    """A read's pairs into the program's own buffers, what is left of them cleared."""
    n = len(a)
    out["posterior"][:n], out["posterior"][n:] = a[:, 0], 0
    out["where"][:n], out["where"][n:] = a[:, 1:], 0
    return out


def _rows(pairs):
    return pairs.view(np.int64).reshape(-1, _PAIR_FIELDS)


def _batch_pairs(b, i):
    """Read i's pairs where the library has them (sa_batch_pairs), without a copy."""
    n = api.lib().sa_batch_pair_count(b._h, i)
    if n <= 0:
        return np.zeros((0, _PAIR_FIELDS), np.int64)
    ptr = ctypes.cast(api.lib().sa_batch_pairs(b._h, i), ctypes.POINTER(ctypes.c_int64))
    return np.ctypeslib.as_array(ptr, shape=(n, _PAIR_FIELDS))


def _padded(a, rows):
    out = np.zeros((rows,) + a.shape[1:], a.dtype)
    out[:len(a)] = a
    return out


def run(state):
    kind, out = state["kind"], state["out"]
    if kind == "single":
        rd = state["read"]
        pairs, ll = api.getAlignedPairsUsingAnchors(state["sm"], rd["reference"], rd["events"], rd["anchors"],
                                                    state["p"], degenerate=state["degenerate"],
                                                    with_log_likelihood=True)
        return {"reads": [_keep(out[0], _rows(pairs))], "log_likelihood": np.array([ll])}
    if kind == "em":
        got, status = api.getExpectationsBatch(state["inputs"], state["p"])
        keep = ("likelihood", "transitions", "event_expectations", "posteriors", "observed")
        return {"reads": [dict({k: g[k] for k in keep}, assignments=_padded(g["assignments"], len(o["posterior"])))
                          for g, o in zip(got, out)], "status": np.array(status)}
    if kind == "noalloc":
        res = api.align_batch_noalloc(state["inputs"], state["p"])
    elif kind == "align":
        res = api.align_batch(state["inputs"], state["p"])
    else:
        res = state["batch"]
        res.run()
        res.download()
    n = len(out)
    rows = (lambda i: _rows(res.pairs(i))) if kind == "noalloc" else (lambda i: _batch_pairs(res, i))
    return {"reads": [_keep(out[i], rows(i)) for i in range(n)],
            "log_likelihood": np.array([res.log_likelihood(i) for i in range(n)], np.float32)}


# ------------------------------------------------------------------------------------------------
# the same in 64 bits, from numpy alone
# ------------------------------------------------------------------------------------------------
# Cells of an anti-diagonal live in slots by column (column x in slot x mod S, S past the widest
# anti-diagonal), so a neighbouring column is a roll; a cell has one value per path of its column.
_CUBIC = np.array([[-0.009350833524763, 0.130659527668286, 0.498799810682272, 0.693203116424741],
                   [-0.014532321752540, 0.139942324101744, 0.495635523139337, 0.692140569840976],
                   [-0.004605031767994, 0.063427417320019, 0.695956496475118, 0.514272634594009],
                   [-0.000458661602210, 0.009695946122598, 0.930734667215156, 0.168037164329057]],
                  dtype=np.float32).astype(np.float64)
_MC, _MX, _MY, _OX, _OY, _EX, _EY, _SX, _SY = range(9)


def _log_add(x, y):
    hi, lo = np.maximum(x, y), np.minimum(x, y)
    with np.errstate(invalid="ignore"):
        d = hi - lo
    near = d < 7.5
    d = np.where(near, d, 0.0)
    c = _CUBIC[(d > 1.0).astype(np.int8) + (d > 2.5) + (d > 4.5)]
    return np.where(near, ((c[..., 0] * d + c[..., 1]) * d + c[..., 2]) * d + c[..., 3] + np.where(near, lo, 0.0), hi)


def _band(anchors, lX, lY, expansion):
    """first column and width of every anti-diagonal's cells"""
    n = lX + lY
    xf, w = np.zeros(n + 1, np.int64), np.zeros(n + 1, np.int64)
    corners = [(0, 0)] + [(int(a) + 1, int(b) + 1) for a, b in anchors] + [(lX, lY)]
    x_lo = y_hi = x_hi = y_lo = 0
    k = 0
    for d in range(n + 1):
        lo, hi = x_lo - y_hi, x_hi - y_lo
        lo += (d + lo) & 1
        hi += (d + hi) & 1
        lo += 2 * max(0, x_lo - (d + lo) // 2)
        lo += 2 * max(0, (d - lo) // 2 - y_hi)
        hi -= 2 * max(0, (d + hi) // 2 - x_hi)
        hi -= 2 * max(0, y_lo - (d - hi) // 2)
        xf[d], w[d] = (d + lo) // 2, (hi - lo) // 2 + 1
        if d == sum(corners[k]) and k + 1 < len(corners):
            (ax, ay), (bx, by) = corners[k], corners[k + 1]
            k += 1
            pd, pm, nd, nm = ax + ay, ax - ay, bx + by, bx - by
            x_lo = min(max((pd + pm - expansion) // 2, 0), lX)
            y_hi = min(max((nd - nm + expansion) // 2, 0), lY)
            x_hi = min(max((nd + nm + expansion) // 2, 0), lX)
            y_lo = min(max((pd - pm - expansion) // 2, 0), lY)
    return xf, w


class _Exact:
    """Forward sweep of all reads at once, then all their traceback windows at once."""

    def __init__(self, case, reads):
        M = _machine(case["machine"])
        self.hdp, tb, self.t = M["hdp"], M["tables"], M["tables"]["t"]
        alphabet = sorted(M["alphabet"])
        self.match, self.gapy, self.gapx = tb["match"], tb["gapy"], tb["gapx"]
        P = self.P = 2 if case.get("sites") else 1
        R = self.R = len(reads)
        self.lX = np.array([len(rd["reference"]) - 5 for rd in reads])
        self.lY = np.array([len(rd["events"]) for rd in reads])
        self.n = self.lX + self.lY
        bands = [_band(rd["anchors"], lx, ly, case["expansion"]) for rd, lx, ly in zip(reads, self.lX, self.lY)]
        top = int(self.n.max()) + 1
        self.wmax = int(max(w.max() for _, w in bands))
        S = self.S = 1 << int(math.ceil(math.log2(self.wmax + 4)))
        self.xf, self.w = np.zeros((R, top), np.int64), np.zeros((R, top), np.int64)
        mX, mY = int(self.lX.max()), int(self.lY.max())
        self.kid = np.full((R, mX + S + 2, P), -1, np.int64)       # k-mer of path p of column x
        self.mean, self.noise = np.zeros((R, mY + 1)), np.ones((R, mY + 1))
        self.scale = np.array([rd["scale"] for rd in reads])
        self.shift = np.array([rd["shift"] for rd in reads])
        a = len(alphabet)
        self.suf = a ** 5
        self.a = a
        self.windows = []
        for r, rd in enumerate(reads):
            self.xf[r, :len(bands[r][0])], self.w[r, :len(bands[r][1])] = bands[r]
            code = {c: i for i, c in enumerate(alphabet)}
            for p in range(P):
                seq = rd["reference"].replace("X", "CE"[p])
                ids = np.zeros(self.lX[r], np.int64)
                digits = np.array([code[c] for c in seq])
                for j in range(6):
                    ids = ids * a + digits[j:j + self.lX[r]]
                if p:   # a column without an X has one path
                    ids[ids == self.kid[r, 1:self.lX[r] + 1, 0]] = -1
                self.kid[r, 1:self.lX[r] + 1, p] = ids
            self.mean[r, 1:self.lY[r] + 1], self.noise[r, 1:self.lY[r] + 1] = rd["events"][:, 0], rd["events"][:, 1]
            back = 0
            for d in range(1, int(self.n[r]) + 1):
                end = d == self.n[r]
                if end or (d >= back + 1000 and self.w[r, d] <= 2 * case["expansion"] + 1):
                    at = d if end else d - 41
                    self.windows.append((r, back, d, at, end))
                    back = at
        self.slots = np.arange(S)

    def cells(self, r, d):
        """columns, rows and band membership of the slots on anti-diagonal d (arrays over reads)"""
        xf, w = self.xf[r, d][:, None], self.w[r, d][:, None]
        x = xf + ((self.slots[None, :] - xf) % self.S)
        return x, d[:, None] - x, x - xf < w

    def paths(self, r, x):
        return np.moveaxis(self.kid[r[:, None], x], -1, 1)     # [rows, P, S]

    def there(self, kid, x, inb):
        """paths that exist: column 0 has the empty path alone"""
        ok = (kid >= 0) & inb[:, None, :]
        ok[:, 0] |= (x == 0) & inb
        return ok

    def emissions(self, r, x, y, inb):
        kid = self.paths(r, x)
        ok = (kid >= 0) & (inb & (y >= 1) & (y <= self.lY[r][:, None]))[:, None, :]
        k = np.where(ok, kid, 0)
        yc = np.clip(y, 0, self.mean.shape[1] - 1)
        mean = self.mean[r[:, None], yc][:, None, :]
        noise = self.noise[r[:, None], yc][:, None, :]
        mu = self.match[k, 0]
        u = mean + mu - self.scale[r][:, None, None] * mu - self.shift[r][:, None, None]
        if self.hdp is not None:
            h = self.hdp
            g, L = h["grid"], h["length"]
            dx = g[1] - g[0]
            il = np.clip(((u - g[0]) / dx).astype(np.int64), 0, L - 2)
            y0, y1, s0, s1 = (h[n][k, il + o] for n, o in
                              (("density", 0), ("density", 1), ("slope", 0), ("slope", 1)))
            tl = (u - g[il]) / dx
            tr = 1.0 - tl
            dens = tr * y0 + tl * y1 + tl * tr * ((s0 * dx - (y1 - y0)) * tr + ((y1 - y0) - s1 * dx) * tl)
            dens = np.where(u <= g[0], y0 - s0 * (g[0] - u), np.where(u >= g[-1], y1 + s1 * (u - g[-1]), dens))
            with np.errstate(divide="ignore"):
                e = np.where(ok & (dens > 0), np.log(np.where(dens > 0, dens, 1.0)), -np.inf)
            return e, e
        lam, nu = self.match[k, 4], self.match[k, 2]
        ig = (np.log(lam) - 1.8378770664093453 - 3 * np.log(noise) - lam * ((noise - nu) / nu) ** 2 / noise) / 2
        out = []
        for tab in (self.match, self.gapy):
            sd = tab[k, 1]
            out.append(np.where(ok, -0.91893853320467267 - np.log(sd) - 0.5 * ((u - mu) / sd) ** 2 + ig, -np.inf))
        return out

    def skip(self, kid):
        if self.hdp is not None:
            return np.full(kid.shape, -2.3025850929940455)
        return np.where(kid >= 0, self.gapx[np.where(kid >= 0, kid, 0)], -np.inf)

    def legal(self, left, right):
        """may path q of column x-1 (left) precede path p of column x (right): [rows, q, p, S]"""
        q, p = left[:, :, None, :], right[:, None, :, :]
        return (q < 0) | (p < 0) | (q % self.suf == p // self.a)

    def fold_paths(self, terms, legal, axis):
        """log_add over the paths on `axis` of terms [..., q, p, S], in ascending order, each path's
        states in theirs; returns the fold from log 0"""
        v = None
        for q in range(self.P):
            take = (slice(None), q) if axis == 1 else (slice(None), slice(None), q)
            for s in terms:
                z = np.where(legal[take], s[take], -np.inf)
                v = z if v is None else _log_add(v, z)
        return v

    def forward(self):
        t = self.t
        top = self.xf.shape[1]
        F = self.F = np.full((self.R, top, 3, self.P, self.S), -np.inf)
        F[:, 0, 1:, 0, 0] = 0.0          # ragged left end
        r = np.arange(self.R)
        roll = lambda v: np.roll(v, 1, axis=-1)  # noqa: E731
        for d in range(1, top):
            live = self.n >= d
            rr = r[live]
            x, y, inb = self.cells(rr, np.full(len(rr), d))
            kid = self.paths(rr, x)
            left = self.paths(rr, np.maximum(x - 1, 0))
            ok = self.there(kid, x, inb)
            eM, eY = self.emissions(rr, x, y, inb)
            eX = self.skip(kid)
            leg = self.legal(left, kid)
            l = [roll(F[rr, d - 1, s])[:, :, None, :] for s in range(3)]
            e = eX[:, None]
            vX = self.fold_paths([l[0] + (e + t[_OX]), l[1] + (e + t[_EX]), l[2] + (e + t[_SX])], leg, 1)
            if d >= 2:
                m = [roll(F[rr, d - 2, s])[:, :, None, :] for s in range(3)]
                e = eM[:, None]
                vM = self.fold_paths([m[0] + (e + t[_MC]), m[1] + (e + t[_MX]), m[2] + (e + t[_MY])], leg, 1)
            else:
                vM = np.full_like(vX, -np.inf)
            u = F[rr, d - 1]
            vY = _log_add(u[:, 0] + (eY + t[_OY]), u[:, 2] + (eY + t[_EY]))
            for s, v in enumerate((vM, vX, vY)):
                F[rr, d, s] = np.where(ok, v, -np.inf)

    def windows_back(self, post, expect=None):
        """post(rows, d, posterior cells): called for every anti-diagonal of every window, all
        windows at the same distance from their start at a time; expect: the transitions' posteriors"""
        t, F = self.t, self.F
        r, T, D, at, end = (np.array(v) for v in zip(*self.windows))
        N = len(r)
        shape = (N, 3, self.P, self.S)
        B1, B2 = np.full(shape, -np.inf), np.full(shape, -np.inf)
        E1 = E2 = (np.full((N, self.P, self.S), -np.inf),) * 2
        total = np.zeros(N)
        self.log_likelihood = np.zeros(self.R)
        back = lambda v: np.roll(v, -1, axis=-1)  # noqa: E731
        for q in range(int((D - T).max())):
            d = np.maximum(D - q, 0)
            live = D - q > T
            x, y, inb = self.cells(r, d)
            kid, right = self.paths(r, x), self.paths(r, x + 1)
            ok = self.there(kid, x, inb) & live[:, None, None]
            E0 = self.emissions(r, x, y, inb)
            if q == 0:
                e = np.where(end[:, None], [(t[_OX] + t[_OY]) / 2, t[_EX], t[_EY]], [t[_MC], t[_MX], t[_MY]])
                B = np.where(ok[:, None], e[:, :, None, None], -np.inf)
            else:
                leg = self.legal(kid, right)
                m = (back(B2[:, 0])[:, None, :, :], back(E2[0])[:, None, :, :])
                lo = (back(B1[:, 1])[:, None, :, :], self.skip(right)[:, None, :, :])
                u = B1[:, 2]
                v = []
                for ts in ((_MC, _OY, _OX), (_MX, None, _EX), (_MY, _EY, _SX)):
                    z = self.fold_paths([m[0] + (m[1] + t[ts[0]])], leg, 2)
                    if ts[1] is not None:
                        z = _log_add(z, u + (E1[1] + t[ts[1]]))
                    v.append(self.fold_into(z, lo[0] + (lo[1] + t[ts[2]]), leg))
                B = np.where(ok[:, None], np.stack(v, axis=1), -np.inf)
            here = live & (d <= at)
            fresh = here & ((at - d) % 10 == 0)
            if fresh.any():
                i = np.flatnonzero(fresh)
                total[i] = self.total(r[i], d[i], q > 0, B[i], B1[i], E1[0][i])
                fin = i[end[i] & (d[i] == D[i])]
                self.log_likelihood[r[fin]] = total[fin]
            i = np.flatnonzero(here)
            if len(i):
                if expect is None:
                    p = np.exp(F[r[i], d[i], 0] + B[i, 0] - total[i, None, None])
                    post(i, d[i], x[i], y[i], kid[i], np.where(ok[i], p, 0.0))
                else:
                    expect(i, r[i], d[i], T[i], x[i], y[i], kid[i], ok[i], B[i], total[i], [e[i] for e in E0])
            B2, B1, E2, E1 = B1, B, E1, E0

    def fold_into(self, v, term, legal):
        for p in range(self.P):
            v = _log_add(v, np.where(legal[:, :, p], term[:, :, p], -np.inf))
        return v

    def total(self, r, d, have_next, B, B1, e1):
        """the total probability through anti-diagonal d, cell by cell in ascending order"""
        t, F = self.t, self.F

        def cells_folded(s):
            v = np.full((s.shape[0], s.shape[-1]), -np.inf)
            for p in range(self.P):
                v = _log_add(v, s[:, p])
            return v

        def fold(v, dd):
            order = (self.xf[r, dd][:, None] + np.arange(self.wmax)[None, :]) % self.S
            v = np.take_along_axis(v, order, axis=1)
            v[np.arange(self.wmax)[None, :] >= self.w[r, dd][:, None]] = -np.inf
            z = np.full(len(v), -np.inf)
            for i in range(self.wmax):
                z = _log_add(z, v[:, i])
            return z
        f = F[r, d]
        s = _log_add(_log_add(f[:, 0] + B[:, 0], f[:, 1] + B[:, 1]), f[:, 2] + B[:, 2])
        z = fold(cells_folded(s), d)
        if have_next:
            x, _, _ = self.cells(r, d + 1)
            leg = self.legal(self.paths(r, np.maximum(x - 1, 0)), self.paths(r, x))
            m = [np.roll(F[r, d - 1, s], 1, axis=-1)[:, :, None, :] for s in range(3)]
            e = e1[:, None]
            thr = self.fold_paths([m[0] + (e + t[_MC]), m[1] + (e + t[_MX]), m[2] + (e + t[_MY])], leg, 1)
            z = _log_add(z, fold(cells_folded(thr + B1[:, 0]), d + 1))
        return z


def _exact_pairs(case, reads):
    X = _Exact(case, reads)
    X.forward()
    found = []

    def post(i, d, x, y, kid, p):
        w, q, s = np.nonzero((p >= 0.01) & ((x > 0) & (y > 0))[:, None, :])
        cell = x[w, s] - X.xf[np.array([v[0] for v in X.windows])[i[w]], d[w]]
        found.append(np.stack([i[w], -d[w], cell, q, np.minimum(p[w, q, s], 1.0) * 1e7]))

    X.windows_back(post)
    f = np.concatenate(found, axis=1)
    f = f[:, np.lexsort((f[3], f[2], f[1], f[0]))]
    owner = np.array([v[0] for v in X.windows])[f[0].astype(np.int64)]
    return {"reads": [{"posterior": _padded(f[4, owner == r], _capacity(n)), "where": None}
                      for r, n in enumerate(_lengths(case))],
            "log_likelihood": X.log_likelihood}


def _exact_expectations(case, reads):
    X = _Exact(case, reads)
    X.forward()
    t, F = X.t, X.F
    lik = np.zeros(X.R)
    trans = np.full((X.R, 3, 3), 0.001)
    terms = []

    def expect(i, r, d, T, x, y, kid, ok, B, total, E):
        one = np.maximum(d - 1, 0)
        two = np.maximum(d - 2, 0)
        np.add.at(lik, r, total)
        z = total[:, None]
        k, okc = kid[:, 0], ok[:, 0]
        l = np.roll(F[r, one], 1, axis=-1)[:, :, 0]
        m = np.where((d - 2 >= T)[:, None, None], np.roll(F[r, two], 1, axis=-1)[:, :, 0], -np.inf)
        u = F[r, one][:, :, 0]
        e, eM, eY = X.skip(k), E[0][:, 0], E[1][:, 0]
        with np.errstate(invalid="ignore"):
            for s, c, src, em, tr in ((0, 1, l, e, _OX), (1, 1, l, e, _EX), (2, 1, l, e, _SX), (0, 0, m, eM, _MC),
                                      (1, 0, m, eM, _MX), (2, 0, m, eM, _MY), (0, 2, u, eY, _OY), (2, 2, u, eY, _EY)):
                p = np.where(okc, np.exp(src[:, s] + B[:, c, 0] + (em + t[tr]) - z), 0.0)
                np.add.at(trans, (r, s, c), np.nan_to_num(p).sum(axis=1))
                if c == 0 and X.hdp is None:
                    w, q = np.nonzero(okc & (k >= 0) & (y >= 1))
                    mu = X.match[k[w, q], 0]
                    xe = X.mean[r[w], y[w, q]] + mu - X.scale[r[w]] * mu - X.shift[r[w]]
                    terms.append(np.stack([r[w], k[w, q], i[w], -d[w], x[w, q], np.full(len(w), s), p[w, q], xe]))

    X.windows_back(None, expect)
    n = len(X.match)
    out = []
    f = np.concatenate(terms, axis=1) if terms else np.zeros((8, 0))
    f = f[:, np.lexsort((f[5], f[4], f[3], f[2], f[1], f[0]))]
    edge = np.flatnonzero(np.diff(f[0] * n + f[1])) + 1 if f.shape[1] else np.zeros(0, np.int64)
    weight = np.full((X.R, n), 0.001)
    ev = np.zeros((X.R, n, 2))
    for g in np.split(f, edge, axis=1) if f.shape[1] else []:
        r, k = int(g[0, 0]), int(g[1, 0])
        e0, po = np.cumsum(g[6] * g[7]), 0.001 + np.cumsum(g[6])
        ev[r, k] = e0[-1], (g[6] * (g[7] - e0 / po) ** 2).sum()
        weight[r, k] = po[-1]
    for r in range(X.R):
        out.append({"likelihood": float(lik[r]), "transitions": trans[r], "event_expectations": ev[r],
                    "posteriors": weight[r], "observed": None, "assignments": None})
    return {"reads": out, "status": None}


def exact(case, seed):
    kmers = case["reads"] * 0.5 * (case["shortest"] + case["longest"])
    cells = 2.6 * kmers * (2 * case["expansion"] + 1) * (4 if case.get("sites") else 1)
    # about 20 s, and a forward store of a few GB
    if cells > (5e6 if case["machine"] == "hdp" or case["kind"] == "em" else 8e6) or 2.6 * case["longest"] > 25000:
        return None
    reads = _reads(case, seed)
    return _exact_expectations(case, reads) if case["kind"] == "em" else _exact_pairs(case, reads)
