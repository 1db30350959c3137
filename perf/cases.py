"""The work that a host program has this library do, as measurable cases.

Sizes are those of the repository's own workloads (bench.py) and tests: blocks
of segmented arrays, column-major (first index fastest), virtual segments of 12
to 48, occupied segments of 5 to 24, problems from o=10/v=48 to o=64/v=512.
Each kind of case below says what it stands for; `listed` fixes one or two
sizes of each, `draw` takes others of the same ranges.

  pair     one block pair of a contraction statement, plain FP64: the drop-in
           entry on host blocks as the interpreter calls it, or the device entry
  step     one pardo step (every block pair of one statement) as a batch, plain
           FP64 or split precision, dense or with zero blocks, replayed as a
           graph or run eagerly
  loop     the ladder's pardo loop: one batch, T held, rebound to the next
           (a,b) slab and run
  triples  a (T) step: both contraction statements and either the energy (W
           never stored, rebound to the loop's next step) or W
  algebra  the block operations between contractions: permute, permuted add,
           scale, accumulate, slice, insert, norm
  energy   an unfused (T) energy: a copy of W divided by the denominators, and
           the energy of W
  sweep    the amplitude update over every block of the amplitude arrays
"""
import itertools
import math
import random

import numpy as np
import torch

SPLIT_FLOPS = 4.0e12  # the most a drawn split-precision case multiplies (FP64-equivalent)
FP64_FLOPS = 2.0e10   # the most a drawn plain FP64 step multiplies
LADDER = ([1, 2, 3, 4], [1, 2, 5, 6], [5, 6, 3, 4])  # R(a,b,i,j) = V(a,b,c,d) T(c,d,i,j)
RING = ([1, 3, 2, 4], [1, 7, 5, 3], [5, 2, 7, 4])    # R(a,i,b,j) = V(a,k,c,i) T(c,b,k,j)
# W(a,i,b,j,c,k) = V1(b,c,d,k) T(a,d,i,j) - V2(l,c,j,k) T(a,b,i,l)
TRIPLES = (([1, 2, 3, 4, 5, 6], [3, 5, 7, 6], [1, 7, 2, 4]), ([1, 2, 3, 4, 5, 6], [8, 5, 4, 6], [1, 3, 2, 8]))


def listed():
    return [
        # one interpreter call on host blocks: the o=10/v=48 ladder's 144x25x144 pair, all latency
        {"name": "pair_host_ladder", "kind": "pair", "host": True, "pattern": "ladder", "v": 12, "o": 5, "w": 12},
        # one device call: an o=40/v=300 ring pair with uneven segments, both operands permuted
        {"name": "pair_ring", "kind": "pair", "host": False, "pattern": "ring", "v": 33, "o": 20, "w": 29},
        # a small pardo step in plain FP64: o=10/v=48, 1024 pairs
        {"name": "step_ladder_fp64", "kind": "step", "pattern": "ladder", "split": False, "slices": 0, "graph": True,
         "v": 48, "vlo": 12, "vhi": 12, "o": 10, "oseg": 5, "zero": 0.0, "ab": 0, "structure": 1},
        # the same step in split precision: launches and idle SMs count
        {"name": "step_ladder", "kind": "step", "pattern": "ladder", "split": True, "slices": 5, "graph": True,
         "v": 48, "vlo": 12, "vhi": 12, "o": 10, "oseg": 5, "zero": 0.0, "ab": 0, "structure": 1},
        # the ring term of o=40/v=300, uneven segments of 24 to 40, all blocks dense, operands sliced every run
        {"name": "step_ring", "kind": "step", "pattern": "ring", "split": True, "slices": 5, "graph": False,
         "v": 300, "vlo": 24, "vhi": 40, "o": 40, "oseg": 20, "zero": 0.0, "ab": 0, "structure": 2},
        # a block-sparse ladder step of o=48/v=400: uneven segments, 30 % of V's blocks zero, 2x2 (a,b) segments
        {"name": "step_sparse", "kind": "step", "pattern": "ladder", "split": True, "slices": 5, "graph": True,
         "v": 400, "vlo": 12, "vhi": 48, "o": 48, "oseg": 24, "zero": 0.3, "ab": 2, "structure": 3},
        # two slabs of the o=64/v=512 ladder's loop, 1 % of T's entries a thousand times larger
        {"name": "loop_ladder", "kind": "loop", "v": 512, "vseg": 32, "o": 64, "oseg": 16, "slabs": 2, "slices": 5},
        # two steps of the o=24/v=240 (T) energy's loop
        {"name": "loop_triples", "kind": "triples", "store": False, "slices": 5, "o": 24, "v": 240, "vlo": 24, "vhi": 24,
         "steps": 2, "structure": 4},
        # a (T) step whose W is kept: uneven virtual segments, W in the denominator's order
        {"name": "step_triples_store", "kind": "triples", "store": True, "slices": 5, "o": 12, "v": 63, "vlo": 17,
         "vhi": 24, "steps": 1, "structure": 5},
        # the block operations on the largest block that the benchmark times
        {"name": "algebra", "kind": "algebra", "e0": 96, "e1": 96, "e2": 96, "e3": 96, "perm": "3214"},
        # the unfused (T) energy of one 24^6 block
        {"name": "energy", "kind": "energy", "rank": 6, "v": 24, "o": 24, "w": 24},
        # the amplitude update of o=40/v=300: 400 blocks of uneven segments
        {"name": "sweep_amplitudes", "kind": "sweep", "v": 300, "vlo": 24, "vhi": 40, "o": 40, "oseg": 20, "structure": 2},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pair", "pair", "step", "step", "step", "loop", "triples", "triples", "algebra", "energy", "sweep"])
    for _ in range(1000):
        if kind == "pair":
            c = {"kind": kind, "host": rng.random() < 0.5, "pattern": rng.choice(["ladder", "ring"]), "v": _log(rng, 8, 40),
                 "o": _log(rng, 4, 24), "w": _log(rng, 8, 40)}
        elif kind == "step":
            split = rng.random() < 0.75
            lo = rng.randint(10, 32)
            c = {"kind": kind, "pattern": rng.choice(["ladder", "ring"]), "split": split,
                 "slices": rng.choice([4, 5, 5, 5, 6, 7]) if split else 0, "graph": rng.random() < 0.5,
                 "v": _log(rng, 40, 400), "vlo": lo, "vhi": rng.randint(lo, 48), "o": _log(rng, 8, 48),
                 "oseg": rng.randint(5, 24), "zero": rng.choice([0.0, 0.0, 0.3]), "ab": rng.choice([0, 1, 2]),
                 "structure": rng.randrange(1000)}
        elif kind == "loop":
            c = {"kind": kind, "v": rng.randint(100, 500), "vseg": rng.choice([16, 24, 32, 32, 40]), "o": rng.randint(20, 64),
                 "oseg": rng.choice([10, 16, 20]), "slabs": 2, "slices": rng.choice([3, 4, 5, 5, 6, 7])}
        elif kind == "triples":
            store = rng.random() < 0.5
            lo = rng.randint(10, 24)
            hi = lo if not store and rng.random() < 0.6 else rng.randint(lo, 28)
            c = {"kind": kind, "store": store, "slices": rng.choice([4, 5, 5, 5, 6]), "o": rng.randint(6, 24),
                 "v": rng.randint(2 * hi + 2, 240), "vlo": lo, "vhi": hi, "steps": 1 if store or lo < hi else 2,
                 "structure": rng.randrange(1000)}
        elif kind == "algebra":
            p = [1, 2, 3, 4]
            rng.shuffle(p)
            c = {"kind": kind, "e0": _log(rng, 8, 96), "e1": _log(rng, 8, 96), "e2": _log(rng, 8, 96), "e3": _log(rng, 8, 96),
                 "perm": "".join(map(str, p))}
        elif kind == "energy":
            r = rng.choice([4, 6])
            hi = 24 if r == 6 else 96
            c = {"kind": kind, "rank": r, "v": rng.randint(8, hi), "o": rng.randint(6, hi), "w": rng.randint(8, hi)}
        else:
            lo = rng.randint(12, 32)
            c = {"kind": kind, "v": _log(rng, 40, 300), "vlo": lo, "vhi": rng.randint(lo, 48), "o": _log(rng, 8, 48),
                 "oseg": rng.randint(5, 24), "structure": rng.randrange(1000)}
        w = work(c)
        if kind == "step" and not c["split"] and w["flops"] > FP64_FLOPS:
            continue
        if w["flops"] > SPLIT_FLOPS or w["bytes"] > 8e9:
            continue
        if kind == "step" and _pairs(c) > 12000:
            continue
        if kind == "triples" and (_triples_elements(c) > (2.0e8 if c["store"] else 2.0e9) or w["flops"] > 2.0e12):
            continue
        return c
    return listed()[2] | {"name": "small step"}


# ------------------------------------------------------------------ segments and blocks
def _segments(total, lo, hi, seed):
    """Segment sizes from lo to hi that add up to total; the last one takes what is left, at least 2."""
    rng, out = random.Random(seed), []
    while total > hi:
        n = rng.randint(lo, hi)
        out.append(n - (total - n == 1))
        total -= out[-1]
    return out + ([total] if total else [])


def _even(total, seg):
    return _segments(total, seg, seg, 0)


def _size(ext):
    return int(np.prod(ext))


class _Array:
    """The blocks of one segmented array in one buffer, each at a 256-byte boundary; absent blocks are zero blocks."""

    def __init__(self, segs, keys):
        self.segs, self.at, n = segs, {}, 0
        for k in keys:
            self.at[k] = n
            n += (_size(self.ext(k)) + 31) // 32 * 32
        self.buf = torch.zeros(max(n, 1), dtype=torch.float64, device="cuda")

    def ext(self, k):
        return [self.segs[q][k[q]] for q in range(len(k))]

    def block(self, k):
        return self.buf[self.at[k]:self.at[k] + _size(self.ext(k))] if k in self.at else None

    def address(self, k):
        return self.buf.data_ptr() + 8 * self.at[k] if k in self.at else 0

    def tensor(self, k):
        """The block as a tensor whose last dimension is the first index."""
        return self.block(k).view(*reversed(self.ext(k)))


def _all(segs):
    return list(itertools.product(*[range(len(s)) for s in segs]))


def _generator(seed, salt):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 1009 + salt)


def _triples(device, rows, d, l, r):
    """The block triples (keys of D, L, R per row) as the array that the batch entries take."""
    out = np.zeros(len(rows), device.TRIPLE_DTYPE)
    for col, arr, q in (("d", d, 0), ("l", l, 1), ("r", r, 2)):
        out[col] = [arr.address(x[q]) for x in rows]
        e = np.ones((len(rows), 6), np.int32)
        e[:, :len(arr.segs)] = [arr.ext(x[q]) for x in rows]
        out[col + "ext"] = e
    return out


def _pattern(a4, labels):
    d, l, r = labels
    return a4.ref.get_contraction_ptrn(len(d), len(l), len(r), d + l + r)[1]


def _einsum(labels, l, r):
    """One block pair in 64 bits; tensors hold the first index last."""
    s = lambda x: "".join(chr(96 + v) for v in reversed(x))
    return torch.einsum("%s,%s->%s" % (s(labels[1]), s(labels[2]), s(labels[0])), l, r)


# ------------------------------------------------------------------ pair
def _pair_shapes(c):
    v, o, w = c["v"], c["o"], c["w"]
    if c["pattern"] == "ladder":
        return LADDER, [v, w, o, o], [v, w, w, v], [w, v, o, o]
    return RING, [v, o, w, o], [v, o, w, o], [w, w, o, o]


def _pair_data(c, seed):
    _, de, le, re = _pair_shapes(c)
    rng = np.random.default_rng(seed)
    return rng.uniform(-1.0, 1.0, _size(le)) / (4 * c["v"]), rng.normal(0.0, 0.1, _size(re))


def _pair_prepare(c, seed):
    import aces4_gb300 as a4

    labels, de, le, re = _pair_shapes(c)
    l, r = _pair_data(c, seed)
    a4.device.init()
    s = {"a4": a4, "labels": labels, "de": de, "le": le, "re": re, "ptrn": _pattern(a4, labels)}
    if c["host"]:
        return s | {"l": l, "r": r, "d": np.zeros(_size(de))}
    return s | {"l": torch.from_numpy(l).cuda(), "r": torch.from_numpy(r).cuda(),
                "d": torch.zeros(_size(de), dtype=torch.float64, device="cuda"), "stream": torch.cuda.current_stream()}


def _pair_run(s, c):
    if c["host"]:
        ierr = s["a4"].ref.tensor_block_contract(s["ptrn"], s["l"], s["le"], s["r"], s["re"], s["d"], s["de"])
        if ierr:
            raise RuntimeError("tensor_block_contract: ierr %d" % ierr)
    else:
        s["a4"].device.contract(s["ptrn"], s["l"], s["le"], s["r"], s["re"], s["d"], s["de"], stream=s["stream"])
    return s["d"]


def _pair_exact(c, seed):
    labels, de, le, re = _pair_shapes(c)
    l, r = _pair_data(c, seed)
    d = _einsum(labels, torch.from_numpy(l).view(*reversed(le)), torch.from_numpy(r).view(*reversed(re))).reshape(-1)
    return d.numpy() if c["host"] else d


def _pair_work(c):
    labels, de, le, re = _pair_shapes(c)
    k = math.prod(e for x, e in zip(labels[1], le) if x not in labels[0])
    return {"bytes": 8 * (_size(de) + _size(le) + _size(re)), "flops": 2 * _size(de) * k}


# ------------------------------------------------------------------ step
def _step_segs(c):
    v, o = _segments(c["v"], c["vlo"], c["vhi"], c["structure"]), _even(c["o"], c["oseg"])
    few = v[:c["ab"]] if c["ab"] else v
    if c["pattern"] == "ladder":
        return [few, few, o, o], [few, few, v, v], [v, v, o, o]
    return [few, o, v, o], [few, o, v, o], [v, v, o, o]


def _step_keys(c):
    rs, vs, ts = _step_segs(c)
    rng = random.Random(c["structure"] + 7)
    live = [k for k in _all(vs) if rng.random() >= c["zero"]]
    return _all(rs), live, _all(ts)


def _step_rows(c):
    """(D key, L key, R key) of every block pair of the statement, zero V blocks among them."""
    rs, vs, ts = _step_segs(c)
    if c["pattern"] == "ladder":
        return [((a, b, i, j), (a, b, x, y), (x, y, i, j)) for a, b, i, j in _all(rs) for x, y in _all(vs[2:])]
    return [((a, i, b, j), (a, k, x, i), (x, b, k, j)) for a, i, b, j in _all(rs) for k, x in _all([vs[1], vs[2]])]


def _step_data(c, seed):
    rs, vs, ts = _step_segs(c)
    rk, vk, tk = _step_keys(c)
    r, v, t = _Array(rs, rk), _Array(vs, vk), _Array(ts, tk)
    v.buf.uniform_(-1.0, 1.0, generator=_generator(seed, 1)).div_(c["v"])
    t.buf.normal_(0.0, 0.1, generator=_generator(seed, 2))
    return r, v, t


def _step_prepare(c, seed):
    import aces4_gb300 as a4

    a4.device.init()
    r, v, t = _step_data(c, seed)
    labels = LADDER if c["pattern"] == "ladder" else RING
    torch.cuda.synchronize()  # the batch reads the blocks on a stream of its own when it is made
    b = a4.device.Batch(_pattern(a4, labels), 4, 4, 4, _triples(a4.device, _step_rows(c), r, v, t),
                        precision=a4.device.PREC_OZAKI_BF16 if c["split"] else a4.device.PREC_FP64, slices=c["slices"] or 5)
    return {"batch": b, "r": r, "v": v, "t": t, "stream": torch.cuda.current_stream()}


def _step_run(s, c):
    if c["graph"]:
        s["batch"].run_graph(s["stream"])
    else:
        s["batch"].run(s["stream"])
    return s["r"].buf


def _step_exact(c, seed):
    if work(c)["flops"] > 6e12:
        return None
    r, v, t = _step_data(c, seed)
    labels = LADDER if c["pattern"] == "ladder" else RING
    for d, l, x in _step_rows(c):
        if l in v.at:
            r.tensor(d).add_(_einsum(labels, v.tensor(l), t.tensor(x)))
    return r.buf


def _pairs(c):
    rs, vs, _ = _step_segs(c)
    return _size([len(x) for x in rs]) * (len(vs[2]) * (len(vs[3]) if c["pattern"] == "ladder" else len(vs[1])))


def _step_work(c):
    rs, vs, ts = _step_segs(c)
    live = set(_step_keys(c)[1])
    n = lambda segs: _size([sum(s) for s in segs])
    held = sum(_size([vs[q][k[q]] for q in range(4)]) for k in live)
    cols = sum(ts[2]) * sum(ts[3]) if c["pattern"] == "ladder" else sum(ts[1]) * sum(ts[3])
    return {"bytes": 8 * (n(rs) + held + n(ts)), "flops": 2 * held * cols}


# ------------------------------------------------------------------ loop
def _loop_segs(c):
    return _even(c["v"] // c["vseg"] * c["vseg"], c["vseg"]), _even(c["o"], c["oseg"])


def _loop_data(c, seed):
    vs, os_ = _loop_segs(c)
    one = [c["vseg"]]
    r = [_Array([one, one, os_, os_], _all([one, one, os_, os_])) for _ in range(c["slabs"])]
    v = [_Array([one, one, vs, vs], _all([one, one, vs, vs])) for _ in range(c["slabs"])]
    t = _Array([vs, vs, os_, os_], _all([vs, vs, os_, os_]))
    for q, x in enumerate(v):
        x.buf.uniform_(-1.0, 1.0, generator=_generator(seed, 10 + q)).div_(c["v"])
    step = 1 << 26
    for q, at in enumerate(range(0, t.buf.numel(), step)):
        x = t.buf[at:at + step]
        g = _generator(seed, 100 + q)
        x.normal_(0.0, 0.01, generator=g)
        x[torch.rand(x.numel(), device="cuda", generator=g) < 0.01] *= 1000.0
    return r, v, t


def _loop_rows(c):
    vs, os_ = _loop_segs(c)
    return [((0, 0, i, j), (0, 0, x, y), (x, y, i, j)) for i, j in _all([os_, os_]) for x, y in _all([vs, vs])]


def _loop_prepare(c, seed):
    import aces4_gb300 as a4

    a4.device.init()
    r, v, t = _loop_data(c, seed)
    rows = _loop_rows(c)
    trips = [_triples(a4.device, rows, r[q], v[q], t) for q in range(c["slabs"])]
    st = torch.cuda.current_stream()
    torch.cuda.synchronize()
    b = a4.device.Batch(_pattern(a4, LADDER), 4, 4, 4, trips[0], precision=a4.device.PREC_OZAKI_BF16, slices=c["slices"])
    b.hold(1, stream=st)  # T is the same for every slab
    return {"batch": b, "r": r, "v": v, "t": t, "trips": trips, "stream": st}


def _loop_run(s, c):
    for x in s["trips"]:
        s["batch"].rebind(x, stream=s["stream"])
        s["batch"].run(s["stream"])
    return [x.buf for x in s["r"]]


def _loop_exact(c, seed):
    r, v, t = _loop_data(c, seed)
    for q in range(c["slabs"]):
        for d, l, x in _loop_rows(c):
            lb, rb, out = v[q].tensor(l), t.tensor(x), r[q].tensor(d)
            k = lb.shape[0] * lb.shape[1]
            out.view(rb.shape[0] * rb.shape[1], -1).addmm_(rb.reshape(-1, k), lb.reshape(k, -1))
    return [x.buf for x in r]


def _loop_work(c):
    v, o = sum(_loop_segs(c)[0]), c["o"]
    ab = c["vseg"] ** 2
    return {"bytes": 8 * (c["slabs"] * ab * (v * v + o * o) + v * v * o * o), "flops": 2 * c["slabs"] * ab * v * v * o * o}


# ------------------------------------------------------------------ triples
def _triples_segs(c):
    return _segments(c["v"], c["vlo"], c["vhi"], c["structure"]), [c["o"]]


def _triples_ab(c):
    """The (a,b) segments of the steps; the last segment may be shorter and is not one of them."""
    return [(0, 1), (1, 0)][:c["steps"]]


def _triples_elements(c):
    vs, os_ = _triples_segs(c)
    return vs[0] * vs[1] * sum(vs) * os_[0] ** 3


def _triples_data(c, seed):
    vs, os_ = _triples_segs(c)
    v1, v2, t = ([vs, vs, vs, os_], [os_, vs, os_, os_], [vs, vs, os_, os_])
    v1, v2, t = (_Array(x, _all(x)) for x in (v1, v2, t))
    v1.buf.uniform_(-1.0, 1.0, generator=_generator(seed, 21)).div_(c["v"])
    v2.buf.uniform_(-1.0, 1.0, generator=_generator(seed, 22)).div_(c["v"])
    t.buf.normal_(0.0, 0.1, generator=_generator(seed, 23))
    rng = np.random.default_rng(seed)
    e = np.concatenate([rng.uniform(-2.0, -0.5, c["o"]), rng.uniform(0.2, 5.0, c["v"])])
    return v1, v2, t, e


def _triples_w(c):
    vs, os_ = _triples_segs(c)
    segs = [vs, os_, vs, os_, vs, os_]
    a, b = _triples_ab(c)[0]
    return segs, [(a, 0, b, 0, x, 0) for x in range(len(vs))]


def _triples_rows(c, a, b):
    """Both statements' (W, L, R) keys of step (a,b); W blocks are named by the first step's."""
    vs, _ = _triples_segs(c)
    wk = _triples_w(c)[1]
    t1 = [(wk[x], (b, x, d, 0), (a, d, 0, 0)) for x in range(len(vs)) for d in range(len(vs))]
    t2 = [(wk[x], (0, x, 0, 0), (a, b, 0, 0)) for x in range(len(vs))]
    return t1, t2


def _triples_prepare(c, seed):
    import aces4_gb300 as a4

    a4.device.init()
    vs, os_ = _triples_segs(c)
    v1, v2, t, e = _triples_data(c, seed)
    segs, wk = _triples_w(c)
    w = _Array(segs, wk) if c["store"] else None
    if w is None:  # the energy form never touches W: its blocks are only named
        w = _Array.__new__(_Array)
        w.segs, w.at, n = segs, {}, 0
        for k in wk:
            w.at[k] = n
            n += (_size(w.ext(k)) + 31) // 32 * 32
        w.buf = torch.empty(n, dtype=torch.float64, device="cuda")
    fock = torch.from_numpy(np.diag(e).ravel(order="F").copy()).cuda()
    ptrn = [_pattern(a4, x) for x in TRIPLES]
    steps = []
    for a, b in _triples_ab(c):
        r1, r2 = _triples_rows(c, a, b)
        terms = [(ptrn[0], _triples(a4.device, r1, w, v1, t), 1), (ptrn[1], _triples(a4.device, r2, w, v2, t), -1)]
        energy = None
        if not c["store"]:
            energy = {"blocks": [w.block(k) for k in wk], "index_values": [[2 + a, 1, 2 + b, 1, 2 + k[4], 1] for k in wk],
                      "ext1": [len(e), len(e)], "e_or_fock": fock, "seg_sizes": os_ + vs, "efact": 1.0}
        steps.append((terms, energy))
    torch.cuda.synchronize()
    f = a4.device.Fused(6, 4, 4, steps[0][0], slices=c["slices"], energy=steps[0][1])
    esum = None if c["store"] else torch.zeros(len(steps), dtype=torch.float64, device="cuda")
    return {"fused": f, "w": w, "v1": v1, "v2": v2, "t": t, "fock": fock, "steps": steps, "esum": esum,
            "stream": torch.cuda.current_stream()}


def _triples_run(s, c):
    if c["store"]:
        s["fused"].run(stream=s["stream"])
        return s["w"].buf
    s["esum"].zero_()
    for q, (terms, energy) in enumerate(s["steps"]):
        if len(s["steps"]) > 1:
            s["fused"].rebind(terms, energy=energy, stream=s["stream"])
        s["fused"].run(s["esum"][q:q + 1], s["stream"])
    return s["esum"]


def _triples_exact(c, seed):
    vs, os_ = _triples_segs(c)
    v1, v2, t, e = _triples_data(c, seed)
    segs, wk = _triples_w(c)
    at = np.concatenate([[0], np.cumsum(vs)]) + c["o"]
    ev = torch.from_numpy(e).cuda()
    occ = ev[:c["o"]]
    if c["store"]:
        w = _Array(segs, wk)
        for rows, labels, left, sign in zip(_triples_rows(c, *_triples_ab(c)[0]), TRIPLES, (v1, v2), (1.0, -1.0)):
            for d, l, r in rows:
                w.tensor(d).add_(_einsum(labels, left.tensor(l), t.tensor(r)), alpha=sign)
        return w.buf
    out = torch.zeros(c["steps"], dtype=torch.float64, device="cuda")
    for q, (a, b) in enumerate(_triples_ab(c)):
        r1, r2 = _triples_rows(c, a, b)
        for x in range(len(vs)):
            w = sum(_einsum(TRIPLES[0], v1.tensor(l), t.tensor(r)) for d, l, r in r1 if d == wk[x])
            w -= _einsum(TRIPLES[1], v2.tensor(r2[x][1]), t.tensor(r2[x][2]))
            seg = lambda k: ev[at[k]:at[k] + vs[k]]
            # dimensions k, c, j, b, i, a
            eps = (occ.view(1, 1, 1, 1, -1, 1) + occ.view(1, 1, -1, 1, 1, 1)) + occ.view(-1, 1, 1, 1, 1, 1)
            eps = eps - seg(a).view(1, 1, 1, 1, 1, -1) - seg(b).view(1, 1, 1, -1, 1, 1) - seg(x).view(1, -1, 1, 1, 1, 1)
            out[q] += (w * (w / eps)).sum()
    return out


def _triples_work(c):
    vs, os_ = _triples_segs(c)
    o, v = os_[0], sum(vs)
    a, b = vs[0], vs[1]
    n = _triples_elements(c)
    read = b * v * v * o + o * v * o * o + a * v * o * o
    return {"bytes": 8 * c["steps"] * (read + (n if c["store"] else 0)), "flops": 2 * c["steps"] * n * (v + o)}


# ------------------------------------------------------------------ algebra
def _algebra_shapes(c):
    ext = [c["e0"], c["e1"], c["e2"], c["e3"]]
    o2n = [int(x) for x in c["perm"]]
    out = [0] * 4
    for i, p in enumerate(o2n):
        out[p - 1] = ext[i]
    sub = [max(1, 3 * x // 4) for x in out]
    return ext, o2n, out, sub, [(x - y) // 2 for x, y in zip(out, sub)]


def _algebra_data(c, seed):
    n = _size(_algebra_shapes(c)[0])
    return [torch.empty(n, dtype=torch.float64, device="cuda").normal_(generator=_generator(seed, 31 + q)) for q in range(2)]


def _algebra_prepare(c, seed):
    import aces4_gb300 as a4

    a4.device.init()
    ext, o2n, out, sub, beg = _algebra_shapes(c)
    x, y = _algebra_data(c, seed)
    new = lambda m: torch.zeros(m, dtype=torch.float64, device="cuda")
    rlab = [0] * 4
    for i, p in enumerate(o2n):  # index i of x is index p of the result
        rlab[i] = p
    return {"dev": a4.device, "ext": ext, "o2n": o2n, "out": out, "sub": sub, "beg": beg, "rlab": rlab, "x": x, "y": y,
            "z": new(x.numel()), "w": new(x.numel()), "u": new(x.numel()), "s": new(_size(sub)), "v": new(x.numel()),
            "stream": torch.cuda.current_stream()}


def _algebra_run(s, c):
    d, st = s["dev"], s["stream"]
    d.permute(s["ext"], s["o2n"], s["x"], s["z"], stream=st)                                      # z = perm(x)
    d.add_sub(False, [1, 2, 3, 4], s["rlab"], s["ext"], s["w"], s["y"], s["x"], stream=st)        # w = y + perm(x)
    d.scale_copy(s["u"], s["w"], -0.5, stream=st)                                                 # u = -0.5 w
    d.add_scaled(s["u"], s["z"], 0.25, stream=st)                                                 # u += 0.25 z
    d.slice_block(s["w"], s["out"], s["s"], s["sub"], s["beg"], stream=st)                        # s = w(sub-block)
    d.insert_block(s["v"], s["out"], s["s"], s["sub"], s["beg"], stream=st)                       # v(sub-block) = s
    return {"z": s["z"], "w": s["w"], "u": s["u"], "s": s["s"], "v": s["v"], "norm2": d.norm2(s["u"], stream=st)}


def _algebra_exact(c, seed):
    ext, o2n, out, sub, beg = _algebra_shapes(c)
    x, y = _algebra_data(c, seed)
    inv = [o2n.index(p + 1) for p in range(4)]  # index of x at position p of the result
    z = x.view(*reversed(ext)).permute(*[3 - inv[3 - q] for q in range(4)]).contiguous()
    w = y.view(*reversed(out)) + z
    u = -0.5 * w + 0.25 * z
    at = tuple(slice(b, b + n) for b, n in zip(reversed(beg), reversed(sub)))
    v = torch.zeros_like(w)
    v[at] = w[at]
    return {"z": z.reshape(-1), "w": w.reshape(-1), "u": u.reshape(-1), "s": w[at].reshape(-1), "v": v.reshape(-1),
            "norm2": float((u * u).sum())}


def _algebra_work(c):
    ext, _, _, sub, _ = _algebra_shapes(c)
    # permute 16, permuted add 24, scaled copy 16, accumulate 24, norm 8 bytes an element; slice and insert 16 each
    return {"bytes": 88 * _size(ext) + 32 * _size(sub), "flops": 6 * _size(ext)}


# ------------------------------------------------------------------ energy
def _energy_shapes(c):
    ext = [c["v"], c["o"], c["w"], c["o"], c["v"], c["o"]][:c["rank"]]
    segs = [c["o"], c["v"], c["w"]]
    return ext, segs, [2, 1, 3, 1, 2, 1][:c["rank"]]


def _energy_data(c, seed):
    ext, segs, _ = _energy_shapes(c)
    w = torch.empty(_size(ext), dtype=torch.float64, device="cuda").normal_(0.0, 0.05, generator=_generator(seed, 41))
    rng = np.random.default_rng(seed)
    return w, np.concatenate([rng.uniform(-2.0, -0.5, segs[0]), rng.uniform(0.2, 5.0, segs[1] + segs[2])])


def _energy_prepare(c, seed):
    import aces4_gb300 as a4

    a4.device.init()
    ext, segs, iv = _energy_shapes(c)
    w, e = _energy_data(c, seed)
    return {"dev": a4.device, "ext": ext, "segs": segs, "iv": iv, "w": w, "d": torch.zeros_like(w), "n": len(e),
            "fock": torch.from_numpy(np.diag(e).ravel(order="F").copy()).cuda(),
            "esum": torch.zeros(1, dtype=torch.float64, device="cuda"), "stream": torch.cuda.current_stream()}


def _energy_run(s, c):
    d, st, e1 = s["dev"], s["stream"], [s["n"], s["n"]]
    d.scale_copy(s["d"], s["w"], 1.0, stream=st)
    d.energy_denominator(s["iv"], s["ext"], s["d"], e1, s["fock"], s["segs"], stream=st)
    s["esum"].zero_()
    d.energy_contract(s["iv"], s["ext"], s["w"], e1, s["fock"], s["segs"], 1.0, s["esum"], stream=st)
    return {"d": s["d"], "esum": s["esum"]}


def _energy_exact(c, seed):
    ext, segs, iv = _energy_shapes(c)
    w, e = _energy_data(c, seed)
    ev = torch.from_numpy(e).cuda()
    at = [0, 0, segs[0], segs[0] + segs[1]]
    term = lambda q: ev[at[iv[q]]:at[iv[q]] + ext[q]].view(*[ext[q] if p == q else 1 for p in reversed(range(len(ext)))])
    eps = term(1) + term(3) + (term(5) if c["rank"] == 6 else 0.0) - term(0) - term(2) - (term(4) if c["rank"] == 6 else 0.0)
    x = w.view(*reversed(ext))
    d = x / eps
    return {"d": d.reshape(-1), "esum": (x * d).sum().view(1)}


def _energy_work(c):
    n = _size(_energy_shapes(c)[0])
    return {"bytes": 40 * n, "flops": 6 * n}  # copy 16, denominators 16, energy 8 bytes an element


# ------------------------------------------------------------------ sweep
def _sweep_segs(c):
    return _segments(c["v"], c["vlo"], c["vhi"], c["structure"]), _even(c["o"], c["oseg"])


def _sweep_data(c, seed):
    vs, os_ = _sweep_segs(c)
    segs = [vs, os_, vs, os_]
    new, old = _Array(segs, _all(segs)), _Array(segs, _all(segs))
    new.buf.normal_(0.0, 0.05, generator=_generator(seed, 51))
    old.buf.normal_(0.0, 0.05, generator=_generator(seed, 52))
    rng = np.random.default_rng(seed)
    return new, old, np.concatenate([rng.uniform(-2.0, -0.5, c["o"]), rng.uniform(0.2, 5.0, c["v"])])


def _sweep_prepare(c, seed):
    import aces4_gb300 as a4

    a4.device.init()
    vs, os_ = _sweep_segs(c)
    new, old, e = _sweep_data(c, seed)
    segs = [vs, os_, vs, os_]
    err, nxt = _Array(segs, _all(segs)), _Array(segs, _all(segs))
    calls = []
    for k in _all(segs):
        p = (k[2], k[3], k[0], k[1])
        iv = [len(os_) + 1 + k[0], 1 + k[1], len(os_) + 1 + k[2], 1 + k[3]]
        calls.append((iv, new.ext(k), new.block(k), new.block(p), old.block(k), old.block(p), err.block(k), nxt.block(k)))
    return {"dev": a4.device, "calls": calls, "new": new, "old": old, "err": err, "next": nxt, "n": len(e), "segs": os_ + vs,
            "fock": torch.from_numpy(np.diag(e).ravel(order="F").copy()).cuda(),
            "norm2": torch.zeros(1, dtype=torch.float64, device="cuda"), "stream": torch.cuda.current_stream()}


def _sweep_run(s, c):
    s["norm2"].zero_()
    for x in s["calls"]:
        s["dev"].update_t2(*x, [s["n"], s["n"]], s["fock"], s["segs"], s["norm2"], stream=s["stream"])
    return {"err": s["err"].buf, "next": s["next"].buf, "norm2": s["norm2"]}


def _sweep_exact(c, seed):
    vs, os_ = _sweep_segs(c)
    new, old, e = _sweep_data(c, seed)
    segs = [vs, os_, vs, os_]
    err, nxt = _Array(segs, _all(segs)), _Array(segs, _all(segs))
    ev = torch.from_numpy(e).cuda()
    at = np.concatenate([[0], np.cumsum(os_ + vs)])
    for k in _all(segs):
        p = (k[2], k[3], k[0], k[1])
        x = new.ext(k)
        term = lambda q, s: ev[at[s]:at[s] + x[q]].view(*[x[q] if r == q else 1 for r in reversed(range(4))])
        no = len(os_)
        eps = term(1, k[1]) + term(3, k[3]) - term(0, no + k[0]) - term(2, no + k[2])
        t = new.tensor(p).permute(2, 3, 0, 1) + new.tensor(k)
        t1 = old.tensor(p).permute(2, 3, 0, 1) + old.tensor(k)
        err.tensor(k).copy_(-0.5 * (t1 - t / eps))
        nxt.tensor(k).copy_((0.5 * t) / eps)
    return {"err": err.buf, "next": nxt.buf, "norm2": (err.buf * err.buf).sum().view(1)}


def _sweep_work(c):
    n = c["v"] ** 2 * c["o"] ** 2
    return {"bytes": 32 * n, "flops": 9 * n}  # both amplitude arrays read, both results written


# ------------------------------------------------------------------ the kinds
_KINDS = {
    "pair": (_pair_prepare, _pair_run, _pair_exact, _pair_work),
    "step": (_step_prepare, _step_run, _step_exact, _step_work),
    "loop": (_loop_prepare, _loop_run, _loop_exact, _loop_work),
    "triples": (_triples_prepare, _triples_run, _triples_exact, _triples_work),
    "algebra": (_algebra_prepare, _algebra_run, _algebra_exact, _algebra_work),
    "energy": (_energy_prepare, _energy_run, _energy_exact, _energy_work),
    "sweep": (_sweep_prepare, _sweep_run, _sweep_exact, _sweep_work),
}


def prepare(case, seed):
    return _KINDS[case["kind"]][0](case, seed) | {"case": case}


def run(state):
    return _KINDS[state["case"]["kind"]][1](state, state["case"])


def exact(case, seed):
    return _KINDS[case["kind"]][2](case, seed)


def work(case):
    return _KINDS[case["kind"]][3](case)
