"""Performance cases of the force library: the calls a block-step driver makes.

Every case goes through the C ABI with host arrays, as the Fortran driver
passes its common blocks (one ctypes call per library call, arguments built
once in ``prepare``).  Kinds of case:

* ``regular``   one regular block: ``gpunb_send_`` of the predicted bodies, then
  ``gpunb_regf_`` over the active ones in calls of up to 1,024 (the driver's
  chunk);
* ``resident``  the same block with the Hermite state kept on the device:
  ``nb6_predict_send_``, then ``gpunb_regf_``;
* ``ensemble``  one regular block of many small clusters together:
  ``nb6_irr_predict_send_``, then ``nb6_regf_seg_``;
* ``potential`` ``gpupot_`` for an energy output, the whole set or one rank's
  share of it;
* ``irregular`` ``irr_simd_firr_vec_`` over resident records and lists;
* ``training``  one epoch of the learned neighbour radius.

The libraries keep one state per process, so a case whose bodies stay on the
device opens them for several states' bodies and gives each its own range of
addresses.
"""
import ctypes as C
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "nbody6ppgpu-beijing_b200"))
from nb6b200 import load_cdll  # noqa: E402
from nb6b200 import mlp as mlp_api  # noqa: E402

CHUNK = 1024          # active bodies per gpunb_regf_ call
LMAX, NNBMAX = 512, 400
ILMAX = 256           # row length of the irregular lists
NNBOPT = 50           # neighbours a body is driven to have
SLOTS = 4             # resident states at a time
TIME = 0.5            # block time of the resident cases


def listed():
    return [
        # a late block of a small cluster: seven bodies due, latency is all
        {"name": "regular-1k-few", "kind": "regular", "n": 1024, "ni": 7, "model": "plummer", "m_flag": 0},
        # an ordinary block of a mid-size cluster with a mass spectrum
        {"name": "regular-16k-massflag", "kind": "regular", "n": 16384, "ni": 531, "model": "plummer", "m_flag": 1},
        # the initial forces: every body active, 64 calls against one j set
        {"name": "regular-64k-all", "kind": "regular", "n": 65536, "ni": 65536, "model": "plummer", "m_flag": 0},
        # a large block of the King N = 1M cluster (5% of its stars in binaries' c.m. bodies)
        {"name": "regular-king1m", "kind": "regular", "n": 996147, "ni": 8192, "model": "king", "m_flag": 0},
        # a small block of a large cluster, its state resident on the device
        {"name": "resident-king500k-few", "kind": "resident", "n": 500009, "ni": 37, "model": "king", "m_flag": 0},
        # a regular block of 64 clusters of 512 to 8,192 bodies, a tenth of them due
        {"name": "ensemble-64", "kind": "ensemble", "clusters": 64, "nmin": 512, "nmax": 8192, "active": 0.1},
        # energy output of a small cluster
        {"name": "potential-5k", "kind": "potential", "n": 5000, "i0": 0, "ni": 5000, "model": "plummer"},
        # one of four ranks' share of the energy output of a mid-size cluster
        {"name": "potential-rank-131k", "kind": "potential", "n": 131071, "i0": 32768, "ni": 32767, "model": "plummer"},
        # energy output of a large cluster on one GPU
        {"name": "potential-king249k", "kind": "potential", "n": 249036, "i0": 0, "ni": 249036, "model": "king"},
        # a typical irregular block: a hundred bodies of a small cluster
        {"name": "irregular-16k-few", "kind": "irregular", "n": 16384, "ni": 101, "model": "plummer"},
        # a large irregular block of a large cluster
        {"name": "irregular-131k-many", "kind": "irregular", "n": 131072, "ni": 32768, "model": "king"},
        # one epoch of the radius model over samples of a few clusters
        {"name": "training-32k", "kind": "training", "samples": 32768, "batch": 1024},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["regular", "regular", "regular", "resident", "ensemble", "potential", "potential",
                       "irregular", "irregular", "training"])
    model = rng.choice(["plummer", "king"])
    if kind in ("regular", "resident"):
        n = _log(rng, 700, 990000 if kind == "regular" else 500000)
        return {"kind": kind, "n": n, "ni": _log(rng, 1, min(n, 8191)), "model": model,
                "m_flag": rng.choice([0, 0, 1])}
    if kind == "ensemble":
        nmin = _log(rng, 300, 1500)
        return {"kind": kind, "clusters": _log(rng, 3, 64), "nmin": nmin, "nmax": _log(rng, nmin + 100, 8192),
                "active": round(math.exp(rng.uniform(math.log(0.005), 0.0)), 4)}
    if kind == "potential":
        n = _log(rng, 700, 240000)
        if rng.random() < 0.5:
            return {"kind": kind, "n": n, "i0": 0, "ni": n, "model": model}
        ranks = rng.randint(2, 8)
        i0 = n // ranks * rng.randrange(ranks)
        return {"kind": kind, "n": n, "i0": i0, "ni": min(n // ranks, n - i0), "model": model}
    if kind == "irregular":
        n = _log(rng, 1000, 130000)
        return {"kind": kind, "n": n, "ni": _log(rng, 1, min(n, 32000)), "model": model}
    return {"kind": kind, "samples": _log(rng, 2000, 32000), "batch": rng.choice([256, 512, 1000, 1024, 2048])}


# ---------------------------------------------------------------- inputs
@functools.lru_cache(maxsize=None)
def _king(w0=6.0):
    """King (1966) model: radius, depth W, density and enclosed mass on a grid
    (G M = 1, virial radius 1), and the 1-D dispersion."""
    erf = math.erf

    def rho(w):
        return 0.0 if w <= 0 else math.exp(w) * erf(math.sqrt(w)) - math.sqrt(4 * w / math.pi) * (1 + 2 * w / 3)

    rho0, h, r, w, u = rho(w0), 0.01, 0.0, w0, 0.0
    rows = [(r, w)]

    def f(r, w, u):
        return u, (-3.0 if r == 0 else -9.0 * rho(w) / rho0 - 2.0 * u / r)

    while w > 0 and r < 100:
        a1, b1 = f(r, w, u)
        a2, b2 = f(r + h / 2, w + h / 2 * a1, u + h / 2 * b1)
        a3, b3 = f(r + h / 2, w + h / 2 * a2, u + h / 2 * b2)
        a4, b4 = f(r + h, w + h * a3, u + h * b3)
        r, w, u = r + h, w + h / 6 * (a1 + 2 * a2 + 2 * a3 + a4), u + h / 6 * (b1 + 2 * b2 + 2 * b3 + b4)
        rows.append((r, max(w, 0.0)))
    q = np.array(rows)
    r, w = q[:, 0], q[:, 1]
    d = np.array([rho(x) for x in w])
    shell = 4 * np.pi * r * r * d
    m = np.concatenate([[0.0], np.cumsum(0.5 * (shell[1:] + shell[:-1]) * np.diff(r))])
    dm, rm, mm = np.diff(m), 0.5 * (r[1:] + r[:-1]), 0.5 * (m[1:] + m[:-1])
    pot = np.sum(mm * dm / rm)
    rv = 0.5 * m[-1] ** 2 / pot
    sig = np.sqrt(np.minimum(w / 3.0, 1.0) + 1e-6)
    sig *= 0.5 ** 0.5 / math.sqrt(3.0 * np.sum(0.5 * (sig[1:] ** 2 + sig[:-1] ** 2) * dm) / m[-1])
    return r / rv, d / m[-1] * rv ** 3, m / m[-1], sig


def _cluster(n, model, rng, spectrum=True):
    """mass, pos, vel, neighbour radius and regular step of n bodies in
    N-body units; radii scatter about the one that holds NNBOPT neighbours."""
    u = rng.random(n) * 0.999 + 1e-9
    if model == "king":
        gr, gd, gm, gs = _king()
        r = np.interp(u, gm, gr)
        dens, sig = np.interp(r, gr, gd), np.interp(r, gr, gs)
    else:
        a = 3.0 * np.pi / 16.0
        q = np.minimum((u ** (-2.0 / 3.0) - 1.0) ** -0.5, 10.0)
        r = a * q
        dens = 3.0 / (4.0 * np.pi * a ** 3) * (1 + q * q) ** -2.5
        sig = np.sqrt(1.0 / (6.0 * a) / np.sqrt(1 + q * q))
    z = 1.0 - 2.0 * rng.random(n)
    ph = 2.0 * np.pi * rng.random(n)
    s = np.sqrt(np.maximum(0.0, 1.0 - z * z))
    pos = np.stack([r * s * np.cos(ph), r * s * np.sin(ph), r * z], axis=1)
    vel = rng.standard_normal((n, 3)) * sig[:, None]
    # two-part power law between 0.08 and 100 Msun (slopes 1.3 and 2.3 about 0.5)
    if spectrum:
        x, p = rng.random(n), rng.random(n) < 0.72
        lo = (0.08 ** -0.3 + x * (0.5 ** -0.3 - 0.08 ** -0.3)) ** (-1 / 0.3)
        hi = (0.5 ** -1.3 + x * (100.0 ** -1.3 - 0.5 ** -1.3)) ** (-1 / 1.3)
        mass = np.where(p, lo, hi)
        mass /= mass.sum()
    else:
        mass = np.full(n, 1.0 / n)
    nnb = min(NNBOPT, max(n // 8, 2))
    rs = np.minimum((3.0 * nnb / (4.0 * np.pi * n * np.maximum(dens, 1e-3))) ** (1.0 / 3.0), 1.5)
    rs *= np.exp(0.06 * rng.standard_normal(n))
    dtr = 0.125 * 2.0 ** -np.ceil(np.log2(np.maximum(0.5 * sig / rs, 1.0)))
    return mass, pos, vel, rs, dtr


def _hermite(n, pos, rng):
    """F = a / 2, FDOT = adot / 6 and the times of the last steps before TIME."""
    r2 = (pos * pos).sum(1)[:, None]
    f = -0.5 * pos / (r2 + 0.3) ** 1.5
    fdot = 0.02 * rng.standard_normal((n, 3))
    t0 = TIME - 2.0 ** -rng.integers(5, 12, n) * rng.integers(0, 2, n)
    return f, fdot, t0


def _inputs(case, seed):
    """Host arrays of a case, from the seed alone."""
    rng = np.random.default_rng([seed, 77])
    d = {}
    kind = case["kind"]
    if kind == "training":
        k = case["samples"]
        x = np.empty((k, 5), dtype=np.float32)
        nnb = rng.poisson(NNBOPT * np.exp(0.3 * rng.standard_normal(k))) + 1
        lr = -3.0 + 0.7 * rng.standard_normal(k)
        x[:, 0], x[:, 1], x[:, 2] = np.log1p(nnb), lr, np.log1p(nnb) - 3.0 * lr
        x[:, 3] = 0.5 * rng.standard_normal(k)
        x[:, 4] = rng.integers(4, 10, k)
        d["x"] = x
        d["y"] = (np.log(NNBOPT / nnb) / 3 + 0.02 * x[:, 3] + 0.05 * rng.standard_normal(k)).astype(np.float32)
        w = np.zeros(4621, dtype=np.float32)
        for lo, hi, fan in ((0, 320, 5), (384, 4480, 64), (4544, 4608, 64)):
            w[lo:hi] = rng.standard_normal(hi - lo) * math.sqrt(2.0 / fan)
        w[4614:4619] = 1.0
        w[4620] = 1.0
        d["model"] = w
        return d
    if kind == "ensemble":
        ns = np.exp(np.random.default_rng(case["clusters"]).uniform(
            math.log(case["nmin"]), math.log(case["nmax"]), case["clusters"])).astype(int)
        parts = [_cluster(int(k), "plummer", rng) for k in ns]
        d["m"], d["x"], d["v"], rs, dtr = (np.concatenate([p[q] for p in parts]) for q in range(5))
        d["j0"] = np.concatenate([[0], np.cumsum(ns)]).astype(np.int32)
        act, seg = [], []
        for c, k in enumerate(ns):
            a = np.sort(rng.choice(int(k), max(1, int(round(case["active"] * k))), replace=False))
            act.append(a + d["j0"][c])
            seg.append(np.full(len(a), c))
        d["act"] = np.concatenate(act)
        d["iseg"] = np.concatenate(seg).astype(np.int32)
    else:
        n = case["n"]
        d["m"], d["x"], d["v"], rs, dtr = _cluster(n, case["model"], rng)
        if kind == "potential":
            return d
        d["act"] = np.sort(rng.choice(n, case["ni"], replace=False))
    if kind != "regular":
        d["f"], d["fdot"], d["t0"] = _hermite(len(d["m"]), d["x"], rng)
    act = d["act"]
    d["rs"] = rs[act]
    d["h2"] = rs[act] ** 2 / (d["m"].mean() if case.get("m_flag") else 1.0)
    d["dtr"] = dtr[act]
    d["xi"], d["vi"] = d["x"][act], d["v"][act]
    if kind in ("resident", "ensemble"):   # the active bodies are corrected to TIME on the host
        d["t0"][act] = TIME
    return {k: np.ascontiguousarray(v) for k, v in d.items()}


def _lists(d):
    """Neighbour ids (0-based, ascending, without the body itself) of the
    active bodies: a flat array and its offsets."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    x = torch.from_numpy(d["x"]).to(dev).T.contiguous()
    act, h2 = torch.from_numpy(d["act"]).to(dev), torch.from_numpy(d["rs"] ** 2).to(dev)
    ids, counts = [], []
    step = max(1, (1 << 26) // x.shape[1])
    for a in range(0, len(act), step):
        i = act[a:a + step]
        r2 = (x[0][None] - x[0][i][:, None]).square_()
        for k in (1, 2):
            r2 += (x[k][None] - x[k][i][:, None]).square_()
        near = r2 < h2[a:a + step, None]
        near[torch.arange(len(i), device=dev), i] = False
        row, col = near.nonzero(as_tuple=True)
        first = torch.zeros(len(i) + 1, dtype=torch.int64, device=dev)
        first[1:] = torch.bincount(row, minlength=len(i)).cumsum(0)
        keep = torch.arange(len(row), device=dev) - first[row] < ILMAX - 1
        ids.append(col[keep].to(torch.int32))
        counts.append(torch.bincount(row[keep], minlength=len(i)))
    counts = torch.cat(counts).cpu().numpy()
    return torch.cat(ids).cpu().numpy(), np.concatenate([[0], np.cumsum(counts)])


# ---------------------------------------------------------------- the library's session
def _fn(name, nargs):
    """The library call `name` on nargs addresses."""
    return C.CFUNCTYPE(None, *[C.c_void_p] * nargs)((name, load_cdll()))


def _p(a):
    return a.ctypes.data


class _Session:
    """Opens the libraries for one case's sizes; hands out ranges of the
    resident addresses."""

    def __init__(self):
        self.key, self.open, self.free = None, [], []

    def use(self, case, n):
        key = tuple(sorted((k, v) for k, v in case.items() if k != "name"))
        if key == self.key:
            return
        one = np.zeros(1, dtype=np.int32)
        for name, nargs in self.open:
            _fn(name, nargs)(*[_p(one)] * nargs)
        self.key, self.open, self.free = key, [], list(range(SLOTS))[::-1]
        kind = case["kind"]
        nb, many, lm = (np.array([v], dtype=np.int32) for v in (n, SLOTS * n, ILMAX))
        if kind in ("regular", "resident", "ensemble"):
            _fn("gpunb_open_", 2)(_p(nb), _p(one))
            self.open.append(("gpunb_close_", 0))
        if kind == "resident":
            _fn("nb6_state_open_", 1)(_p(many))
            z = np.zeros((SLOTS * n, 3))
            _fn("nb6_state_set_", 7)(_p(many), _p(z), _p(z), _p(z), _p(z), _p(z), _p(z))
            self.open.append(("nb6_state_close_", 0))
        if kind in ("irregular", "ensemble"):
            _fn("irr_simd_open_", 3)(_p(many), _p(lm), _p(one))
            self.open.append(("irr_simd_close_", 1))


_S = _Session()


class State:
    """The arrays, calls and outputs of one prepared case."""

    def __init__(self):
        self.slot = self.key = None
        self.calls, self.out, self.keep = [], {}, []

    def take_slot(self):
        self.slot, self.key = _S.free.pop(), _S.key

    def __del__(self):
        if self.slot is not None and self.key == _S.key:
            _S.free.append(self.slot)

    def arr(self, v, dtype):
        a = np.ascontiguousarray(v, dtype=dtype)
        self.keep.append(a)
        return a

    def i32(self, v):
        return _p(self.arr(np.reshape(v, -1), np.int32))

    def f64(self, v):
        return _p(self.arr(v, np.float64))

    def call(self, name, *args):
        self.calls.append((_fn(name, len(args)), args))


def _force_outputs(s, ni):
    s.out = {"acc": np.zeros((ni, 3)), "jrk": np.zeros((ni, 3)), "pot": np.zeros(ni),
             "list": np.zeros((ni, LMAX), dtype=np.int32)}


def _regf_calls(s, d, case):
    ni = len(d["act"])
    _force_outputs(s, ni)
    o = s.out
    lmax, nnbmax, mf = s.i32(LMAX), s.i32(NNBMAX), s.i32(case["m_flag"])
    for a in range(0, ni, CHUNK):
        k = slice(a, min(a + CHUNK, ni))
        s.call("gpunb_regf_", s.i32(k.stop - a), s.f64(d["h2"][k]), s.f64(d["dtr"][k]), s.f64(d["xi"][k]),
               s.f64(d["vi"][k]), _p(o["acc"][k]), _p(o["jrk"][k]), _p(o["pot"][k]), lmax, nnbmax,
               _p(o["list"][k]), mf)


def _set_records(s, d, first):
    """irr_simd_set_jp_ of every body, from 1-based address `first`."""
    n = len(d["m"])
    fn = _fn("irr_simd_set_jp_", 7)
    addr = np.arange(first, first + n, dtype=np.int32)
    base = [_p(addr)] + [_p(d[k]) for k in ("x", "v", "f", "fdot", "m", "t0")]
    step = (4, 24, 24, 24, 24, 8, 8)
    for k in range(n):
        fn(*[b + t * k for b, t in zip(base, step)])
    return addr


def prepare(case, seed):
    d = _inputs(case, seed)
    kind = case["kind"]
    s = State()
    s.kind = kind
    if kind == "training":
        s.d, s.batch = d, case["batch"]
        return s
    n = len(d["m"])
    _S.use(case, n)
    if kind == "regular":
        s.call("gpunb_send_", s.i32(n), s.f64(d["m"]), s.f64(d["x"]), s.f64(d["v"]))
        _regf_calls(s, d, case)
    elif kind == "resident":
        s.take_slot()
        first = s.slot * n + 1
        _fn("nb6_state_update_", 8)(s.i32(n), s.i32(np.arange(first, first + n)), s.f64(d["m"]), s.f64(d["t0"]),
                                    s.f64(d["x"]), s.f64(d["v"]), s.f64(d["f"]), s.f64(d["fdot"]))
        s.call("nb6_predict_send_", s.f64([TIME]), s.i32(first), s.i32(n))
        _regf_calls(s, d, case)
    elif kind == "ensemble":
        s.take_slot()
        _set_records(s, d, s.slot * n + 1)
        j0 = d["j0"]
        nseg = len(j0) - 1
        s.call("nb6_irr_predict_send_", s.f64([TIME]), s.i32(nseg), s.i32(j0[:-1] + s.slot * n + 1),
               s.i32(np.diff(j0)))
        ni = len(d["act"])
        _force_outputs(s, ni)
        o = s.out
        s.call("nb6_regf_seg_", s.i32(ni), s.i32(d["iseg"]), s.f64(d["h2"]), s.f64(d["dtr"]), s.f64(d["xi"]),
               s.f64(d["vi"]), _p(o["acc"]), _p(o["jrk"]), _p(o["pot"]), s.i32(LMAX), s.i32(NNBMAX),
               _p(o["list"]), s.i32(0), s.i32(nseg), s.i32(j0))
    elif kind == "potential":
        s.out = {"pot": np.zeros(case["ni"])}
        s.call("gpupot_", s.i32(0), s.i32(case["i0"] + 1), s.i32(case["ni"]), s.i32(n), s.f64(d["m"]),
               s.f64(d["x"]), _p(s.out["pot"]))
    else:
        s.take_slot()
        addr = _set_records(s, d, s.slot * n + 1)
        ids, off = _lists(d)
        rows = np.zeros(len(ids) + len(off) + 8, dtype=np.int32)   # [nnb, ids] one after the other
        start = off[:-1] + np.arange(len(off) - 1)
        rows[start] = np.diff(off)
        rows[np.arange(len(ids)) + np.repeat(np.arange(1, len(off)), np.diff(off))] = ids + addr[0]
        act = addr[d["act"]]
        fn, pa, pr = _fn("irr_simd_set_list_", 2), _p(act), _p(rows)
        for k, r in enumerate(start.tolist()):
            fn(pa + 4 * k, pr + 4 * r)
        ni = len(act)
        s.first = int(addr[0])
        s.out = {"acc": np.zeros((ni, 3)), "jrk": np.zeros((ni, 3)), "nnbid": np.zeros(ni, dtype=np.int32)}
        s.call("irr_simd_firr_vec_", s.f64([TIME]), s.i32(ni), s.i32(act), _p(s.out["acc"]), _p(s.out["jrk"]),
               _p(s.out["nnbid"]))
    return s


def run(s):
    if s.kind == "training":
        mlp_api.set_model(s.d["model"])
        loss = mlp_api.train(s.d["x"], s.d["y"], epochs=1, batch=s.batch, lr=2e-3, seed=3)
        return {"loss": loss, "model": mlp_api.get_model()}
    for fn, args in s.calls:
        fn(*args)
    if s.kind == "irregular":   # ids within the state's own bodies, whatever addresses it was given
        return dict(s.out, nnbid=s.out["nnbid"] - s.first)
    return s.out


def work(case):
    """Bytes: bodies and active rows in, forces and lists out, once each.
    Operations: 60 per force and jerk pair, 11 per potential pair."""
    kind = case["kind"]
    if kind == "training":
        return {"bytes": 24 * case["samples"], "flops": 6 * 4544 * case["samples"]}
    if kind == "potential":
        return {"bytes": 32 * case["n"] + 8 * case["ni"], "flops": 11 * case["n"] * case["ni"]}
    out = 64 + 56 + 4 * (NNBOPT + 1)
    if kind == "ensemble":
        ns = np.exp(np.random.default_rng(case["clusters"]).uniform(
            math.log(case["nmin"]), math.log(case["nmax"]), case["clusters"])).astype(int)
        ni = np.maximum(1, np.round(case["active"] * ns))
        return {"bytes": float(112 * ns.sum() + out * ni.sum()), "flops": float(60 * (ni * ns).sum())}
    n, ni = case["n"], case["ni"]
    if kind == "irregular":
        e = ni * min(NNBOPT, max(n // 8, 2))
        return {"bytes": 112 * min(n, e + ni) + 4 * e + 56 * ni, "flops": 60 * e}
    return {"bytes": (56 if kind == "regular" else 112) * n + out * ni, "flops": 60 * n * ni}


# ---------------------------------------------------------------- the same in 64 bits
def _predict(d, dev):
    t = {k: torch.from_numpy(d[k]).to(dev) for k in ("x", "v", "f", "fdot", "t0")}
    h = (TIME - t["t0"])[:, None]
    return ((t["fdot"] * h + t["f"]) * h + t["v"]) * h + t["x"], (t["fdot"] * 1.5 * h + t["f"]) * 2 * h + t["v"]


def _regular(m, x, v, xi, vi, h2, dtr, m_flag):
    """Regular acceleration, jerk and potential of (xi, vi) from (m, x, v)."""
    x, v = x.T.contiguous(), v.T.contiguous()
    out = torch.zeros((len(h2), 7), dtype=torch.float64, device=m.device)
    step = max(1, (1 << 22) // len(m))
    for a in range(0, len(h2), step):
        k = slice(a, a + step)
        dx = [x[c][None] - xi[k, c][:, None] for c in range(3)]
        dv = [v[c][None] - vi[k, c][:, None] for c in range(3)]
        r2 = dx[0] * dx[0] + dx[1] * dx[1] + dx[2] * dx[2]
        p = [dx[c] + dtr[k][:, None] * dv[c] for c in range(3)]
        near = torch.minimum(r2, p[0] * p[0] + p[1] * p[1] + p[2] * p[2]) < (
            h2[k][:, None] * m[None] if m_flag else h2[k][:, None])
        ri = torch.where(near, 0.0, r2.rsqrt())
        mr = m[None] * ri
        ri2 = ri * ri
        mr3 = mr * ri2
        al = -3.0 * ri2 * (dx[0] * dv[0] + dx[1] * dv[1] + dx[2] * dv[2])
        for c in range(3):
            out[k, c] = (mr3 * dx[c]).sum(1)
            out[k, 3 + c] = (mr3 * (dv[c] + al * dx[c])).sum(1)
        out[k, 6] = mr.sum(1)
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "training":
        return None
    d = _inputs(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    m = torch.from_numpy(d["m"]).to(dev)
    if kind == "potential":
        x = torch.from_numpy(d["x"]).to(dev).T.contiguous()
        pot = torch.zeros(case["ni"], dtype=torch.float64, device=dev)
        step = max(1, (1 << 22) // len(m))
        for a in range(0, case["ni"], step):
            i = torch.arange(case["i0"] + a, case["i0"] + min(a + step, case["ni"]), device=dev)
            r2 = (x[0][None] - x[0][i][:, None]).square_()
            for k in (1, 2):
                r2 += (x[k][None] - x[k][i][:, None]).square_()
            pot[a:a + step] = torch.where(r2 > 0, r2.rsqrt(), 0.0) @ m
        return {"pot": pot}
    if kind == "irregular":
        x, v = _predict(d, dev)
        ids, off = (torch.from_numpy(a).to(dev).long() for a in _lists(d))
        act = torch.from_numpy(d["act"]).to(dev)
        row = torch.repeat_interleave(torch.arange(len(act), device=dev), off.diff())
        dx, dv = x[ids] - x[act[row]], v[ids] - v[act[row]]
        r2 = (dx * dx).sum(1, keepdim=True)
        mr3 = m[ids][:, None] / (r2 * r2.sqrt())
        j = mr3 * (dv - 3.0 * (dx * dv).sum(1, keepdim=True) / r2 * dx)
        zero = torch.zeros((len(act), 3), dtype=torch.float64, device=dev)
        return {"acc": zero.index_add(0, row, mr3 * dx), "jrk": zero.index_add(0, row, j), "nnbid": None}
    xi, vi, h2, dtr = (torch.from_numpy(d[k]).to(dev) for k in ("xi", "vi", "h2", "dtr"))
    x, v = (torch.from_numpy(d[k]).to(dev) for k in ("x", "v")) if kind == "regular" else _predict(d, dev)
    if kind == "ensemble":
        seg = torch.from_numpy(d["iseg"]).to(dev)
        out = torch.cat([_regular(m[a:b], x[a:b], v[a:b], xi[seg == c], vi[seg == c], h2[seg == c],
                                  dtr[seg == c], 0)
                         for c, (a, b) in enumerate(zip(d["j0"][:-1].tolist(), d["j0"][1:].tolist()))])
    else:
        out = _regular(m, x, v, xi, vi, h2, dtr, case["m_flag"])
    return {"acc": out[:, :3], "jrk": out[:, 3:6], "pot": out[:, 6], "list": None}
