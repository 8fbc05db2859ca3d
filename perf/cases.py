"""The joins a user of this library runs, at the sizes they run them.

A case is a dict of plain values.  Four forms of use:

* "join"    two device-resident relations joined by name (join_device): the
            lazy hash and sort-merge joins
* "host"    two relations in ordinary (pageable) host memory joined by name
            (join), as a program that was linked against the CPU joins calls it
* "batch"   many independent window pairs joined by one call
            (batch_join_device)
* "stream"  two timestamped streams in pinned host memory joined in tumbling
            windows by an eager join (stream_join)

Relations hold 8-byte tuples, key << 32 | payload, payload = row number.  Keys:
"dense" R = a permutation of 1..n, S drawn from R's keys with Zipf skew theta
(a foreign key); "sparse" the same with the keys spread over all 32 bits (a
hashed or external identifier); "dup" both sides uniform over n / 4 values (an
equi-join of two non-unique columns).  Outputs are match counts and 64-bit
checksums, whole numbers.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import alliancedb_b200 as adb

LAZY = ("PRO", "RJ_st", "PRH", "PRHO", "NPO", "NPO_st", "m-way", "m-pass", "m-way+skew")
EAGER = ("SHJ_JM_NP", "SHJ_JB_NP", "SHJ_JBCR_NP", "PMJ_JM_NP")


def _join(name, algo, n_r, n_s, keys="dense", theta=0.0, kind="join"):
    return {"name": name, "kind": kind, "algo": algo, "n_r": n_r, "n_s": n_s, "keys": keys, "theta": theta}


def listed():
    return [
        # one small window joined by itself: latency and launches are everything
        _join("pro_4k", "PRO", 1 << 12, 1 << 12),
        # a small lookup table against a larger, ragged probe side
        _join("npo_50k_300k", "NPO", 50021, 300007, "sparse"),
        # the plain radix join of the benchmark's first configuration
        _join("pro_4m", "PRO", 1 << 22, 1 << 22),
        # an ordinary hash join on scattered 32-bit identifiers, ragged sizes
        _join("npo_3m_5m", "NPO", 3000017, 5000011, "sparse"),
        # an ordinary sort-merge join of two non-unique columns
        _join("mway_1m_dup", "m-way", 1000003, 1200007, "dup"),
        # the large configurations: PRO's headline size, and NPO and m-way under skew
        _join("pro_128m", "PRO", 1 << 27, 1 << 27),
        _join("npo_128m_zipf1", "NPO", 1 << 27, 1 << 27, theta=1.0),
        _join("mway_128m_zipf05", "m-way", 1 << 27, 1 << 27, theta=0.5),
        # the drop-in call: both relations in the caller's own memory
        _join("host_pro_16m", "PRO", 1 << 24, 1 << 24, kind="host"),
        # batched windows, sizes log-uniform in [2^10, 2^22] per side
        {"name": "batch_512", "kind": "batch", "windows": 512, "lo": 10.0, "hi": 22.0},
        # two streams of 1.6 M tuples/s in 1000 ms windows, four windows, eager hash join
        {"name": "shj_stream", "kind": "stream", "algo": "SHJ_JM_NP", "rate": 1600.0, "window_ms": 1000, "windows": 4},
        # the same streams, two windows, joined by the progressive sort-merge join
        {"name": "pmj_stream", "kind": "stream", "algo": "PMJ_JM_NP", "rate": 1600.0, "window_ms": 1000, "windows": 2},
    ]


def _logu(rng, lo, hi):
    return max(1, int(2.0 ** rng.uniform(lo, hi)))


def draw(rng):
    form = rng.random()
    if form < 0.6:
        keys = rng.choice(["dense", "sparse", "dup"])
        algo = rng.choice(LAZY)
        n_r = _logu(rng, 10, 27)
        # S of a like size, or many times larger or smaller
        n_s = min(1 << 27, max(1, int(n_r * 2.0 ** rng.uniform(-3, 3)))) | 1
        theta = 0.0 if keys == "dup" else rng.choice([0.0, 0.0, 0.5, 0.75, 1.0, 1.5])
        c = _join("", algo, n_r, n_s, keys, theta)
    elif form < 0.68:
        c = _join("", rng.choice(LAZY), _logu(rng, 12, 24), _logu(rng, 12, 24), rng.choice(["dense", "sparse"]),
                  kind="host")
    elif form < 0.82:
        hi = rng.uniform(13, 22)
        lo = rng.uniform(8, hi - 3)
        mean = (2.0 ** hi - 2.0 ** lo) / ((hi - lo) * math.log(2.0))
        windows = min(_logu(rng, 3, 12), int(2.0e8 / mean))
        c = {"kind": "batch", "windows": max(4, windows), "lo": lo, "hi": hi}
    else:
        rate = 2.0 ** rng.uniform(4, 10.6)
        c = {"kind": "stream", "algo": rng.choice(EAGER), "rate": rate, "window_ms": rng.choice([100, 250, 1000]),
             "windows": rng.randint(1, 4)}
    c.pop("name", None)
    return c


# --------------------------------------------------------------------------
# Inputs
# --------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed & 0x7FFFFFFF)


def _spread(k):
    """A bijection of 32-bit values: row identifiers scattered over all 32 bits."""
    m = 0xFFFFFFFF
    k = ((k ^ (k >> 16)) * 0x7FEB352D) & m
    k = ((k ^ (k >> 15)) * 0x846CA68B) & m
    return k ^ (k >> 16)


def _zipf(n, size, theta, g):
    """Ranks 0..n-1 with density ~ (rank + 1)^-theta (its continuous form, inverted)."""
    u = torch.rand(size, generator=g, device="cuda", dtype=torch.float64)
    if theta == 0.0:
        x = u * n
    elif theta == 1.0:
        x = torch.exp(u * math.log(n + 1.0)) - 1.0
    else:
        a = 1.0 - theta
        x = (u * ((n + 1.0) ** a - 1.0) + 1.0) ** (1.0 / a) - 1.0
    return x.to(torch.int64).clamp_(0, n - 1)


def _words(keys):
    return (keys << 32) | torch.arange(keys.numel(), device="cuda")


def _relations(c, seed):
    g = _gen(seed)
    n_r, n_s = c["n_r"], c["n_s"]
    if c["keys"] == "dup":
        top = max(1, n_r // 4)
        r = torch.randint(1, top + 1, (n_r,), generator=g, device="cuda")
        s = torch.randint(1, top + 1, (n_s,), generator=g, device="cuda")
    else:
        r = torch.randperm(n_r, generator=g, device="cuda") + 1
        if c["keys"] == "sparse":
            r = _spread(r)
        s = r[_zipf(n_r, n_s, c["theta"], g)]
    return _words(r), _words(s)


def _windows(c, seed):
    """Sizes and keys of the batch's windows: keys uniform over four times the
    window's size, a quarter of the windows Zipf(0.8) over that range with each
    side's own hot keys (the benchmark's batch: about one match per four tuples)."""
    rng = np.random.default_rng(seed)
    g = _gen(seed)
    w = c["windows"]
    sizes = [np.floor(2.0 ** rng.uniform(c["lo"], c["hi"], size=w)).astype(np.int64) for _ in range(2)]
    span = 4 * np.maximum(sizes[0], sizes[1])
    zipf = rng.random(w) < 0.25
    offs, keys, wins = [], [], []
    for n, mult, shift in zip(sizes, (2654435761, 2246822519), (17, 91)):
        off = np.concatenate([[0], np.cumsum(n)]).astype(np.uint64)
        win = torch.repeat_interleave(torch.arange(w, device="cuda"), torch.from_numpy(n).cuda())
        top = torch.from_numpy(span).cuda()[win]
        u = torch.rand(win.numel(), generator=g, device="cuda", dtype=torch.float64)
        z = ((u * ((top + 1.0) ** 0.2 - 1.0) + 1.0) ** 5.0 - 1.0).to(torch.int64)
        # the hot ranks anywhere in the range, other ones on each side
        z = (torch.minimum(z, top - 1) + shift) * mult % top
        f = torch.minimum((u * top).to(torch.int64), top - 1)
        keys.append(1 + torch.where(torch.from_numpy(zipf).cuda()[win], z, f))
        offs.append(off)
        wins.append(win)
    # payload = row number inside the window
    rels = [(k << 32) | (torch.arange(k.numel(), device="cuda") - torch.from_numpy(o.astype(np.int64)).cuda()[v])
            for k, o, v in zip(keys, offs, wins)]
    return rels, offs, wins


def _streams(c, seed):
    """Two timestamp-ordered streams, Poisson arrivals, every key four times on average per window."""
    rng = np.random.default_rng(seed)
    n = max(4, int(c["rate"] * c["window_ms"] * c["windows"]))
    space = max(1, int(c["rate"] * c["window_ms"]) * 2 // 3)
    end = c["window_ms"] * c["windows"] - 1
    out = []
    for _ in range(2):
        st = np.empty(n, dtype=adb.STREAM_TUPLE)
        ts = np.cumsum(rng.exponential(1.0 / c["rate"], size=n))
        st["ts_ms"] = np.minimum(ts, end).astype(np.uint64)
        st["key"] = rng.integers(1, space + 1, size=n, dtype=np.uint32)
        st["payload"] = np.arange(n, dtype=np.uint32)
        out.append(st)
    return out


def _pinned(a):
    buf = torch.empty(a.nbytes, dtype=torch.uint8, pin_memory=True)
    v = buf.numpy().view(a.dtype)
    v[:] = a
    return v, buf


def prepare(case, seed):
    kind = case["kind"]
    if kind == "join":
        r, s = _relations(case, seed)
        return {"kind": kind, "algo": case["algo"], "r": r, "s": s, "params": adb.default_params()}
    if kind == "host":
        r, s = (t.cpu().numpy().view(np.uint64) for t in _relations(case, seed))
        return {"kind": kind, "algo": case["algo"], "r": r, "s": s, "params": adb.default_params()}
    if kind == "batch":
        (r, s), (ro, so), _ = _windows(case, seed)
        torch.cuda.synchronize()   # batch_join_device takes no stream: its inputs are complete
        return {"kind": kind, "r": r, "s": s, "ro": ro, "so": so}
    (r, kr), (s, ks) = (_pinned(a) for a in _streams(case, seed))
    params = adb.default_params(window_size=case["window_ms"], nthreads=8, batch_tuples=max(1, int(case["rate"])))
    return {"kind": kind, "algo": case["algo"], "r": r, "s": s, "keep": (kr, ks), "params": params}


def run(state):
    kind = state["kind"]
    if kind == "join":
        r, s = state["r"], state["s"]
        out = adb.join_device(state["algo"], r.data_ptr(), r.numel(), s.data_ptr(), s.numel(), state["params"],
                              stream=torch.cuda.current_stream())
        return np.array([out.count, out.checksum], dtype=np.uint64)
    if kind == "host":
        out = adb.join(state["algo"], state["r"], state["s"], state["params"])
        return np.array([out.count, out.checksum], dtype=np.uint64)
    if kind == "batch":
        counts, sums, _ = adb.batch_join_device(state["r"].data_ptr(), state["ro"], state["s"].data_ptr(), state["so"])
        return {"counts": counts, "checksums": sums}
    wins = adb.stream_join(state["algo"], state["r"], state["s"], state["params"], max_windows=64)
    return np.array([(w.window_start_ms, w.n_r, w.n_s, w.count, w.checksum) for w in wins], dtype=np.uint64)


def work(case):
    """Every input tuple read once (8 bytes, 16 in a stream); the results are a
    few words.  The arithmetic is integer hashing: no floating-point operations."""
    kind = case["kind"]
    if kind in ("join", "host"):
        n, b = case["n_r"] + case["n_s"], 8
    elif kind == "stream":
        n, b = 2 * max(4, int(case["rate"] * case["window_ms"] * case["windows"])), 16
    else:   # mean of a log-uniform size, two sides
        lo, hi = case["lo"], case["hi"]
        mean = (2.0 ** hi - 2.0 ** lo) / ((hi - lo) * math.log(2.0))
        n, b = int(2 * mean * case["windows"]), 8
    return {"bytes": n * b, "flops": 0}


# --------------------------------------------------------------------------
# The joins' values from their definition
# --------------------------------------------------------------------------
def _i64(v):
    return v - (1 << 64) if v >> 63 else v


def _shr(z, k):
    return (z >> k) & ((1 << (64 - k)) - 1)


def _fmix(z):
    z = (z ^ _shr(z, 30)) * _i64(0xBF58476D1CE4E5B9)
    z = (z ^ _shr(z, 27)) * _i64(0x94D049BB133111EB)
    return z ^ _shr(z, 31)


def _exact_join(r, s, r_win=None, s_win=None, windows=1):
    """Per-window (count, checksum) of the equi-join of two arrays of tuple words."""
    low = 0xFFFFFFFF

    def key(t, w):
        k = _shr(t, 32)
        return k if w is None else (w << 32) | k

    rk, order = torch.sort(key(r, r_win))
    rs = r[order]
    counts = torch.zeros(windows, dtype=torch.int64, device="cuda")
    sums = torch.zeros(windows, dtype=torch.int64, device="cuda")
    part = 1 << 22
    for b in range(0, s.numel(), part):
        sv = s[b:b + part]
        wv = None if s_win is None else s_win[b:b + part]
        sk = key(sv, wv)
        lo = torch.searchsorted(rk, sk)
        n = torch.searchsorted(rk, sk, right=True) - lo
        half = _fmix(((sv & low) << 32) | _shr(sv, 32))
        ends = torch.cumsum(n, 0)
        at, total = 0, int(ends[-1])
        done = 0
        while at < sv.numel():      # at most about 2^27 matches at a time
            to = int(torch.searchsorted(ends, done + (1 << 27), right=True))
            to = min(max(to, at + 1), sv.numel())
            c = n[at:to]
            i = torch.repeat_interleave(torch.arange(at, to, device="cuda"), c)
            first = torch.cumsum(c, 0) - c
            j = lo[i] + torch.arange(i.numel(), device="cuda") - torch.repeat_interleave(first, c)
            h = _fmix(((_shr(sv[i], 32) << 32) | (rs[j] & low)) ^ half[i])
            if wv is None:
                counts[0] += h.numel()
                sums[0] += h.sum()
            else:
                counts.index_add_(0, wv[i], torch.ones_like(h))
                sums.index_add_(0, wv[i], h)
            done = int(ends[to - 1])
            at = to
        assert done == total
    return counts, sums


def _u64(t):
    return t.cpu().numpy().view(np.uint64)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("join", "host"):
        c, k = _exact_join(*_relations(case, seed))
        return np.array([_u64(c)[0], _u64(k)[0]], dtype=np.uint64)
    if kind == "batch":
        (r, s), _, (rw, sw) = _windows(case, seed)
        c, k = _exact_join(r, s, rw, sw, case["windows"])
        return {"counts": _u64(c), "checksums": _u64(k)}
    sides = _streams(case, seed)
    size = case["window_ms"]
    base = min(int(a["ts_ms"][0]) for a in sides) // size * size
    n_win = (max(int(a["ts_ms"][-1]) for a in sides) - base) // size + 1
    rel = [torch.from_numpy((a["key"].astype(np.int64) << 32) | a["payload"].astype(np.int64)).cuda() for a in sides]
    win = [torch.from_numpy(((a["ts_ms"].astype(np.int64)) - base) // size).cuda() for a in sides]
    c, k = _exact_join(rel[0], rel[1], win[0], win[1], n_win)
    n = [torch.bincount(w, minlength=n_win).cpu().numpy() for w in win]
    start = base + size * np.arange(n_win)
    return np.stack([start.astype(np.uint64), n[0].astype(np.uint64), n[1].astype(np.uint64), _u64(c), _u64(k)],
                    axis=1)
