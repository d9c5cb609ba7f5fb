"""The work that the library's speed is measured on: what its users call, each
through a public entry point, from the smallest calls to the largest.

A case is a dict of plain values with an ``op``:

* ``fill``    -- one batch draw of an engine (raw words, U01, Normal,
  Exponential) into a tensor the program keeps;
* ``gamma``   -- Gamma streams, one shape per block of samples;
* ``step``    -- the library's part of one SMC step of a program with its own
  model: Weight.add_log, weighted estimate, resampling, parent indices,
  selection of the particles;
* ``filter``  -- a whole plain FP64 particle filter, the reference's step order;
* ``batched`` -- many uneven filters at once, FP32 moves;
* ``adjoint`` -- the filters' log-likelihoods and their gradients;
* ``score``   -- the log-likelihoods and the Fisher-identity score.
"""
import math

import numpy as np
import torch

import mckl_b200 as mb

SCHEMES = ("multinomial", "stratified", "systematic", "residual", "residual_stratified", "residual_systematic")


def listed():
    return [
        # a host program's scalar-sized draw (initial states, a proposal's noise): launch latency
        {"name": "normal_f64_small", "op": "fill", "engine": "Philox4x32", "dist": "normal", "dtype": "f64", "n": 1000,
         "skip": 3},
        # the raw engine at the size the reference's own RNG benchmark draws
        {"name": "philox_words", "op": "fill", "engine": "Philox4x32", "dist": "words", "dtype": "u32", "n": 1 << 26,
         "skip": 0},
        # a large Monte Carlo draw in double precision, odd length
        {"name": "threefry_normal_f64", "op": "fill", "engine": "Threefry4x64", "dist": "normal", "dtype": "f64",
         "n": (1 << 24) + 1, "skip": 0},
        # a single-precision draw from the middle of a stream (not on a block boundary)
        {"name": "ars_exponential_f32", "op": "fill", "engine": "ARS", "dist": "exponential", "dtype": "f32",
         "n": 5000003, "skip": 5},
        # Gamma with a shape per block of samples, shapes on both sides of 1
        {"name": "gamma_blocks_f32", "op": "gamma", "engine": "Threefry4x64", "dtype": "f32", "blocks": 4096,
         "block": 4096},
        # one SMC step of a small sampler with its own model, odd particle count
        {"name": "step_small", "op": "step", "N": 1001, "dim": 2, "scheme": "residual"},
        # the same at the plain filter's particle count
        {"name": "step_large", "op": "step", "N": 1 << 20, "dim": 4, "scheme": "systematic"},
        # a filter of the size a parameter search runs, parents recorded
        {"name": "filter_small", "op": "filter", "N": 4000, "T": 100, "scheme": "stratified", "record": True},
        # the plain filter at the size the reference is quoted on
        {"name": "filter_large", "op": "filter", "N": 1 << 20, "T": 64, "scheme": "systematic", "record": False},
        # uneven filters, particle counts log-uniform over the batched configuration's range
        {"name": "batched_f32", "op": "batched", "F": 1024, "T": 100, "nmin": 256, "nmax": 65536},
        # gradients over a set of parameters, as an optimiser asks for them
        {"name": "adjoint", "op": "adjoint", "F": 256, "T": 100, "nmin": 8192, "nmax": 8192},
        {"name": "score", "op": "score", "F": 256, "T": 100, "nmin": 8192, "nmax": 8192},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["fill", "fill", "gamma", "step", "filter", "batched", "adjoint", "score"])
    if op == "fill":
        dist = rng.choice(["words", "u01", "normal", "exponential"])
        return {"op": op, "engine": rng.choice(["Philox4x32", "Threefry4x64", "ARS"]), "dist": dist,
                "dtype": "u32" if dist == "words" else rng.choice(["f32", "f64"]), "n": _log(rng, 500, 1 << 26),
                "skip": rng.choice([0, 0, rng.randrange(1, 8)])}
    if op == "gamma":
        return {"op": op, "engine": rng.choice(["Philox4x32", "Threefry4x64", "ARS"]),
                "dtype": rng.choice(["f32", "f64"]), "blocks": _log(rng, 16, 4096), "block": rng.randrange(1000, 4097)}
    if op == "step":
        return {"op": op, "N": _log(rng, 256, 1 << 20), "dim": rng.randrange(1, 5), "scheme": rng.choice(SCHEMES)}
    if op == "filter":
        N = _log(rng, 256, 1 << 20)
        return {"op": op, "N": N, "T": rng.randrange(32, 65), "scheme": rng.choice(SCHEMES[:4]), "record": N < 10000}
    if op == "batched":
        return {"op": op, "F": _log(rng, 16, 1024), "T": rng.randrange(50, 101), "nmin": _log(rng, 256, 4096),
                "nmax": _log(rng, 4096, 65536)}
    n = _log(rng, 500, 8192)
    return {"op": op, "F": _log(rng, 32, 256), "T": rng.randrange(50, 101), "nmin": n, "nmax": n}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _observations(r, F, T, phi, sx, sy):
    """AR(1) states and their noisy observations, [F, T + 1] (y_0 is not used)."""
    x = sx / np.sqrt(1 - phi * phi) * r.standard_normal(F)
    y = np.zeros((F, T + 1))
    for t in range(1, T + 1):
        x = phi * x + sx * r.standard_normal(F)
        y[:, t] = x + sy * r.standard_normal(F)
    return y


def _key(engine, seed):
    r = np.random.default_rng([seed, 1])
    return tuple(int(k) for k in r.integers(1, 1 << 31, {"Philox4x32": 2}.get(engine, 4)))


def _engine(case, seed):
    return mb.ENGINES[case["engine"]](key=_key(case["engine"], seed))


def _out(dtype, n):
    return torch.empty(n, dtype={"u32": torch.int32, "f32": torch.float32, "f64": torch.float64}[dtype], device="cuda")


def _filters(case, seed):
    r = np.random.default_rng([seed, 2])
    F, T = case["F"], case["T"]
    phi, sx, sy = r.uniform(0.5, 0.99, F), r.uniform(0.5, 2.0, F), r.uniform(0.2, 1.0, F)
    N = np.rint(np.exp(r.uniform(math.log(case["nmin"]), math.log(case["nmax"]), F))).astype(np.uint64)
    return dict(N=N, y=_observations(r, F, T, phi, sx, sy), phi=phi, sx=sx, sy=sy,
                mkeys=r.integers(1, 1 << 31, (F, 2)).astype(np.uint32),
                rkeys=r.integers(1, 1 << 31, (F, 2)).astype(np.uint32))


def _step_inputs(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    N, dim = case["N"], case["dim"]
    x = torch.randn((dim, N), generator=g, dtype=torch.float64, device="cuda")
    # the log-likelihood of one observation, as uneven as a filter's usually is
    v = -0.5 * (1.7 * torch.randn(N, generator=g, dtype=torch.float64, device="cuda")) ** 2 - 0.4
    return x, v


def prepare(case, seed):
    op = case["op"]
    if op == "fill":
        rng = _engine(case, seed)
        if case["skip"]:
            rng.discard(case["skip"])
        return {"case": case, "rng": rng, "out": _out(case["dtype"], case["n"])}
    if op == "gamma":
        alpha = np.random.default_rng([seed, 3]).uniform(0.5, 10.0, case["blocks"])
        return {"case": case, "rng": _engine(case, seed), "alpha": alpha,
                "out": _out(case["dtype"], case["blocks"] * case["block"])}
    if op == "step":
        x, v = _step_inputs(case, seed)
        return {"case": case, "x": x, "v": v, "W": mb.Weight(case["N"]),
                "rng": mb.Philox4x32(key=_key("Philox4x32", seed))}
    if op == "filter":
        r = np.random.default_rng([seed, 4])
        phi, sx, sy = 0.9, 1.0, 0.7
        y = _observations(r, 1, case["T"], np.array([phi]), np.array([sx]), np.array([sy]))[0]
        return {"case": case, "y": y, "par": (phi, sx, sy, sx / math.sqrt(1 - phi * phi)),
                "mkey": _key("Philox4x32", seed), "rkey": _key("Philox4x32", seed + 1)}
    w = _filters(case, seed)
    b = mb.BatchedFilters(w["N"], w["y"], w["phi"], w["sx"], w["sy"], w["mkeys"], w["rkeys"], fp64=op != "batched")
    if op == "adjoint":
        b.config(1024, 1)  # the block shape the autograd binding uses
    return {"case": case, "b": b, "w": w}


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
    case = state["case"]
    op = case["op"]
    if op == "fill":
        rng, r, n, dist = state["rng"].copy(), state["out"], case["n"], case["dist"]
        if dist == "words":
            return mb.rand(rng, n, r)
        if dist == "u01":
            return mb.u01_distribution(rng, n, r)
        if dist == "normal":
            return mb.normal_distribution(rng, n, r)
        return mb.exponential_distribution(rng, n, r, lam=1.5)
    if op == "gamma":
        return mb.gamma_blocks(state["rng"], case["block"], state["alpha"], state["out"])
    if op == "step":
        W, rng = state["W"], state["rng"].copy()
        x = state["x"] * 0.9  # the program's own move
        W.set_equal()
        W.add_log(state["v"])
        est = mb.weighted_estimate(x, W.data, col_major=True)
        w = W.data
        rep = mb.resample(SCHEMES.index(case["scheme"]), rng, w)
        idx = mb.rep_to_index(rep, case["N"])
        mb.select(idx, x)
        return {"W": w, "ess": W.ess(), "log_nc": W.log_nc, "est": est, "rep": rep, "idx": idx, "x": x}
    if op == "filter":
        phi, sx, sy, sd0 = state["par"]
        r = mb.pf_ar1_plain(case["N"], state["y"], phi, sx, sy, sd0, state["mkey"], state["rkey"],
                            scheme=SCHEMES.index(case["scheme"]), record=case["record"])
        return r
    b, w = state["b"], state["w"]
    if op == "batched":
        b.set_y(w["y"])
        b.run(graph=True)
        return b.results()
    b.set_params(w["phi"], w["sx"], w["sy"])
    return b.adjoint() if op == "adjoint" else b.score()


# ---------------------------------------------------------------------------
# what one pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    op = case["op"]
    if op == "fill":
        size = {"u32": 4, "f32": 4, "f64": 8}[case["dtype"]]
        flops = {"words": 0, "u01": 2, "normal": 40, "exponential": 25}[case["dist"]]
        return {"bytes": case["n"] * size, "flops": case["n"] * flops}
    if op == "gamma":
        n = case["blocks"] * case["block"]
        return {"bytes": n * {"f32": 4, "f64": 8}[case["dtype"]] + 8 * case["blocks"], "flops": n * 80}
    if op == "step":
        N, dim = case["N"], case["dim"]
        # v and W in, W and rep and idx out, the particles in and out twice (move, selection)
        return {"bytes": 8 * N * (5 + 4 * dim), "flops": N * (60 + 3 * dim)}
    if op == "filter":
        N, T = case["N"], case["T"]
        # y in; particles and weights out, and the parents of each step when recorded
        return {"bytes": 8 * (T + 1) + 16 * N + (8 * N * (T + 1) if case["record"] else 0), "flops": 140 * N * T}
    # log-uniform particle counts: their mean
    a, b = case["nmin"], case["nmax"]
    mean = a if a == b else (b - a) / math.log(b / a)
    ps = case["F"] * case["T"] * mean
    per = {"batched": 60, "adjoint": 300, "score": 600}[op]
    return {"bytes": 8.0 * case["F"] * (case["T"] + 8), "flops": ps * per}


# ---------------------------------------------------------------------------
# the same values in 64 bits, in plain torch: engine words from the generators'
# definitions, the transforms in double, sums in any order
# ---------------------------------------------------------------------------
_M32 = 0xFFFFFFFF


def _philox_words(key, first, blocks):
    c = first + torch.arange(blocks, dtype=torch.int64, device="cuda")
    s = [c & _M32, c >> 32, torch.zeros_like(c), torch.zeros_like(c)]
    a, b = key[0] & _M32, key[1] & _M32
    for _ in range(10):
        p2, p0 = s[2] * 0xCD9E8D57, s[0] * 0xD2511F53
        s = [a ^ s[1] ^ ((p2 >> 32) & _M32), p2 & _M32, b ^ s[3] ^ ((p0 >> 32) & _M32), p0 & _M32]
        a, b = (a + 0x9E3779B9) & _M32, (b + 0xBB67AE85) & _M32
    return torch.stack(s, 1).reshape(-1)


def _i64(v):
    v &= (1 << 64) - 1
    return v - (1 << 64) if v >> 63 else v


def _threefry_words(key, first, blocks):
    c = first + torch.arange(blocks, dtype=torch.int64, device="cuda")
    par = list(key) + [0x1BD11BDAA9FC1A22 ^ key[0] ^ key[1] ^ key[2] ^ key[3]]
    s = [c, torch.zeros_like(c), torch.zeros_like(c), torch.zeros_like(c)]

    def inject(n):
        for i in range(4):
            s[i] = s[i] + _i64(par[(n + i) % 5] + (n if i == 3 else 0))

    def rotl(x, k):
        return (x << k) | ((x >> (64 - k)) & ((1 << k) - 1))

    rot = [(14, 16), (52, 57), (23, 40), (5, 37), (25, 33), (46, 12), (58, 22), (32, 32)]
    inject(0)
    for r in range(20):
        k0, k1 = rot[r % 8]
        s[0], s[2] = s[0] + s[1], s[2] + s[3]
        s[1], s[3] = s[2] ^ rotl(s[3], k1), s[0] ^ rotl(s[1], k0)
        if r % 4 == 3:
            inject(r // 4 + 1)
    return torch.stack([w for x in s for w in (x & _M32, (x >> 32) & _M32)], 1).reshape(-1)


def _ars_words(key, first, blocks):
    def xtime(v):
        return ((v << 1) ^ (0x1B if v & 0x80 else 0)) & 0xFF

    def gmul(a, b):
        p = 0
        while b:
            p ^= a if b & 1 else 0
            a, b = xtime(a), b >> 1
        return p

    sbox = []
    for v in range(256):
        inv = next((u for u in range(256) if gmul(v, u) == 1), 0)
        o = 0x63
        for k in range(5):
            o ^= ((inv << k) | (inv >> (8 - k))) & 0xFF
        sbox.append(o)
    S = torch.tensor(sbox, device="cuda")
    X2 = torch.tensor([xtime(v) for v in range(256)], device="cuda")

    def round_key(n):
        lo = (key[0] | (key[1] << 32)) + 0x9E3779B97F4A7C15 * n
        hi = (key[2] | (key[3] << 32)) + 0xBB67AE8584CAA73B * n
        b = (lo & ((1 << 64) - 1)).to_bytes(8, "little") + (hi & ((1 << 64) - 1)).to_bytes(8, "little")
        return torch.tensor(list(b), device="cuda")

    c = first + torch.arange(blocks, dtype=torch.int64, device="cuda")
    st = torch.zeros((blocks, 16), dtype=torch.int64, device="cuda")
    for i in range(8):
        st[:, i] = (c >> (8 * i)) & 0xFF
    st = st ^ round_key(0)
    shift = torch.tensor([(4 * ((i // 4 + i % 4) % 4) + i % 4) for i in range(16)], device="cuda")
    for n in range(1, 6):
        st = S[st][:, shift]
        if n < 5:
            a = st.reshape(-1, 4, 4)
            t = a[:, :, 0] ^ a[:, :, 1] ^ a[:, :, 2] ^ a[:, :, 3]
            st = (a ^ t[:, :, None] ^ X2[a ^ a.roll(-1, 2)]).reshape(-1, 16)
        st = st ^ round_key(n)
    w = st.reshape(-1, 4, 4)
    return (w[:, :, 0] | (w[:, :, 1] << 8) | (w[:, :, 2] << 16) | (w[:, :, 3] << 24)).reshape(-1)


_WORDS = {"Philox4x32": (_philox_words, 4), "Threefry4x64": (_threefry_words, 8), "ARS": (_ars_words, 4)}


def _words(engine, key, skip, n):
    """Stream words [skip, skip + n) of a freshly keyed engine (its first block has counter 1)."""
    fn, per = _WORDS[engine]
    out = []
    first, left = skip // per, (skip % per + n + per - 1) // per
    while left:
        m = min(left, 1 << 20)
        out.append(fn(key, 1 + first, m))
        first, left = first + m, left - m
    return torch.cat(out)[skip % per:skip % per + n]


def _u01oc(w, dtype):
    return ((w >> 8).double() + 1) * 2.0 ** -24 if dtype == "f32" else (w.double() + 1) * 2.0 ** -32


def _normals(words, n, dtype):
    """The Normal(0, 1) draws of one call from its words (n, two more when n is odd)."""
    K = 2048 if dtype == "f32" else 1024
    u = _u01oc(words, dtype)

    def pairs(a):
        h = a.shape[1] // 2
        r, t = torch.sqrt(-2 * torch.log(a[:, :h])), 2 * math.pi * a[:, h:2 * h]
        return torch.cat([r * torch.sin(t), r * torch.cos(t)], 1).reshape(-1)

    m = n // K
    z = [pairs(u[:m * K].reshape(m, K))] if m else []
    if n % K > 1:
        z.append(pairs(u[m * K:n - n % 2].reshape(1, -1)))
    if n % 2:
        z.append((torch.sqrt(-2 * torch.log(u[n])) * torch.cos(2 * math.pi * u[n + 1])).reshape(1))
    return torch.cat(z)


def _exact_fill(case, seed):
    n, dist, dtype, engine, key = case["n"], case["dist"], case["dtype"], case["engine"], _key(case["engine"], seed)
    if dist == "words":
        return None
    need = 2 * n if (dist, dtype) == ("u01", "f64") else n + 2
    w = _words(engine, key, case["skip"], need)
    if dist == "u01":
        if dtype == "f64":
            return w[0::2].double() * 2.0 ** -64 + w[1::2].double() * 2.0 ** -32
        return w[:n].double() * 2.0 ** -32
    if dist == "normal":
        return _normals(w, n, dtype)
    return torch.log(_u01oc(w[:n], dtype)) / -1.5


def _exact_filter(case, seed):
    """Only where sums in another order leave every resampling decision as it is:
    a uniform then lies within a rounding of a cumulative weight with a
    probability of about N^2 2^-50 per step."""
    N, T = case["N"], case["T"]
    if N > 20000 or case["scheme"] not in ("stratified", "systematic"):
        return None
    s = prepare(case, seed)
    phi, sx, sy, sd0 = s["par"]
    per = N + 2 * (N % 2)
    w = _words("Philox4x32", s["mkey"], 0, per * (T + 1))
    x = sd0 * _normals(w[:per], N, "f64")
    rw = _words("Philox4x32", s["rkey"], 0, 2 * N * (T + 1))
    W = torch.full((N,), 1.0 / N, dtype=torch.float64, device="cuda")
    at, ll, ess = 0, 0.0, [float(N)]
    slots = torch.arange(N, device="cuda")
    for t in range(1, T + 1):
        x = phi * x + sx * _normals(w[t * per:(t + 1) * per], N, "f64")
        lw = torch.log(W) - math.log(sy) - 0.5 * math.log(2 * math.pi) - (s["y"][t] - x) ** 2 * (0.5 / sy ** 2)
        e = torch.exp(lw - lw.max())
        ll += float(lw.max() + torch.log(e.sum()))
        W = e / e.sum()
        ess.append(float(1 / (W * W).sum()))
        if ess[-1] < 0.5 * N:
            m = 1 if case["scheme"] == "systematic" else N
            u = rw[at:at + 2 * m].double().reshape(m, 2)
            at += 2 * m
            u = (slots.double() + u[:, 0] * 2.0 ** -64 + u[:, 1] * 2.0 ** -32) / N
            c = torch.searchsorted(u, torch.cumsum(W, 0))
            c[-1] = N
            rep = torch.diff(c, prepend=c[:1] * 0)
            idx = torch.where(rep > 0, slots, -1)
            idx[idx < 0] = torch.repeat_interleave(slots, torch.clamp(rep - 1, min=0))
            x = x[idx]
            W = torch.full_like(W, 1.0 / N)
    return {"loglik": ll, "ess": np.array(ess), "resampled": None, "anc": None, "x": x, "W": W, "ties": None}


def exact(case, seed):
    op = case["op"]
    if op == "fill":
        return _exact_fill(case, seed)
    if op == "step":
        x, v = _step_inputs(case, seed)
        W = torch.softmax(v, 0)
        N = case["N"]
        return {"W": W, "ess": float(1 / (W * W).sum()), "log_nc": float(torch.logsumexp(v, 0)) - math.log(N),
                "est": (0.9 * x) @ W, "rep": None, "idx": None, "x": None}
    if op == "filter":
        return _exact_filter(case, seed)
    # Gamma's rejections, and the genealogies of FP32 filters and of thousands of
    # large ones, have no short restatement: the outputs are compared by type
    return None
