"""The calls that this library is used for, as cases that can be timed and compared.

``listed()`` gives the fixed cases, ``draw(rng)`` more of the same ranges.  Kinds:

* ``pf``      the constant-velocity Student-t filter over a whole series (``CVFilter``: set the
              observations, initialize, iterate, read the history), N = 10^3 to 2^24;
* ``batch``   many filters of different sizes and lengths run to their ends (``CVBatch.run``);
* ``stream``  resident filters that get one observation at a time (``CVBatch.step``, as a server
              or a control loop steps them);
* ``gmm``     the tempered sampler for a Gaussian mixture (``GmmSampler``), a whole schedule;
* ``kit``     a program's own model in torch: the library's weight update, ESS / CESS, resampling
              and particle gather around it;
* ``mn``      resampling M weights to N particles (a change of the particle number).
"""
import math

import numpy as np
import torch

from vsmc_b200 import capi

SCHEMES = ("Multinomial", "Residual", "Stratified", "Systematic", "ResidualStratified",
           "ResidualSystematic")
FORMS = {"fp64": capi.FP64, "mixed": capi.MIXED}


def listed():
    return [
        # the reference example's own size: 1000 particles, 100 observations; the final particles
        # are read too
        dict(name="pf_1000", kind="pf", N=1000, T=100, scheme="Multinomial", form="fp64",
             state=True),
        # a tracking filter of ordinary size
        dict(name="pf_65536", kind="pf", N=65536, T=50, scheme="Systematic", form="fp64",
             state=False),
        # a large filter in the mixed form, a size that is no multiple of anything
        dict(name="pf_1000003_mixed", kind="pf", N=1000003, T=16, scheme="Stratified",
             form="mixed", state=False),
        # the largest filter, in both forms (the benchmark's size and scheme)
        dict(name="pf_16m", kind="pf", N=1 << 24, T=8, scheme="Multinomial", form="fp64",
             state=False),
        dict(name="pf_16m_mixed", kind="pf", N=1 << 24, T=8, scheme="Multinomial", form="mixed",
             state=False),
        # many filters at once, N log-uniform on [2^10, 2^16]
        dict(name="batch_256", kind="batch", filters=256, Nlo=1 << 10, Nhi=1 << 16, Tlo=50,
             Thi=200, scheme="Multinomial", form="fp64"),
        # resident filters stepped observation by observation, N log-uniform on [2^10, 2^18]
        dict(name="stream_48_mixed", kind="stream", filters=48, Nlo=1 << 10, Nhi=1 << 18, T=24,
             scheme="Systematic", form="mixed"),
        # the tempered mixture sampler at its default size, in both forms
        dict(name="gmm_65536", kind="gmm", N=65536, n=1000, iters=20, sweeps=5,
             scheme="Systematic", form="fp64"),
        dict(name="gmm_65536_mixed", kind="gmm", N=65536, n=1000, iters=20, sweeps=5,
             scheme="Systematic", form="mixed"),
        # one step of a program's own model: small, where launches count, and large and odd
        dict(name="kit_1000", kind="kit", N=1000, dim=4, scheme="Stratified"),
        dict(name="kit_3000001", kind="kit", N=3000001, dim=4, scheme="ResidualSystematic"),
        # a million weights to fewer particles
        dict(name="mn_1000000_300007", kind="mn", M=1000000, N=300007, scheme="Residual"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pf", "pf", "batch", "stream", "gmm", "kit", "kit", "mn"])
    scheme, form = rng.choice(SCHEMES), rng.choice(["fp64", "mixed"])
    if kind == "pf":
        N = _log_int(rng, 1000, 1 << 24)
        T = max(4, min(100, int((1 << 26) / N)))
        return dict(kind=kind, N=N, T=rng.randint(max(4, T // 2), T), scheme=scheme, form=form,
                    state=N <= 4096)
    if kind == "batch":
        return dict(kind=kind, filters=rng.randint(32, 320), Nlo=1 << 10, Nhi=1 << 16,
                    Tlo=rng.randint(20, 60), Thi=rng.randint(80, 160), scheme=scheme, form=form)
    if kind == "stream":
        return dict(kind=kind, filters=_log_int(rng, 4, 64), Nlo=1 << 10, Nhi=1 << 18,
                    T=rng.randint(8, 32), scheme=scheme, form=form)
    if kind == "gmm":
        return dict(kind=kind, N=_log_int(rng, 1000, 65536), n=_log_int(rng, 200, 1000),
                    iters=rng.randint(16, 20), sweeps=rng.choice([1, 3, 5]), scheme=scheme,
                    form=form)
    if kind == "kit":
        return dict(kind=kind, N=_log_int(rng, 1000, 8000000), dim=rng.choice([1, 2, 4, 6]),
                    scheme=scheme)
    return dict(kind=kind, M=_log_int(rng, 1000, 2000000), N=_log_int(rng, 1000, 2000000),
                scheme=scheme)


# ------------------------------------------------------------------ inputs --

def _rng(seed):
    return np.random.default_rng([int(seed) & 0x7fffffff, 20])


def _series(T, seed):
    """An observation series of the model (dt 0.1, unit start velocity, scaled Student-t noise)."""
    r = _rng(seed)
    p, v = np.zeros(2), np.ones(2)
    out = np.zeros((T, 2))
    for t in range(T):
        if t:
            p = p + 0.1 * v + 0.02 * r.standard_normal(2)
            v = v + 0.5 * r.standard_normal(2)
        out[t] = p + 0.1 * r.standard_t(10, 2)
    return np.ascontiguousarray(out[:, 0]), np.ascontiguousarray(out[:, 1])


def _filter_seed(seed):
    return 101 + 7919 * (int(seed) % 100003)


def _sizes(case, seed):
    """Particle numbers, log-uniform between Nlo and Nhi, the same total work for every seed:
    the quantiles of the range, in the seed's order."""
    k = case["filters"]
    q = (np.arange(k) + 0.5) / k
    lo, hi = math.log(case["Nlo"]), math.log(case["Nhi"])
    return np.exp(lo + (hi - lo) * _rng(seed).permutation(q)).astype(np.int64)


def _lengths(case, seed):
    k = case["filters"]
    q = (np.arange(k) + 0.5) / k
    T = case["Tlo"] + (case["Thi"] - case["Tlo"]) * _rng(seed + 1).permutation(q)
    return T.astype(np.int64)


def _weights(n, seed):
    """Log-weight increments as a likelihood gives them: lognormal weights with an effective
    sample size of about a third."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) % (1 << 31))
    z = torch.randn(n, generator=g, device="cuda", dtype=torch.float64)
    return -0.5 * 1.05 * z * z - 0.35 * z, g


def _gmm_data(case, seed):
    r = _rng(seed)
    z = r.integers(0, 4, case["n"])
    return np.array([-3.0, 0.0, 3.0, 6.0])[z] + 0.55 * r.standard_normal(case["n"])


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case, kind=kind)
    if "form" in case:
        opts = dict(scheme=getattr(capi, case["scheme"]), form=FORMS[case["form"]])
    stream = torch.cuda.current_stream().cuda_stream if torch.cuda.is_available() else None
    if kind == "pf":
        s["obs"] = _series(case["T"], seed)
        s["f"] = capi.CVFilter(case["N"], case["T"], seed=_filter_seed(seed), stream=stream,
                               **opts)
    elif kind in ("batch", "stream"):
        N = _sizes(case, seed)
        T = _lengths(case, seed) if kind == "batch" else np.full(len(N), case["T"])
        s["series"] = [_series(int(t), seed + 17 * k) for k, t in enumerate(T)]
        s["T"] = T
        s["b"] = capi.CVBatch(len(N), stream=stream, **opts)
        s["slots"] = [s["b"].admit(int(n), int(t), seed=_filter_seed(seed) + k, stream_id=k)
                      for k, (n, t) in enumerate(zip(N, T))]
        if kind == "stream":
            x = np.array([ser for ser in s["series"]])
            s["xy"] = np.ascontiguousarray(x.transpose(2, 1, 0))  # [T][2][filters]
            s["first"] = [(x[k, 0, :1], x[k, 1, :1]) for k in range(len(N))]
    elif kind == "gmm":
        s["g"] = capi.GmmSampler(_gmm_data(case, seed), N=case["N"], iters=case["iters"],
                                 sweeps=case["sweeps"], seed=_filter_seed(seed), stream=stream,
                                 **opts)
    elif kind == "kit":
        N, dim = case["N"], case["dim"]
        s["inc"], g = _weights(N, seed)
        s["x"] = torch.randn((dim, N), generator=g, device="cuda", dtype=torch.float64)
        s["y"] = torch.empty_like(s["x"])
        s["lw"] = torch.zeros(N, device="cuda", dtype=torch.float64)
        s["w"] = torch.full((N,), 1.0 / N, device="cuda", dtype=torch.float64)
        s["rep"] = torch.empty(N, device="cuda", dtype=torch.int32)
        s["cf"] = torch.empty(N, device="cuda", dtype=torch.int32)
        s["bytes"] = capi.resample_workspace_size(N)
        s["ws"] = torch.empty(s["bytes"], device="cuda", dtype=torch.uint8)
        s["seed"] = 1 + int(seed) % 1000003
    else:
        inc, _ = _weights(case["M"], seed)
        w = torch.exp(inc)
        s["w"] = w / w.sum()
        s["rep"] = torch.empty(case["M"], device="cuda", dtype=torch.int32)
        s["cf"] = torch.empty(case["N"], device="cuda", dtype=torch.int32)
        s["bytes"] = capi.resample_mn_workspace_size(case["M"], case["N"])
        s["ws"] = torch.empty(s["bytes"], device="cuda", dtype=torch.uint8)
        s["seed"] = 1 + int(seed) % 1000003
    return s


# -------------------------------------------------------------------- runs --

def _run_pf(s):
    f = s["f"]
    f.set_observations_host(*s["obs"])
    f.initialize()
    f.iterate(s["case"]["T"] - 1)
    out = dict(f.history(), log_evidence=f.log_evidence())
    if s["case"]["state"]:
        out["x"], out["lw"] = f.read_state()
    return out


def _run_batch(s):
    b, slots = s["b"], s["slots"]
    b.set_observations(slots, s["series"])
    b.initialize(slots)
    b.run(slots)
    steps = b.read_steps(slots, s["T"])
    return dict(ess=steps["ess"], logz_inc=steps["logz_inc"], resampled=steps["resampled"],
                log_evidence=b.read_last(slots)["log_evidence"])


def _run_stream(s):
    b, slots, xy = s["b"], s["slots"], s["xy"]
    b.set_observations(slots, s["first"])
    b.initialize(slots)
    last = b.read_last(slots)
    got = [last]
    for t in range(1, s["case"]["T"]):
        b.append_observations(slots, xy[t, 0], xy[t, 1])
        b.step(slots)
        last = b.read_last(slots)
        got.append(last)
    return {k: np.array([g[k] for g in got]) for k in ("ess", "logz_inc", "resampled",
                                                       "log_evidence")}


def _run_gmm(s):
    g = s["g"]
    g.initialize()
    g.iterate(s["case"]["iters"])
    smc, path = g.log_evidence()
    params, lw, words = g.read_params()
    return dict(g.history(), smc=smc, path=path, params=params, lw=lw,
                words=words.astype(np.int64))


def _run_kit(s):
    c, stream = s["case"], torch.cuda.current_stream().cuda_stream
    N, lw, w, inc = c["N"], s["lw"], s["w"], s["inc"]
    lw.zero_()  # the weights are equal after the last step's resampling
    w.fill_(1.0 / N)
    ahead = capi.weight_ess(N, lw.data_ptr(), w.data_ptr(), inc.data_ptr(), True, stream=stream)
    cess = capi.weight_cess(N, w.data_ptr(), inc.data_ptr(), True, stream=stream)
    ess = capi.weight_add_log(N, lw.data_ptr(), w.data_ptr(), inc.data_ptr(), stream=stream)
    rng = capi.threefry_state(seed=s["seed"])
    words = capi.resample(getattr(capi, c["scheme"]), N, w.data_ptr(), rng, s["rep"].data_ptr(),
                          s["cf"].data_ptr(), s["ws"].data_ptr(), s["bytes"], stream=stream)
    capi.copy_f64(N, c["dim"], s["x"].data_ptr(), s["y"].data_ptr(), s["cf"].data_ptr(),
                  stream=stream)
    return dict(ahead=ahead, cess=cess, ess=ess, lw=lw, w=w, rep=s["rep"], cf=s["cf"], y=s["y"],
                words=words)


def _run_mn(s):
    c = s["case"]
    rng = capi.threefry_state(seed=s["seed"])
    words = capi.resample_mn(getattr(capi, c["scheme"]), c["M"], c["N"], s["w"].data_ptr(), rng,
                             s["rep"].data_ptr(), s["cf"].data_ptr(), s["ws"].data_ptr(),
                             s["bytes"], stream=torch.cuda.current_stream().cuda_stream)
    return dict(rep=s["rep"], cf=s["cf"], words=words)


_RUN = dict(pf=_run_pf, batch=_run_batch, stream=_run_stream, gmm=_run_gmm, kit=_run_kit,
            mn=_run_mn)


def run(state):
    return _RUN[state["kind"]](state)


# -------------------------------------------------------------------- work --

def work(case):
    """Bytes: each step reads and writes the particles' state and log-weights (5 values) once, and
    a resampling reads the weights, and writes and reads the ancestors; flops: the operations of
    the model and of the two polar normal pairs of a particle's step, counting a log, exp, divide
    or square root as 10."""
    kind = case["kind"]
    if kind in ("pf", "batch", "stream"):
        real = 8 if case["form"] == "fp64" else 4
        if kind == "pf":
            steps = case["N"] * case["T"]
        else:
            N = _sizes(case, 0)
            steps = int((N * (_lengths(case, 0) if kind == "batch" else case["T"])).sum())
        # about four steps in five resample
        return dict(bytes=steps * (10 * real + 0.8 * (real + 8)), flops=steps * 150)
    if kind == "gmm":
        # a likelihood evaluation: 4 densities (a quadratic, an exp, a sum) and a log a point
        evals = case["N"] * (1 + 3 * case["sweeps"] * case["iters"])
        return dict(bytes=case["N"] * case["iters"] * (2 * 14 * 8 + 3 * 8),
                    flops=evals * case["n"] * (4 * 15 + 11))
    if kind == "kit":
        N = case["N"]
        # inc twice (ess and cess need it before the update), w, lw; w to counts and ancestors;
        # the gather
        return dict(bytes=N * (8 + 8 + 8 + 16 + 8 + 8 + 4 + 16 * case["dim"]), flops=N * 60)
    return dict(bytes=case["M"] * 12 + case["N"] * 4, flops=(case["M"] + case["N"]) * 20)


# ------------------------------------------------------------------- exact --
# The same quantities in numpy's doubles: the counter-based engines word for word, the filter and
# the resampling as the algorithms are defined.

_M32 = np.uint64(0xffffffff)


def _philox(c0, c1, c2, c3, k0, k1):
    """Philox4x32-10 (Salmon et al. 2011) on arrays of 32-bit words held in uint64."""
    for r in range(10):
        a = np.uint64(0xCD9E8D57) * c2
        b = np.uint64(0xD2511F53) * c0
        c0, c1, c2, c3 = ((a >> np.uint64(32)) ^ k0 ^ c1, a & _M32,
                          (b >> np.uint64(32)) ^ k1 ^ c3, b & _M32)
        k0, k1 = (k0 + np.uint64(0x9E3779B9)) & _M32, (k1 + np.uint64(0xBB67AE85)) & _M32
    return c0, c1, c2, c3


def _threefry(seed, first, count):
    """Words first .. first + count of a Threefry4x64-20 engine with key (seed, 0, 0, 0)."""
    rot = ((14, 16), (52, 57), (23, 40), (5, 37), (25, 33), (46, 12), (58, 22), (32, 32))
    b0 = first // 4
    n = (first + count + 3) // 4 - b0
    z = np.zeros(n, np.uint64)
    key = [np.uint64(seed), np.uint64(0), np.uint64(0), np.uint64(0)]
    key.append(np.uint64(0x1BD11BDAA9FC1A22) ^ key[0])
    x = [np.arange(b0 + 1, b0 + 1 + n, dtype=np.uint64), z.copy(), z.copy(), z.copy()]
    with np.errstate(over="ignore"):
        x = [v + k for v, k in zip(x, key)]
        for r in range(20):
            for j, (a, b) in enumerate(((0, 1), (2, 3)) if r % 2 == 0 else ((0, 3), (2, 1))):
                x[a] = x[a] + x[b]
                q = rot[r % 8][j]
                x[b] = ((x[b] << np.uint64(q)) | (x[b] >> np.uint64(64 - q))) ^ x[a]
            if r % 4 == 3:
                t = (r + 1) // 4
                x = [v + key[(t + i) % 5] for i, v in enumerate(x)]
                x[3] = x[3] + np.uint64(t)
    return np.stack(x, 1).reshape(-1)[first - 4 * b0:first - 4 * b0 + count]


def _unit(words):
    return np.minimum(words.astype(np.float64) * 2.0 ** -64, 1.0 - 2.0 ** -53)


def _normals(step, N, stream, key):
    """The four normals of each particle's step: two accepted polar points of its own stream, the
    second coordinate of a point first (as std::normal_distribution gives them)."""
    x, y = np.zeros((2, N)), np.zeros((2, N))
    got = np.zeros(N, np.int64)
    left, blk = np.arange(N), 0
    while left.size:
        blk += 1
        one = np.ones(left.size, np.uint64)
        w = _philox(one * np.uint64(blk), one * np.uint64(step), left.astype(np.uint64),
                    one * np.uint64(stream), one * np.uint64(key), one * np.uint64(0))
        a = 2.0 * _unit(w[0] | (w[1] << np.uint64(32))) - 1.0
        b = 2.0 * _unit(w[2] | (w[3] << np.uint64(32))) - 1.0
        r2 = a * a + b * b
        ok = (r2 <= 1.0) & (r2 != 0.0)
        m = np.sqrt(-2.0 * np.log(r2[ok]) / r2[ok])
        i = left[ok]
        x[got[i], i], y[got[i], i] = b[ok] * m, a[ok] * m
        got[i] += 1
        left = left[got[left] < 2]
    return x[0], y[0], x[1], y[1]


def _sorted_uniforms(words):
    n = words.size
    terms = np.log(1.0 - _unit(words)) / np.arange(n, 0, -1.0)
    return 1.0 - np.exp(np.cumsum(terms))


def _counts(scheme, w, N, seed, offset):
    """Replication counts of M weights over N uniforms, and the engine words drawn."""
    M, base, n = w.size, 0, N
    if scheme.startswith("Residual"):
        full = N * w
        base = np.floor(full)
        w = full - base
        w = w * (1.0 / np.cumsum(w)[-1])
        base = base.astype(np.int64)
        n = N - int(base.sum())
    if n == 0:
        return base, 1 if scheme.endswith("Systematic") else 0
    acc = np.cumsum(w)[:-1]
    if scheme in ("Multinomial", "Residual"):
        u = _sorted_uniforms(_threefry(seed, offset, n))
    elif scheme.endswith("Stratified"):
        u = _unit(_threefry(seed, offset, n)) * (1.0 / n) + np.arange(n) * (1.0 / n)
    else:
        u = _unit(_threefry(seed, offset, 1))[0] * (1.0 / n) + np.arange(n) * (1.0 / n)
    at = np.concatenate([np.searchsorted(u, acc, side="right"), [n]])
    at = np.maximum.accumulate(at)
    rep = np.diff(at, prepend=0)
    words = 1 if scheme.endswith("Systematic") else min(n, int(at[-2] if M > 1 else 0) + 1)
    return base + rep, words if M > 1 else 0


def _ancestors(rep):
    cf = np.arange(rep.size)
    cf[rep == 0] = np.repeat(np.arange(rep.size), np.maximum(rep - 1, 0))
    return cf


def _filter(N, ox, oy, scheme, seed, stream):
    """The constant-velocity Student-t filter over a whole series, from its definition."""
    seed = seed % 0xffffffff
    T = len(ox)
    h = dict(ess=np.zeros(T), resampled=np.zeros(T, np.int64), logz_inc=np.zeros(T),
             mean_x=np.zeros(T), mean_y=np.zeros(T))
    lw, s1, offset = np.zeros(N), float(N), 0
    for t in range(T):
        n1, n2, n3, n4 = _normals(t, N, stream, seed + 1)
        if t == 0:
            x, y, vx, vy = 2.0 * n1, 2.0 * n2, 1.0 * n3, 1.0 * n4
        else:
            x, y = x + (0.02 * n1 + 0.1 * vx), y + (0.02 * n2 + 0.1 * vy)
            vx, vy = vx + 0.5 * n3, vy + 0.5 * n4
        a, b = 10.0 * (x - ox[t]), 10.0 * (y - oy[t])
        lw = lw - 5.5 * (np.log(1.0 + a * a / 10.0) + np.log(1.0 + b * b / 10.0))
        top = lw.max()
        lw = lw - top
        e = np.exp(lw)
        S = e.sum()
        h["logz_inc"][t] = top + math.log(S) - math.log(s1)
        h["ess"][t] = S * S / (e * e).sum()
        s1 = S
        if h["ess"][t] < 0.5 * N:
            h["resampled"][t] = 1
            w = e * (1.0 / np.cumsum(e)[-1])
            rep, words = _counts(scheme, w, N, seed + 2, offset)
            offset += words
            cf = _ancestors(rep)
            x, y, vx, vy = x[cf], y[cf], vx[cf], vy[cf]
            lw, s1, e, S = np.zeros(N), float(N), np.ones(N), float(N)
        h["mean_x"][t], h["mean_y"][t] = (e * x).sum() / S, (e * y).sum() / S
    return h, (np.array([x, y, vx, vy]), lw)


def exact(case, seed):
    kind = case["kind"]
    if kind == "pf":
        if case["N"] * case["T"] > 4000000:
            return None
        ox, oy = _series(case["T"], seed)
        h, (x, lw) = _filter(case["N"], ox, oy, case["scheme"], _filter_seed(seed), 0)
        out = dict(h, resampled=None, log_evidence=float(h["logz_inc"].sum()))
        if case["state"]:
            out["x"], out["lw"] = x, lw
        return out
    if kind == "kit":
        N = case["N"]
        s = prepare(case, seed)
        inc, x = s["inc"].cpu().numpy(), s["x"].cpu().numpy()
        e = np.exp(inc - inc.max())
        ess = float(e.sum() ** 2 / (e * e).sum())
        b = np.exp(inc)
        cess = float((b / N).sum() ** 2 / (b * b / N).sum())
        w = e / e.sum()
        rep, _ = _counts(case["scheme"], w, N, 1 + int(seed) % 1000003, 0)
        return dict(ahead=ess, cess=cess, ess=ess, lw=inc - inc.max(), w=w, rep=None, cf=None,
                    y=x[:, _ancestors(rep)], words=None)
    # batch and stream: thousands of steps; gmm: 10^9 density evaluations and more; mn: whole
    # numbers only
    return None
