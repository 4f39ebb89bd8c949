"""Performance cases of the framework: what users of the search have it do,
through its public entry points, over the range of sizes they run.

    listed()              the standing cases
    draw(rng)             one more case of the same ranges
    prepare(case, seed)   inputs and handles a program has before the call
    run(state)            one pass; returns all of its outputs
    work(case)            bytes and floating-point operations of one pass
    exact(case, seed)     the outputs in 64-bit arithmetic (plain torch)

A case is a dict of plain values.  Its "kind" names the call:

    stages      one or a few overlap-save steps through the stage calls
                (prepare_segments, power_planes, sum_harmonics), the way a
                caller of the reference's pipeline functions works
    search      AccelSearch.search of DM-trial series in device memory (as
                dedispersion leaves them) and its candidate list
    host        the same from pinned host memory
    spectra     AccelSearch.search_spectra of whitened spectra
    trial_prep  one trial's transform and whitening (rfft, whiten)
    dedisperse  a filterbank summed into DM trials
    refine      candidate refinement (optimize) after a search
    serve       a burst of requests through the server

Input values are what the path meets: N(0,1) noise, a few accelerated
sinusoids well above or well below the threshold, red noise where the
spectrum is whitened.
"""
import functools
import math

import numpy as np
import torch

DT = 64e-6


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # One overlap-save step through the stage calls at the small
        # configuration (zmax 50, 4 harmonics, 2048-point segments): the
        # smallest call, as the step loop of a ported driver makes it.
        dict(name="stages_one_step", kind="stages", zmax=50, numharm=4, fftlen=2048, nseg=1),
        # A short observation of one DM trial: launches and latency count.
        dict(name="search_short_trial", kind="search", zmax=50, numharm=4, fftlen=2048, ntrials=1,
             nmin=1 << 16, nmax=1 << 16, chunk=0, fp16=0, short=0),
        # One ordinary DM trial (67 s at 64 us) with the library's defaults.
        dict(name="search_one_trial", kind="search", zmax=200, numharm=8, fftlen=8192, ntrials=1,
             nmin=1 << 20, nmax=1 << 20, chunk=0, fp16=0, short=0),
        # The production batch: trials of 2^20 .. 2^22 samples searched
        # together at the benchmark's launch shape (L = 4096, 512 segments).
        dict(name="search_batch", kind="search", zmax=200, numharm=8, fftlen=4096, ntrials=32,
             nmin=1 << 20, nmax=1 << 22, chunk=512, fp16=0, short=0),
        # Trials as an acquisition or file reader hands them over: pinned host
        # series of uneven (even, 5-smooth to prime-ish) lengths.
        dict(name="search_host_series", kind="host", zmax=200, numharm=8, fftlen=8192, ntrials=6,
             nmin=600_000, nmax=1_500_000, chunk=0, fp16=0, short=0),
        # Wide acceleration range on spectra whitened elsewhere, with the
        # half-size FP16 template bank.
        dict(name="spectra_z300_fp16", kind="spectra", zmax=300, numharm=8, fftlen=8192, ntrials=1,
             nmin=1_234_566, nmax=1_234_566, chunk=0, fp16=1, short=0),
        # Sixteen harmonics with the longest segments (narrow-pulse pulsars).
        dict(name="search_16_harmonics", kind="search", zmax=100, numharm=16, fftlen=16384, ntrials=2,
             nmin=1 << 20, nmax=3 << 19, chunk=0, fp16=0, short=0),
        # One long trial's transform and whitening, power-of-two length.
        dict(name="trial_prep_pow2", kind="trial_prep", n=1 << 22),
        # The same for an observation of arbitrary length (half length with a
        # large prime factor), as a stream of observations has.
        dict(name="trial_prep_any_length", kind="trial_prep", n=2 * 609_997),
        # A 1024-channel band into 128 DM trials.
        dict(name="dedisperse_1024ch", kind="dedisperse", nchan=1024, nout=1 << 18, ndm=128, dm0=0.0,
             ddm=1.0),
        # Refinement of a search's candidates (positions, harmonics' powers).
        dict(name="refine_candidates", kind="refine", zmax=200, numharm=8, fftlen=8192, n=1 << 20,
             ncand=64),
        # A burst of requests of mixed lengths and acceleration ranges.
        dict(name="serve_burst", kind="serve", requests=24, nmin=1 << 18, nmax=1 << 21, fftlen=8192,
             chunk=128),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["stages", "search", "search", "host", "spectra", "trial_prep", "dedisperse", "refine",
                       "serve"])
    zmax = rng.choice([50, 100, 200, 300])
    if kind == "stages":
        nh, L = rng.choice([(4, 2048), (8, 4096), (8, 8192), (2, 1024)])
        return dict(kind=kind, zmax=min(zmax, 200 if L > 2048 else 50), numharm=nh, fftlen=L,
                    nseg=_log(rng, 1, 40))
    if kind in ("search", "host", "spectra"):
        nh, L = rng.choice([(8, 8192), (8, 8192), (8, 4096), (4, 4096), (4, 2048), (1, 8192), (16, 16384)])
        if L == 2048:
            zmax = 50
        elif L == 4096:
            zmax = min(zmax, 200)
        n = 2 * _log(rng, 1 << 15, 1 << 20)
        if rng.random() < 0.5:
            n = 1 << (n.bit_length() - 1)
        return dict(kind=kind, zmax=zmax, numharm=nh, fftlen=L, ntrials=rng.choice([1, 1, 2, 5, 8]), nmin=n,
                    nmax=n if rng.random() < 0.5 else 2 * n, chunk=rng.choice([0, 0, 128, 512]),
                    fp16=int(rng.random() < 0.15), short=int(rng.random() < 0.15))
    if kind == "trial_prep":
        k = _log(rng, 1 << 15, 1 << 22)
        if rng.random() < 0.3:
            k = 1 << (k.bit_length() - 1)
        elif rng.random() < 0.3:
            k = 3 << max(13, k.bit_length() - 2)
        return dict(kind=kind, n=2 * k)
    if kind == "dedisperse":
        return dict(kind=kind, nchan=_log(rng, 48, 1024), nout=_log(rng, 4000, 1 << 18), ndm=_log(rng, 3, 128),
                    dm0=float(rng.choice([0, 0, 30, 200])), ddm=float(rng.choice([0.25, 1.0, 1.0, 3.0, 20.0])))
    if kind == "refine":
        return dict(kind=kind, zmax=min(zmax, 200), numharm=rng.choice([4, 8]), fftlen=8192,
                    n=1 << rng.randint(18, 21), ncand=_log(rng, 4, 128))
    n = _log(rng, 1 << 18, 1 << 19)
    return dict(kind="serve", requests=rng.randint(1, 16), nmin=n, nmax=4 * n, fftlen=rng.choice([8192, 4096]),
                chunk=128)


# ------------------------------------------------------------------- geometry
# The bank and step geometry of the search, for work() and exact().
def _halfwidth(z):
    z = abs(z)
    m = max(int(z * (0.00089 * z + 0.3131) + 16), 16)
    return int(0.6 * z) if z > 100 and m > 0.6 * z else m


def _required_z(p, q, zfull):
    x = abs(zfull) * p
    v = 2 * ((2 * x + 2 * q) // (4 * q))
    return v if zfull >= 0 else -v


def _uselen(zmax, L):
    return (L - 2 - 4 * _halfwidth(zmax)) & ~1


def _bank(zmax, numharm, L):
    """[(p, q, zmax_h, rows, L_h, halfwidth)] in the summing order 1, 1/2, 1/4, 3/4, ..."""
    U = _uselen(zmax, L)
    out = []
    q = 1
    while q <= numharm:
        for p in range(1, q + 1, 2):
            zh = _required_z(p, q, zmax)
            need = U * p // q + 2 + 4 * _halfwidth(zh)
            out.append((p, q, zh, zh + 1, 1 << (need - 1).bit_length(), _halfwidth(zh)))
        q *= 2
    return U, out


def _step(startr, U, p, q, hw):
    """(rlo, columns, first bin, bins normalised) of harmonic p/q in the step at startr."""
    a0 = (2 * 2 * startr * p + q) // (2 * q)
    a1 = (2 * (2 * startr + U - 1) * p + q) // (2 * q)
    rlo, rhi = a0 >> 1, (a1 + 1) >> 1
    return rlo, U if q == 1 else 2 * (rhi - rlo) + 2, rlo - hw, rhi - rlo + 2 * hw + 1


def _steps(n, U):
    rlo = int(np.floor(np.float64(np.float32(n) * np.float32(DT))))
    half, nb = U // 2, n // 2
    return rlo, max(0, -(-(nb - half - rlo) // half))


def _lengths(case, seed):
    rng = np.random.default_rng(1000 + seed)
    lo, hi, m = case["nmin"], case["nmax"], case.get("ntrials", case.get("requests", 1))
    if lo == hi:
        return [lo] * m
    if lo & (lo - 1) == 0 and case["kind"] == "search":  # the production batch's lengths
        opts = [k for k in (lo, 3 * lo // 2, 2 * lo, 3 * lo, 4 * lo) if k <= hi]
        return [int(opts[i % len(opts)]) for i in rng.permutation(m)]
    # evenly over the logarithm (the sum does not depend on the seed), shuffled
    f = (np.arange(m) + 0.5) / m
    n = [2 * int(round(0.5 * lo * (hi / lo) ** x)) for x in f]
    return [n[i] for i in rng.permutation(m)]


def _mean_total_cells(case):
    """(overlap-save steps, samples) of one pass."""
    U = _uselen(case["zmax"], case["fftlen"])
    ns = _lengths(case, 0)
    return sum(_steps(n, U)[1] for n in ns), sum(ns)


def _row_flops(L, width):
    # two half-length inverse transforms, the template product, |y|^2
    M = L // 2
    return 2 * 5 * M * math.log2(M) + 2 * 6 * M + 3 * width


def _search_flops(zmax, numharm, L, steps):
    U, bank = _bank(zmax, numharm, L)
    per = sum(rows * _row_flops(Lh, U * p // q) + 2.5 * Lh * math.log2(Lh // 2)
              for p, q, _, rows, Lh, _ in bank) + (numharm - 1) * U * bank[0][3]
    return steps * per


def _fft_flops(n):
    return 2.5 * n * math.log2(n)


def work(case):
    k = case["kind"]
    if k == "stages":
        U, bank = _bank(case["zmax"], case["numharm"], case["fftlen"])
        planes = sum(r * (U * p // q) for p, q, _, r, _, _ in bank)
        segs = sum(Lh // 2 for *_, Lh, _ in bank)
        stages = case["numharm"].bit_length()
        # segments and planes are outputs of one call and inputs of the next
        b = case["nseg"] * (3 * 8 * segs + 2 * 4 * planes + 4 * stages * bank[0][3] * U)
        return {"bytes": b, "flops": _search_flops(case["zmax"], case["numharm"], case["fftlen"], case["nseg"])}
    if k in ("search", "host", "spectra"):
        steps, samples = _mean_total_cells(case)
        f = _search_flops(case["zmax"], case["numharm"], case["fftlen"], steps)
        return {"bytes": 4 * samples, "flops": f + (0 if k == "spectra" else _fft_flops(samples))}
    if k == "trial_prep":
        return {"bytes": 8 * case["n"], "flops": _fft_flops(case["n"]) + 6 * case["n"] // 2}
    if k == "dedisperse":
        mx = int(_delays(case).max())
        return {"bytes": 4 * (case["nchan"] * (case["nout"] + mx) + case["ndm"] * case["nout"]),
                "flops": case["nchan"] * case["ndm"] * case["nout"]}
    if k == "refine":
        # 75 grid points, every harmonic a correlation with its response
        taps = sum(2 * _halfwidth(case["zmax"] * h / (2 * case["numharm"])) for h in range(1, case["numharm"] + 1))
        return {"bytes": case["ncand"] * 8 * taps, "flops": case["ncand"] * 76 * taps * 8}
    steps = samples = f = 0
    for i, n in enumerate(_lengths(case, 0)):
        z = (50, 100, 200, 300)[i % 4]
        z = min(z, 200) if case["fftlen"] == 4096 else z
        s = _steps(n, _uselen(z, case["fftlen"]))[1]
        f += _search_flops(z, 8, case["fftlen"], s) + _fft_flops(n)
        samples += n
    return {"bytes": 4 * samples, "flops": f}


# --------------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(77_000 + seed)
    return g


def _signal(rng, n, rlo, zmax):
    """A sinusoid of power 120..250 (threshold: about 21), drifting by z bins."""
    amp = math.sqrt(4 * rng.uniform(120, 250) / n)
    return amp, rng.uniform(0.05, 0.35) * n + 0.25, rng.uniform(-0.6, 0.6) * zmax


def _series(n, g, sig=None):
    x = torch.randn(n, generator=g, device="cuda", dtype=torch.float32)
    if sig is not None:
        amp, r0, z = sig
        t = torch.arange(n, device="cuda", dtype=torch.float64) / n
        x += (amp * torch.cos(2 * math.pi * (r0 * t + 0.5 * z * t * t))).float()
    return x


def _trials(case, seed):
    """The trials of a search: the first, and about one in ten, hold a signal."""
    rng, g = np.random.default_rng(2000 + seed), _gen(seed)
    out = []
    for i, n in enumerate(_lengths(case, seed)):
        out.append(_series(n, g, _signal(rng, n, 16, case["zmax"]) if i % 10 == 0 else None))
    return out


def _delays(case):
    """The DM trials' delays in samples (1500 MHz top, 300 MHz band)."""
    f = 1500.0 - np.arange(case["nchan"]) * (300.0 / case["nchan"])
    dm = (case["dm0"] + case["ddm"] * np.arange(case["ndm"], dtype=np.float32)).astype(np.float64)[:, None]
    return np.floor(4.148808e3 * dm * (1.0 / (f * f) - 1.0 / 1500.0 ** 2) / DT + 0.5).astype(np.int32)


def _context(case):
    from gpu_accelsearch_gb300.search import AccelSearch
    return AccelSearch(zmax=case["zmax"], numharm=case["numharm"], fftlen=case["fftlen"],
                       chunk_segments=case.get("chunk", 0), template_fp16=bool(case.get("fp16", 0)),
                       short_transforms=bool(case.get("short", 0)))


def prepare(case, seed):
    k = case["kind"]
    if k == "stages":
        s = _context(case)
        spec, startr = _stage_inputs(case, seed)
        mk = lambda *shape: torch.zeros(shape, device="cuda", dtype=torch.float32)  # noqa: E731
        ns = case["nseg"]
        return dict(kind=k, s=s, spec=spec, startr=startr, dhalf=mk(ns, s.dhalf_stride, 2),
                    planes=mk(ns, s.plane_stride), stage=mk(ns, s.nstages, s.harmonics[0].numzs, s.uselen))
    if k == "search":
        x = _trials(case, seed)
        return dict(kind=k, s=_context(case), x=x, n=[t.numel() for t in x])
    if k == "host":
        x = [t.cpu().pin_memory() for t in _trials(case, seed)]
        return dict(kind=k, s=_context(case), x=x, n=[t.numel() for t in x])
    if k == "spectra":
        x = [_white_spectrum(t) for t in _trials(case, seed)]
        rlo = [_steps(n, _uselen(case["zmax"], case["fftlen"]))[0] for n in _lengths(case, seed)]
        return dict(kind=k, s=_context(case), x=x, rlo=rlo)
    if k == "trial_prep":
        from gpu_accelsearch_gb300.search import AccelSearch
        n = case["n"]
        s = AccelSearch(zmax=50, numharm=4, fftlen=2048, chunk_segments=16)
        return dict(kind=k, s=s, x=_red_series(n, seed), n=n,
                    spec=torch.empty((n // 2 + 1, 2), device="cuda", dtype=torch.float32))
    if k == "dedisperse":
        fb, dl = _filterbank(case, seed)
        return dict(kind=k, fb=fb, dl=dl, nout=case["nout"],
                    out=torch.empty((case["ndm"], case["nout"]), device="cuda", dtype=torch.float32))
    if k == "refine":
        s = _context(case)
        spec, cands, rlo = _refine_inputs(case, seed)
        return dict(kind=k, s=s, spec=spec, cands=cands, rlo=rlo, tobs=case["n"] * DT)
    from gpu_accelsearch_gb300.serving import Server
    x = [(t.cpu().numpy(), z) for t, z in _requests(case, seed)]
    srv = Server(hbm_budget_bytes=50e9, fftlen=case["fftlen"], numharm=8, chunk_segments=case["chunk"])
    # a running server has its banks: one small request per zmax builds them
    for z in sorted({z for _, z in x}):
        rid = srv.submit(x[0][0][: 1 << 17], DT, z)
        srv.wait(rid)
        srv.release(rid)
    return dict(kind=k, srv=srv, x=x)


def _stage_inputs(case, seed):
    U, ns = _uselen(case["zmax"], case["fftlen"]), case["nseg"]
    nb = U // 2 * (ns + 60)
    g = _gen(seed)
    spec = torch.randn((nb, 2), generator=g, device="cuda", dtype=torch.float32) * math.sqrt(0.5)
    spec[U // 2 * 40 + 316] += 9.0  # a steady tone in the first segment
    return spec, [16 + U // 2 * (40 + i) for i in range(ns)]


def _white_spectrum(x):
    n = x.numel()
    return torch.view_as_real(torch.fft.rfft(x)[: n // 2] / math.sqrt(n)).contiguous()


def _red_series(n, seed):
    """White noise plus red noise (a random walk, 4096 knots), without its mean.
    Noise whose level falls so fast over the last two whitening blocks that it
    reaches zero in the tail (about one draw in fifty; the whitened tail is
    NaN there, as in the reference) is drawn again."""
    g = _gen(seed)
    while True:
        x = torch.randn(n, generator=g, device="cuda", dtype=torch.float32)
        step = max(1, n // 4096)
        walk = torch.cumsum(torch.randn(n // step + 2, generator=g, device="cuda", dtype=torch.float32), 0) * 0.05
        t = torch.arange(n, device="cuda", dtype=torch.int64)
        i = t // step
        f = (t - i * step).float() / step
        x += walk[i] + f * (walk[i + 1] - walk[i])
        x -= x.double().mean().float()
        (s0, s1), (n0, n1) = (v[-2:] for v in _blocks(n // 2))
        p = torch.fft.rfft(x)[: n // 2].abs() ** 2
        m0, m1 = p[s0: s0 + n0].median(), p[s1: s1 + n1].median()
        if float(m1 + 1.6 * (m1 - m0)) > 0.3 * float(m0):
            return x


@functools.lru_cache(8)
def _blocks(nb):
    """First bin and width of the whitening blocks: widths 6 ln(bin), at most 200."""
    start, length, at, w = [1], [6], 7, int(6 * math.log(7))
    while at + w < nb:
        start.append(at)
        length.append(w)
        at += w
        w = min(200, int(6 * math.log(at)))
    return start, length


def _filterbank(case, seed):
    from gpu_accelsearch_gb300.dedisperse import dm_delays
    dms = (case["dm0"] + case["ddm"] * np.arange(case["ndm"], dtype=np.float32)).astype(np.float32)
    dl, mx = dm_delays(case["nchan"], 1500.0, -300.0 / case["nchan"], DT, dms)
    fb = torch.randn((case["nchan"], case["nout"] + mx), generator=_gen(seed), device="cuda", dtype=torch.float32)
    return fb, dl


def _refine_inputs(case, seed):
    """A whitened spectrum with tones, and grid candidates next to them."""
    from gpu_accelsearch_gb300.search import CAND_DTYPE
    rng, n = np.random.default_rng(3000 + seed), case["n"]
    U, _ = _bank(case["zmax"], case["numharm"], case["fftlen"])
    rlo, steps = _steps(n, U)
    spec = torch.randn((n // 2, 2), generator=_gen(seed), device="cuda", dtype=torch.float32) * math.sqrt(0.5)
    c = np.zeros(case["ncand"], CAND_DTYPE)
    tones = []
    for i in range(case["ncand"]):
        nh = min(case["numharm"], 1 << (i % 4))
        r, z = float(rng.integers(4 * U, n // 2 - 4 * U)), 2.0 * float(rng.integers(-case["zmax"] // 4, case["zmax"] // 4))
        c[i] = (0, min(steps - 1, int((r - rlo) // (U // 2))), r, z, nh, 40.0, 6.0)
        # a drifting tone slightly off the grid, at most +-80 bins wide
        tones.append((int(r), r + rng.uniform(-0.4, 0.4) - 0.5 * z, z + rng.uniform(-0.8, 0.8)))
    j = torch.arange(-80, 81, device="cuda")
    for b, r0, z in tones:
        spec[b + j] += 8.0 * torch.view_as_real(_response((r0 - (b + j)).double(), z)).float()
    return spec, c, rlo


def _requests(case, seed):
    rng, g = np.random.default_rng(4000 + seed), _gen(seed)
    out = []
    for i, n in enumerate(_lengths(case, 0)):
        z = (50, 100, 200, 300)[i % 4]
        z = min(z, 200) if case["fftlen"] == 4096 else z
        out.append((_series(n, g, _signal(rng, n, 16, z) if i % 8 == 0 else None), z))
    return [out[i] for i in rng.permutation(len(out))]


# ----------------------------------------------------------------------- run
def _split(c):
    """The candidate list as columns, in arrays of a fixed capacity."""
    cap = max(16384, len(c["r"]))
    return {f: np.pad(np.asarray(c[f]), (0, cap - len(c[f]))) for f in ("trial", "step", "numharm", "r", "z", "power", "sigma")}


def run(state):
    k = state["kind"]
    if k == "stages":
        s, ns = state["s"], len(state["startr"])
        s.prepare_segments(state["spec"].data_ptr(), state["spec"].shape[0], state["startr"],
                           state["dhalf"].data_ptr())
        s.power_planes(state["dhalf"].data_ptr(), ns, state["planes"].data_ptr())
        n = s.sum_harmonics(state["planes"].data_ptr(), state["startr"], state["stage"].data_ptr())
        return {"segments": state["dhalf"], "planes": state["planes"], "sums": state["stage"], "count": n}
    if k == "search":
        s = state["s"]
        s.search([t.data_ptr() for t in state["x"]], DT, on_device=True, nsamples=state["n"])
        return _split(s.candidates())
    if k == "host":
        s = state["s"]
        s.search_ptrs([t.data_ptr() for t in state["x"]], state["n"], DT, False)
        return _split(s.candidates())
    if k == "spectra":
        s = state["s"]
        s.search_spectra([t.data_ptr() for t in state["x"]], [t.shape[0] for t in state["x"]], state["rlo"])
        return _split(s.candidates())
    if k == "trial_prep":
        s, n = state["s"], state["n"]
        s.rfft(state["x"].data_ptr(), n, state["spec"].data_ptr())
        s.whiten(state["spec"].data_ptr(), n // 2)
        return {"spectrum": state["spec"]}
    if k == "dedisperse":
        from gpu_accelsearch_gb300.dedisperse import dedisperse
        fb = state["fb"]
        dedisperse(fb.data_ptr(), fb.shape[0], fb.shape[1], state["dl"], state["out"].data_ptr(), state["nout"],
                   torch.cuda.current_stream().cuda_stream)
        return {"trials": state["out"]}
    if k == "refine":
        o = state["s"].optimize(state["cands"], state["rlo"], state["tobs"],
                                spectra=[(state["spec"].data_ptr(), state["spec"].shape[0])])
        return {f: np.ascontiguousarray(o[f]) for f in ("r", "z", "power", "sigma", "harm_power", "f", "fdot",
                                                        "period", "pdot")}
    srv = state["srv"]
    ids = [srv.submit(x, DT, z) for x, z in state["x"]]
    out = []
    for rid in ids:
        srv.wait(rid)
        out.append(srv.result(rid)[0])
        srv.release(rid)
    r = _split(np.concatenate(out))
    r["counts"] = np.array([len(c) for c in out], np.int64)
    return r


# --------------------------------------------------------------------- exact
# The same outputs in 64-bit arithmetic from the mathematics: responses by
# Gauss-Legendre quadrature, torch.fft in complex128.
@functools.lru_cache(1)
def _nodes():
    u, w = np.polynomial.legendre.leggauss(1024)
    return torch.from_numpy(0.5 * (u + 1)).cuda(), torch.from_numpy(0.5 * w).cuda()


def _response(x, z):
    """Integral over u in [0, 1] of exp(i pi (2 x u + z u^2)): complex128."""
    u, w = _nodes()
    ph = math.pi * (2 * x[:, None] * u[None, :] + z * (u * u)[None, :])
    return torch.complex((torch.cos(ph) * w).sum(1), (torch.sin(ph) * w).sum(1))


def _templates(zh, L):
    """conj of the template spectra [rows][L] of a harmonic, z = -zh .. zh step 2."""
    k = torch.zeros((zh + 1, L), dtype=torch.complex128, device="cuda")
    for j in range(zh + 1):
        z = -zh + 2 * j
        hw = _halfwidth(z)
        t = torch.arange(-2 * hw, 2 * hw, device="cuda")
        # stored in single precision, as the reference keeps its responses
        k[j, t % L] = _response(-0.5 * z - 0.5 * t.double(), float(z)).to(torch.complex64).to(torch.complex128)
    return torch.fft.fft(k).conj()


def _rsqrt(x):
    """The reference's normalisation: magic-constant start, one Newton step."""
    i = x.to(torch.float32).view(torch.int32)
    y = (0x5F3759DF - (i >> 1)).view(torch.float32).double()
    return y * (1.5 - 0.5 * x * y * y)


def _lower_median(p):
    return torch.sort(p).values[(p.numel() - 1) // 2]


class _Exact:
    def __init__(self, case):
        self.U, self.bank = _bank(case["zmax"], case["numharm"], case["fftlen"])
        self.K = [_templates(zh, L) for _, _, zh, _, L, _ in self.bank]
        self.width = [max(_step(1_000_000 + s, self.U, p, q, hw)[1] for s in range(4 * q))
                      for p, q, _, _, _, hw in self.bank]
        self.cuts = [_power_cut(6.0, 1 << s) for s in range(case["numharm"].bit_length())]

    def segment(self, spec, startr, h):
        p, q, _, _, L, hw = self.bank[h]
        _, _, lo, nd = _step(startr, self.U, p, q, hw)
        j = torch.arange(lo, lo + L // 2, device="cuda")
        ok = (j >= 0) & (j < spec.numel())
        d = torch.where(ok, spec[j.clamp(0, spec.numel() - 1)], torch.zeros((), dtype=spec.dtype, device="cuda"))
        a = d[:nd]
        m = _lower_median(a.real ** 2 + a.imag ** 2)
        d[:nd] = a * _rsqrt(m / math.log(2.0))
        return torch.fft.fft(d)

    def plane(self, D, h):
        hw, w = self.bank[h][5], self.width[h]
        y = torch.fft.ifft(torch.cat([D, D])[None, :] * self.K[h])[:, 2 * hw: 2 * hw + w]
        return y.real ** 2 + y.imag ** 2

    def sums(self, planes, startr):
        U, zmax = self.U, self.bank[0][2]
        zz = torch.arange(-zmax, zmax + 1, 2, device="cuda")
        col = torch.arange(U, device="cuda")
        out, s = [], None
        for h, (p, q, zh, _, _, hw) in enumerate(self.bank):
            if h == 0:
                s = planes[0][:, :U].clone()
            else:
                rlo = _step(startr, U, p, q, hw)[0]
                ri = ((2 * (2 * startr + col) * p + q) // (2 * q) - 2 * rlo) & 0xFFFF
                sz = torch.sign(zz) * (zz.abs() * p // q)
                d = sz - _required_z(p, q, -zmax)
                s = s + planes[h][(torch.sign(d) * (d.abs() // 2))[:, None], ri[None, :]]
            if ((h + 1) & h) == 0:
                out.append(s.clone())
        return out

    def search(self, specs, rlos):
        got = {f: [] for f in ("trial", "step", "numharm", "r", "z", "power")}
        for t, (spec, rlo) in enumerate(zip(specs, rlos)):
            half = self.U // 2
            step, startr = 0, rlo
            while startr + half < spec.numel():
                pl = [self.plane(self.segment(spec, startr, h), h) for h in range(len(self.bank))]
                for st, s in enumerate(self.sums(pl, startr)):
                    zi, ri = torch.nonzero(s > np.float32(self.cuts[st]).item(), as_tuple=True)
                    if zi.numel():
                        zi_, ri_ = zi.cpu().numpy(), ri.cpu().numpy()
                        m = len(zi_)
                        got["trial"].append(np.full(m, t, np.int32))
                        got["step"].append(np.full(m, step, np.int32))
                        got["numharm"].append(np.full(m, 1 << st, np.int32))
                        got["r"].append(startr + 0.5 * ri_)
                        got["z"].append(-self.bank[0][2] + 2.0 * zi_)
                        got["power"].append(s[zi, ri].cpu().numpy())
                step, startr = step + 1, startr + half
        o = {f: np.concatenate(v) if v else np.zeros(0) for f, v in got.items()}
        o["sigma"] = np.array([_sigma(p, int(n)) for p, n in zip(o["power"], o["numharm"])])
        return o


def _log_gamma_q(n, x):
    return -x + math.log(sum(x ** k / math.factorial(k) for k in range(n)))


def _log_tail(s):
    return float(torch.special.log_ndtr(torch.tensor(-s, dtype=torch.float64)))


def _bisect(f, lo, hi):
    for _ in range(100):
        mid = 0.5 * (lo + hi)
        lo, hi = (mid, hi) if f(mid) > 0 else (lo, mid)
    return 0.5 * (lo + hi)


def _power_cut(sigma, n):
    t = _log_tail(sigma)
    return _bisect(lambda x: _log_gamma_q(n, x) - t, 0.0, 4096.0)


def _sigma(power, n):
    t = _log_gamma_q(n, float(power))
    return 0.0 if t >= math.log(0.5) else _bisect(lambda s: _log_tail(s) - t, 0.0, 200.0)


def _whiten(spec):
    """Spectrum [nb] complex128 divided by its running level (block medians)."""
    nb = spec.numel()
    start, length = _blocks(nb)
    s, n = torch.tensor(start, device="cuda"), torch.tensor(length, device="cuda")
    p = spec.real ** 2 + spec.imag ** 2
    j = torch.arange(int(n.max()), device="cuda")
    blk = torch.where(j[None, :] < n[:, None], p[(s[:, None] + j[None, :]).clamp(max=nb - 1)],
                      torch.full((), math.inf, dtype=torch.float64, device="cuda"))
    med = torch.sort(blk, 1).values.gather(1, ((n - 1) // 2)[:, None])[:, 0] / math.log(2.0)
    # the level is flat up to the first block's middle, then linear from
    # middle to middle, the last slope continued
    mid = s + n // 2
    slope = (med[1:] - med[:-1]) / (0.5 * (n[1:] + n[:-1]))
    r = torch.searchsorted(mid, torch.arange(nb, device="cuda"), right=True)
    sl = torch.cat([torch.zeros(1, dtype=torch.float64, device="cuda"), slope, slope[-1:]])
    base = torch.cat([med[:1], med])
    off = torch.cat([mid[:1], mid])
    # the tail continues from the last block's level
    k = (torch.arange(nb, device="cuda") - off[r]).double()
    out = spec * _rsqrt(base[r] + sl[r] * torch.where(r > 0, k, torch.zeros_like(k)))
    out[0] = 1.0
    return out


def _flat(z):
    return torch.view_as_real(z)


def _exact_refine(case, seed):
    """Three nested 5 x 5 grids around each candidate, the harmonics' power summed."""
    spec, cands, rlo = _refine_inputs(case, seed)
    X = torch.view_as_complex(spec.double())
    U, bank = _bank(case["zmax"], case["numharm"], case["fftlen"])
    hw = {(p, q): h for p, q, _, _, _, h in bank}
    out = []
    for c in cands:
        H = int(c["numharm"])
        startr = rlo + int(c["step"]) * (U // 2)
        n2 = []
        for h in range(1, H + 1):
            g = math.gcd(h, H)
            _, _, lo, nd = _step(startr, U, h // g, H // g, hw[h // g, H // g])
            j = torch.arange(lo, lo + nd, device="cuda")
            v = torch.where((j >= 0) & (j < X.numel()), X[j.clamp(0, X.numel() - 1)], torch.zeros_like(X[:1]))
            n2.append(_rsqrt(_lower_median(v.real ** 2 + v.imag ** 2) / math.log(2.0)) ** 2)

        def powers(r, z):
            got = []
            for h in range(1, H + 1):
                rr, zz = r * h / H, z * h / H
                w = _halfwidth(zz)
                j = torch.arange(math.ceil(rr - w), math.ceil(rr - w) + 2 * w, device="cuda")
                f = _response(rr - 0.5 * zz - j.double(), zz).conj()
                a = (torch.where((j >= 0) & (j < X.numel()), X[j.clamp(0, X.numel() - 1)], torch.zeros_like(f)) * f).sum()
                got.append(n2[h - 1] * (a.real ** 2 + a.imag ** 2))
            return torch.stack(got)

        r, z = float(c["r"]), float(c["z"])
        for dr, dz in ((0.25, 1.0), (1 / 16, 0.25), (1 / 64, 1 / 16)):
            at = [(r + (g // 5 - 2) * dr, z + (g % 5 - 2) * dz) for g in range(25)]
            p = torch.stack([powers(*x).sum() for x in at]).tolist()
            best = max(range(25), key=lambda g: (p[g], g == 12))
            r, z = at[best]
        p = powers(r, z).cpu().numpy()
        out.append((r, z, float(p.sum()), _sigma(p.sum(), H), np.pad(p, (0, 16 - H))))
    r, z, power, sigma = (np.array([o[i] for o in out]) for i in range(4))
    t = case["n"] * DT
    f, fdot = r / t, z / t ** 2
    return {"r": r, "z": z, "power": power, "sigma": sigma, "harm_power": np.stack([o[4] for o in out]), "f": f,
            "fdot": fdot, "period": 1 / f, "pdot": -fdot / f ** 2}


def exact(case, seed):
    k = case["kind"]
    if k == "stages":
        e = _Exact(case)
        spec, startr = _stage_inputs(case, seed)
        spec = torch.view_as_complex(spec.double())
        seg, pln, sm, count = [], [], [], 0
        pad4 = lambda v: (v + 3) & ~3  # noqa: E731
        dstride = (sum(b[4] // 2 for b in e.bank) + 31) & ~31
        pstride = (sum(b[3] * pad4(w) for b, w in zip(e.bank, e.width)) + 63) & ~63
        for r in startr:
            D = [e.segment(spec, r, h) for h in range(len(e.bank))]
            P = [e.plane(d, h) for h, d in enumerate(D)]
            S = e.sums(P, r)
            count += sum(int((s > np.float32(c).item()).sum()) for s, c in zip(S, e.cuts))
            d = torch.cat([_flat(x) for x in D])
            seg.append(torch.nn.functional.pad(d, (0, 0, 0, dstride - d.shape[0])))
            p = torch.cat([torch.nn.functional.pad(x, (0, pad4(w) - w)).reshape(-1) for x, w in zip(P, e.width)])
            pln.append(torch.nn.functional.pad(p, (0, pstride - p.numel())))
            sm.append(torch.stack(S))
        return {"segments": torch.stack(seg), "planes": torch.stack(pln), "sums": torch.stack(sm), "count": count}
    if k in ("search", "host", "spectra"):
        # with FP16 templates the list is another one (their stated error is
        # 1e-3); a batch of many trials takes minutes in 64 bits
        if case.get("fp16") or _mean_total_cells(case)[0] * _bank(case["zmax"], case["numharm"], case["fftlen"])[1][0][3] > 200_000:
            return None
        e = _Exact(case)
        ns = _lengths(case, seed)
        rlo = [_steps(n, e.U)[0] for n in ns]
        x = _trials(case, seed)
        if k == "spectra":
            specs = [torch.view_as_complex(_white_spectrum(t).double()) for t in x]
        else:
            specs = [_whiten(torch.fft.rfft(t.double())[: t.numel() // 2]) for t in x]
        return _split(e.search(specs, rlo))
    if k == "trial_prep":
        n = case["n"]
        z = torch.fft.rfft(_red_series(n, seed).double())
        z[: n // 2] = _whiten(z[: n // 2].clone())
        return {"spectrum": _flat(z)}
    if k == "dedisperse":
        fb, _ = _filterbank(case, seed)
        dl, out = _delays(case), torch.zeros((case["ndm"], case["nout"]), dtype=torch.float64, device="cuda")
        if case["nchan"] * case["ndm"] > 1 << 18:
            return None
        for c in range(case["nchan"]):
            row = fb[c].double()
            j = torch.from_numpy(dl[:, c].astype(np.int64)).cuda()[:, None]
            for d0 in range(0, case["ndm"], 32):
                out[d0: d0 + 32] += row[j[d0: d0 + 32] + torch.arange(case["nout"], device="cuda")[None, :]]
        return {"trials": out}
    if k == "refine":
        return _exact_refine(case, seed)
    return None  # a burst of requests takes minutes in 64 bits
