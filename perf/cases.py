"""What a user of the framework has it do, as cases to be timed.

The framework is the coherent search of the Polgraw all-sky pipeline and the
steps beside it.  A case is one call (or one short sequence of calls) that a
search, followup or coincidence program makes through the Python mirror of
the C-ABI (polgraw_gb300.lib):

* kind "search": one batch of sky points of one data segment
  (Context.job_core for a single point, Context.search_batch for several);
* kind "segments": several segments of uneven length together
  (Segments.search);
* kind "fstat", "grad": the followup's demodulated F-statistic and its
  adjoint gradient at a batch of points (Followup.fstatnet, fstatnet_grad);
* kind "coinc": the coincidence step over the trigger records of several
  frames (Coinc.run).

Sizes are those of the repository's configurations, tests and benchmark: 1, 2
and 6 sidereal days at dt = 2 s (N = 43082, 86164, 258492), 1 day at dt = 8 s
(N = 10771), segments of N = 60000 .. 260000, one to three detectors, 4096
followup candidates, 24 frames of 2^18 trigger records.

Inputs are Gaussian noise with gaps of zeros and injected signals, on a
circular-orbit ephemeris with sidereal rotation.  A search returns the
candidates' indices (whole numbers), their F-statistic and the trigger
records, a coincidence run its records and their members, each in the
caller's arrays of fixed capacity with the number found.  The mixed-precision
forms compute F and what follows from it (the SNR, the amplitudes, the
gradient) in 32 bits and hand it back in arrays of doubles; those outputs are
returned here in the 32 bits that they have.
"""
import importlib
import importlib.util
import math
import os
import sys

import numpy as np
import torch


def _package():
    """The package, whose folder's name is not an identifier."""
    name = "polgraw_gb300"
    if name not in sys.modules:
        d = os.path.join(os.getcwd(), "polgraw-allsky_gb300")
        spec = importlib.util.spec_from_file_location(name, os.path.join(d, "__init__.py"),
                                                      submodule_search_locations=[d])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return importlib.import_module(name + ".lib")


# ---------------------------------------------------------------------------
# the cases

def _search(name, dets, N, **kw):
    c = dict(name=name, kind="search", dets=dets, N=N, dt=2.0, band=666, fftpad=1, nsky=1, nspin=64, m5=-1e-9,
             precision="mixed", phase="fixed", trl=20.0, white=False, nospin=False, graphs=False, gaps=0.1)
    c.update(kw)
    return c


def listed():
    return [
        # one sky point of a 1-day segment at dt = 8 s, a few spindowns: the
        # smallest call, made once per sky point by a program that keeps
        # job_core() as its interface (the sizes of the golden cases)
        _search("sky_short", "H1L1", 10771, dt=8.0, band=100, nspin=9, m5=-2e-8),
        # the plain method: one detector, 2 days, one sky point x 64 spindowns
        _search("sky_h1", "H1", 86164, nspin=64),
        # the network search, the bulk of the work: 2 days of two detectors,
        # a block of the sky lattice x 200 spindowns in CUDA graphs, as the
        # benchmark runs it
        _search("net_h1l1", "H1L1", 86164, nsky=96, nspin=200, graphs=True),
        # three detectors, launched without graphs (the library's default)
        _search("net_h1l1v1", "H1L1V1", 86164, nsky=24, nspin=100),
        # long segment: 6 days, fftpad 2 (nfftf = 2^19), 400 spindowns
        _search("long_h1l1", "H1L1", 258492, fftpad=2, nsky=6, nspin=400, m5=5e-10),
        # 1 day, fftpad 2, with the FP64 spindown phase (phase mode f64)
        _search("day_f64phase", "H1L1", 43082, fftpad=2, nsky=12, nspin=75, phase="f64"),
        # the all-FP64 form, which users take to validate candidates
        _search("day_fp64", "H1L1", 43082, nsky=3, nspin=30, precision="fp64"),
        # five segments of uneven, odd lengths in one call (one CUDA graph)
        dict(name="segments", kind="segments", nseg=5, nmin=60000, nmax=260000, nsky=6, nspin=75, fftpad=2),
        # followup: F at 4096 candidates of three detectors, 2 days
        dict(name="fu_fstat", kind="fstat", dets="H1L1V1", N=86164, dt=2.0, band=666, npts=4096,
             precision="mixed", phase="f64"),
        # F and its gradient at the same candidates (one ascent step)
        dict(name="fu_grad", kind="grad", dets="H1L1V1", N=86164, dt=2.0, band=666, npts=4096,
             precision="mixed", phase="f64"),
        # the 3^4 grid around one candidate that precedes its maximisation;
        # also about the batch of a simplex over some tens of candidates
        dict(name="fu_grid", kind="fstat", dets="H1L1", N=43082, dt=2.0, band=666, npts=81,
             precision="mixed", phase="f64"),
        # coincidences among 24 frames of 2^18 trigger records
        dict(name="coinc", kind="coinc", frames=24, per_frame=1 << 18, mincoin=4, lines=256, sky=1024, signals=1000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["search"] * 6 + ["segments", "fstat", "fstat", "grad", "grad", "coinc"])
    if kind == "search":
        N = rng.choice([rng.randrange(5000, 30000), rng.randrange(30000, 131072), rng.randrange(60000, 260001)])
        fftpad = rng.choice([1, 2])
        c = _search("", rng.choice(["H1", "H1L1", "H1L1", "H1L1", "L1V1", "H1L1V1"]), N, fftpad=fftpad,
                    gaps=rng.choice([0.0, 0.1, 0.4]), graphs=rng.random() < 0.4,
                    phase=rng.choice(["fixed"] * 4 + ["f64", "ff"]), white=rng.random() < 0.1,
                    nospin=rng.random() < 0.05)
        if N < 30000:
            c.update(dt=8.0, band=100, m5=-2e-8)
        if rng.random() < 0.15:
            c["precision"], c["phase"] = "fp64", "fixed"
        # templates of the call: spindown transforms up to the largest listed case's
        per = (1 << (N - 1).bit_length()) * fftpad * (24 if c["precision"] == "fp64" else 1)
        most = max(8, (96 * 200 * 131072 // 3) // per)
        total = _log(rng, 4, most)
        c["nspin"] = max(1, min(400, total, _log(rng, 1, 400)))
        c["nsky"] = max(1, min(300, total // c["nspin"]))
        if c["nospin"]:
            c["nspin"] = 1
    elif kind == "segments":
        c = dict(kind="segments", nseg=rng.randrange(2, 7), nmin=rng.randrange(20000, 100000),
                 nmax=rng.randrange(110000, 260001), nsky=rng.randrange(1, 6), nspin=rng.randrange(5, 76),
                 fftpad=rng.choice([1, 2]))
    elif kind == "coinc":
        c = dict(kind="coinc", frames=rng.randrange(3, 25), per_frame=_log(rng, 500, 1 << 18),
                 mincoin=rng.choice([3, 4]), lines=rng.choice([64, 256]), sky=rng.choice([256, 1024]),
                 signals=rng.choice([24, 1000]))
    else:
        N, dt, band = rng.choice([(rng.randrange(8000, 20000), 8.0, 100), (rng.randrange(30000, 130000), 2.0, 666)])
        c = dict(kind=kind, dets=rng.choice(["H1", "H1L1", "H1L1V1"]), N=N, dt=dt, band=band, npts=_log(rng, 1, 2048),
                 precision="fp64" if rng.random() < 0.1 else "mixed", phase=rng.choice(["f64", "f64", "f64", "ff"]))
        if c["precision"] == "fp64":
            c["npts"] = min(c["npts"], 256)
    c.pop("name", None)
    return c


# ---------------------------------------------------------------------------
# inputs (plain numpy)

OMEGA_R = 7.2921151467064e-5
OBLIQUITY = 84381.448 / 3600.0 / (180.0 / math.pi)
SITE = {  # latitude, longitude, orientation of the arms (degrees), noise level
    "H1": (46.45515, -119.40766, 170.9994, 1.0),
    "L1": (30.56289, -90.77424, 242.7165, 1.3),
    "V1": (43.63141, 10.50450, 115.5674, 1.0),
}


def _dets(case):
    return [case["dets"][k:k + 2] for k in range(0, len(case["dets"]), 2)]


def _position(det, N, dt):
    """Detector position in units of c dt, (N, 3), and its sidereal angle at
    the first sample: a circular 1 AU orbit plus the Earth's rotation."""
    lat, lon = (math.radians(v) for v in SITE[det][:2])
    t = np.arange(N) * dt
    unit = 299792.458 * dt
    ph = 0.7 + 2 * math.pi / (365.25 * 86400.0) * t
    r = 1.49597870691e8 / unit
    phir = 1.0 + lon
    e = 6378.140 / unit
    p = np.empty((N, 3))
    p[:, 0] = r * np.cos(ph) + e * math.cos(lat) * np.cos(phir + OMEGA_R * t)
    p[:, 1] = r * math.cos(OBLIQUITY) * np.sin(ph) + e * math.cos(lat) * np.sin(phir + OMEGA_R * t)
    p[:, 2] = r * math.sin(OBLIQUITY) * np.sin(ph) + e * math.sin(lat)
    return p, phir


def _amod(det):
    """Coefficients c1..c9 of the amplitude modulation."""
    lat, _, gam = (math.radians(v) for v in SITE[det][:3])
    s2, c2, sp, cp = math.sin(2 * gam), math.cos(2 * gam), math.sin(lat), math.cos(lat)
    return [.25 * s2 * (1 + sp * sp), -.5 * c2 * sp, .5 * s2 * math.sin(2 * lat), -c2 * cp, .75 * s2 * cp * cp,
            c2 * sp, .5 * s2 * (1 + sp * sp), c2 * cp, .5 * s2 * math.sin(2 * lat)]


def _modulation(k, phir, N, dt, delta, alpha, xp=np, i=None):
    """a(t), b(t) of one detector with coefficients k."""
    w = OMEGA_R * dt * (np.arange(N, dtype=np.float64) if i is None else i)
    sd, cd, c2d = xp.sin(delta), xp.cos(delta), xp.cos(delta) ** 2
    c, s = xp.cos(alpha - phir - w), xp.sin(alpha - phir - w)
    a = k[0] * (2 - c2d) * (2 * c * c - 1) + 2 * k[1] * (2 - c2d) * c * s + k[2] * sd * cd * c + k[3] * sd * cd * s \
        + k[4] * c2d
    b = k[5] * sd * (2 * c * c - 1) + 2 * k[6] * sd * c * s + k[7] * cd * c + k[8] * cd * s
    return a, b


def _source(delta, alpha):
    return np.array([math.cos(alpha) * math.cos(delta), math.sin(alpha) * math.cos(delta), math.sin(delta)])


def _data(dets, N, dt, oms, rng, signals, gaps):
    """Noise, gaps and signals (f, s, delta, alpha, snr) of each detector."""
    out, amp = [], [0.55, 0.32, -0.38, 0.51]
    i = np.arange(N, dtype=np.float64)
    xs, sig = [], [np.zeros((len(dets), N)) for _ in signals]
    for n, d in enumerate(dets):
        p, phir = _position(d, N, dt)
        x = rng.standard_normal(N) * SITE[d][3]
        keep = np.ones(N, dtype=bool)
        for _ in range(int(round(gaps * 40))):
            g = int(rng.integers(0, N))
            keep[g:g + N // 40] = False
        k = _amod(d)
        for q, (f, s, delta, alpha, snr) in enumerate(signals):
            a, b = _modulation(k, phir, N, dt, delta, alpha)
            sh = p @ _source(delta, alpha)
            ph = f * i + s * i * i + (oms + f + 2 * s * i) * sh
            sig[q][n] = amp[0] * a * np.cos(ph) + amp[2] * a * np.sin(ph) + amp[1] * b * np.cos(ph) + \
                amp[3] * b * np.sin(ph)
        xs.append((x, keep, p, phir, k))
    for n, (x, keep, p, phir, k) in enumerate(xs):
        for q, (_, _, _, _, snr) in enumerate(signals):
            x = x + snr / math.sqrt(float((sig[q] ** 2).sum())) * sig[q][n]
        x = np.where(keep, x, 0.0)
        out.append(dict(x=x, pos=p, phir=phir, amod=k, sig2=float(N / keep.sum() * x.var(ddof=1))))
    return out


def _sky(pm, mm, nn, spacing):
    """Declination and right ascension of a point of the square lattice."""
    be1, be2 = nn * spacing, mm * spacing
    se, ce = math.sin(OBLIQUITY), math.cos(OBLIQUITY)
    sd = be1 * se - (2 * pm - 3) * math.sqrt(1 - be1 * be1 - be2 * be2) * ce
    cd = math.sqrt(1 - sd * sd)
    return math.asin(sd), math.fmod(math.atan2((be1 - se * sd) / (ce * cd), be2 / cd) + 2 * math.pi, 2 * math.pi)


def _segment(case, rng):
    """Everything a search of one segment is given, in plain values."""
    N, dt, fftpad = case["N"], case["dt"], case["fftpad"]
    nfft = 1 << (N - 1).bit_length()
    fpo = 10. + 0.96875 * case["band"] * (0.5 / dt)
    oms = 2 * math.pi * fpo * dt
    spacing = math.sqrt(math.pi / 2000)
    # two signals on one point of the lattice, and the sky points around it
    half = int(1 / spacing) + 1
    lattice = [(1, mm, nn) for mm in range(-half, half + 1) for nn in range(-half, half + 1)
               if (mm * mm + nn * nn) * spacing ** 2 < 0.98]
    at = int(rng.integers(len(lattice) // 4, 3 * len(lattice) // 4))
    first = max(0, min(at - case["nsky"] // 2, len(lattice) - case["nsky"]))
    tasks = lattice[first:first + case["nsky"]]
    delta, alpha = _sky(*lattice[at], spacing)
    m5 = 0.0 if case["nospin"] else case["m5"]
    signals = [(float(rng.uniform(0.3, 2.7)), m5 * float(rng.uniform(0, max(1, case["nspin"] - 1))), delta, alpha,
                float(rng.uniform(7.5, 9.5))) for _ in range(2)]
    B = 0.5 / dt
    return dict(N=N, dt=dt, fftpad=fftpad, nfft=nfft, fpo=fpo, oms=oms, B=B, spacing=spacing, m5=case["m5"],
                nmin=int(fftpad * 4096 * B), nmax=int((nfft // 2 - 4096 * B) * fftpad), tasks=tasks,
                nspin=case["nspin"], trl=case["trl"], white=case["white"], nospin=case["nospin"],
                dets=_data(_dets(case), N, dt, oms, rng, signals, case["gaps"]))


def _segment_cases(case, rng):
    out = []
    for _ in range(case["nseg"]):
        N = int(rng.integers(case["nmin"], case["nmax"] + 1))
        out.append(_search("", "H1L1", N, fftpad=case["fftpad"], nsky=case["nsky"], nspin=case["nspin"], gaps=0.0))
    return out


def _points(case, rng):
    """Data with four signals and npts points within half a peak width."""
    N, dt = case["N"], case["dt"]
    oms = 2 * math.pi * (10. + 0.96875 * case["band"] * (0.5 / dt)) * dt
    sc = 8.0 / dt * (10771.0 / N) ** 2 if dt > 4 else 1.0
    signals = [(float(rng.uniform(0.3, 2.7)), float(rng.uniform(-1e-8, 1e-8)) * sc, float(rng.uniform(-1.2, 1.2)),
                float(rng.uniform(0, 6.28)), float(rng.uniform(10, 15))) for _ in range(4)]
    dets = _data(_dets(case), N, dt, oms, rng, signals, 0.1)
    pts = np.empty((case["npts"], 4))
    for q, (f, s, delta, alpha, _) in enumerate(signals):
        w = [2 * math.pi / N, 2 * math.pi / float(N) ** 2, 0.0, 0.0]
        sd, cd, sa, ca = math.sin(delta), math.cos(delta), math.sin(alpha), math.cos(alpha)
        for d in dets:
            for j, v in ((2, [-ca * sd, -sa * sd, cd]), (3, [-sa * cd, ca * cd, 0.0])):
                w[j] = max(w[j], float(np.ptp(d["pos"] @ np.array(v))))
        w[2:] = [2 * math.pi / (oms * v) for v in w[2:]]
        n = len(pts[q::4])
        pts[q::4] = np.array([f, s, delta, alpha]) + rng.uniform(-0.5, 0.5, (n, 4)) * np.array(w)
    return dict(N=N, dt=dt, oms=oms, dets=dets, points=pts)


def _triggers(case, rng):
    """Trigger records (f, s, delta, alpha, snr) of each frame: a lattice of
    lines, spindowns and sky positions with exact duplicates, a continuous
    part around the lines, and signals that most frames have."""
    N, refr = 86164, (case["frames"] + 1) // 2
    oms = 2 * math.pi * (10. + 0.96875 * 666 * 0.25) * 2.0
    step_f, step_s = 4.0 / N, 8.0 / float(N) ** 2
    fl = rng.uniform(0.3, 2.8, case["lines"])
    sky_d, sky_a = rng.uniform(-1.3, 1.3, case["sky"]), rng.uniform(0, 6.2, case["sky"])
    sg = rng.random((case["signals"], 5))
    snrs = np.array([5.5, 6.5, 7.0, 7.0, 8.25, 9.0])
    out = []
    for fr in range(1, case["frames"] + 1):
        n = case["per_frame"]
        r = np.empty((n, 5))
        line, sky = rng.integers(0, case["lines"], n), rng.integers(0, case["sky"], n)
        lat = rng.random(n) < 0.5
        u = rng.random((3, n))
        r[:, 0] = fl[line] + step_f * np.where(lat, np.floor(9 * u[0]) - 4, 40 * (u[0] - 0.5))
        r[:, 1] = step_s * np.where(lat, 2 * np.floor(3 * u[1]) - 2, 16 * (u[1] - 0.5))
        off = np.where(lat, 0.0, 1e-4 * (u[2] - 0.5))
        r[:, 2], r[:, 3] = sky_d[sky] + off, sky_a[sky] - off
        r[:, 4] = np.where(lat, snrs[(6 * u[2]).astype(np.int64)], 4 + 6 * u[2])
        js = np.nonzero(rng.random(case["signals"]) < 0.8)[0]
        s = np.empty((len(js), 5))
        s[:, 1] = (sg[js, 1] - 0.5) * 64 * step_s
        s[:, 0] = 0.3 + 2.5 * sg[js, 0] - 2 * s[:, 1] * N * (refr - fr)
        s[:, 2], s[:, 3], s[:, 4] = -1.3 + 2.6 * sg[js, 2], 6.2 * sg[js, 3], 7 + 3 * sg[js, 4]
        put = rng.permutation(n)[:len(js)]
        r[put] = s[:len(put)]
        out.append(r)
    # cells 8 x 16 wide in (f N, s N^2) and 2e6 in the sky coordinates, turned
    c0, s0, c1, s1 = math.cos(0.3), math.sin(0.3), math.cos(0.5), math.sin(0.5)
    Q = np.array([[c0, -s0, 0, 0], [s0, c0, 0, 0], [0, 0, c1, -s1], [0, 0, s1, c1]])
    fisher = Q @ np.diag([8.0 ** -2, 16.0 ** -2, 2.0e6 ** -2, 2.0e6 ** -2]) @ Q.T
    return dict(N=N, oms=oms, refr=refr, frames=out, fisher=fisher, mincoin=case["mincoin"])


# ---------------------------------------------------------------------------
# what a program has before the call, and the call

def _settings(L, g, nifo):
    s = L.Settings()
    s.fpo, s.dt, s.B, s.oms, s.omr = g["fpo"], g["dt"], g["B"], g["oms"], OMEGA_R * g["dt"]
    s.Smin, s.Smax = 2 * math.pi * 0.5e-9 * g["dt"] ** 2, 2 * math.pi * 0.5e-8 * g["dt"] ** 2
    s.sepsm, s.cepsm = math.sin(OBLIQUITY), math.cos(OBLIQUITY)
    s.N, s.nfft, s.fftpad, s.interpftpad = g["N"], g["nfft"], g["fftpad"], 2
    s.nod, s.s, s.nd, s.nifo = max(1, round(g["N"] * g["dt"] / 86164.0)), 1, 2, nifo
    s.Ninterp, s.nfftf = 2 * g["nfft"], g["fftpad"] * g["nfft"]
    s.nmin, s.nmax = g["nmin"], g["nmax"]
    s.M[0], s.M[5] = 2 * math.pi / s.nfftf, g["m5"]
    s.M[10] = s.M[15] = g["spacing"] * g["oms"]
    return s


def _detectors(L, dets):
    return L.make_detectors([d["x"] for d in dets], [d["pos"].reshape(-1) for d in dets], [d["sig2"] for d in dets],
                            [math.sin(d["phir"]) for d in dets], [math.cos(d["phir"]) for d in dets],
                            [d["amod"] for d in dets])


def _context(L, case, g):
    arr, keep = _detectors(L, g["dets"])
    nifo = len(g["dets"])
    ctx = L.Context(_settings(L, g, nifo), arr, nifo, precision=1 if case["precision"] == "fp64" else 0,
                    phase_mode=L.PHASE_NAMES[case["phase"]])
    o, r = L.Opts(g["trl"], int(g["white"]), int(g["nospin"]), 1), L.Range()
    r.spndr[0], r.spndr[1], r.sst = 0, g["nspin"] - 1, 0
    return ctx, o, r


def prepare(case, seed):
    L = _package()
    rng = np.random.default_rng([int(seed), 77])
    if case["kind"] == "search":
        g = _segment(case, rng)
        ctx, o, r = _context(L, case, g)
        ctx.set_graphs(case["graphs"])
        return dict(kind="search", ctx=ctx, opts=o, range=r, tasks=g["tasks"], fp64=case["precision"] == "fp64",
                    out=_room(case), filled={})
    if case["kind"] == "segments":
        parts = []
        for c in _segment_cases(case, rng):
            g = _segment(c, rng)
            parts.append((*_context(L, c, g), g["tasks"]))
        return dict(kind="segments", seg=L.Segments([p[0] for p in parts]), tasks=[p[3] for p in parts],
                    opts=[p[1] for p in parts], ranges=[p[2] for p in parts], out=[_room(case) for _ in parts],
                    filled=[{} for _ in parts])
    if case["kind"] == "coinc":
        t = _triggers(case, rng)
        cc = L.Coinc(L.coinc_cfg(N=t["N"], oms=t["oms"], vedva_m=L.vedva(t["fisher"]), refr=t["refr"],
                                 mincoin=t["mincoin"]))
        for k, r in enumerate(t["frames"]):
            cc.add_frame(k + 1, r)
        n = case["frames"] * case["per_frame"]
        most, members = n // 8 + 1024, n // 4 + 32768
        return dict(kind="coinc", cc=cc, out=dict(
            w=np.zeros(most, np.int32), first=np.zeros(most, np.int32), mean=np.zeros((most, 5)),
            frame=np.zeros(members, np.int32), position=np.zeros(members, np.int32)), filled={})
    g = _points(case, rng)
    s = L.Settings()
    s.N, s.oms, s.omr = g["N"], g["oms"], OMEGA_R * g["dt"]
    arr, keep = _detectors(L, g["dets"])
    fu = L.Followup(s, arr, len(g["dets"]), precision=1 if case["precision"] == "fp64" else 0,
                    phase_mode=L.PHASE_NAMES[case["phase"]])
    return dict(kind=case["kind"], fu=fu, points=g["points"], fp64=case["precision"] == "fp64")


def _room(case):
    """A caller's arrays for the candidates of one batch."""
    n = case["nsky"] * case["nspin"]
    n = 512 if n <= 64 else 4096 if n <= 1000 else 16384
    return dict(index=np.zeros((n, 5), np.int32), F=np.zeros(n, np.float32), record=np.zeros((n, 4)),
                snr=np.zeros(n, np.float64 if case.get("precision") == "fp64" else np.float32))


def _put(to, rows, at):
    """The rows found into the caller's arrays, zeros behind them where a
    call before this one left rows."""
    for k, v in rows.items():
        n = len(v)
        to[k][:n] = v
        to[k][n:max(n, at.get(k, len(to[k])))] = 0
        at[k] = n
    return to


def _found(to, at, rec, idx, fnum):
    """Candidates: whole-number indices, F, the trigger records' coordinates
    (formed in FP64 by every form) and SNR, and the number of spindowns."""
    index = np.stack([idx[k] for k in ("pm", "mm", "nn", "ss", "ii")], axis=1)
    _put(to, dict(index=index, F=idx["F"], record=rec[:, :4], snr=rec[:, 4]), at)
    return dict(to, found=len(rec), spindowns=int(fnum))


def run(state):
    k = state["kind"]
    if k == "search":
        t = state["tasks"]
        if len(t) == 1:
            return _found(state["out"], state["filled"], *state["ctx"].job_core(*t[0], state["opts"], state["range"]))
        return _found(state["out"], state["filled"], *state["ctx"].search_batch(t, state["opts"], state["range"]))
    if k == "segments":
        found = state["seg"].search(state["tasks"], state["opts"], state["ranges"])
        return [_found(to, at, *r) for to, at, r in zip(state["out"], state["filled"], found)]
    if k == "coinc":
        r = state["cc"].run()
        _put(state["out"], dict(w=r.w, first=r.first, mean=r.mean, frame=r.fra, position=r.ops), state["filled"])
        return dict(state["out"], found=len(r.w), members=len(r.fra), frameinfo=r.frameinfo)
    as_is = (lambda v: v) if state["fp64"] else (lambda v: v.astype(np.float32))
    if k == "fstat":
        out = state["fu"].fstatnet(state["points"])
        return dict(F=as_is(out[:, 5]), amplitudes=as_is(out[:, :4]), snr=as_is(out[:, 4]), snr_amp=as_is(out[:, 10]),
                    point=out[:, 6:10])
    F, g = state["fu"].fstatnet_grad(state["points"])
    return dict(F=as_is(F), dF=as_is(g))


def work(case):
    """Inputs read once and results written once; flops of the transforms
    (5 L log2 L), the phase and detector sums and the F-statistic."""
    def search(c):
        N, nifo, nfft = c["N"], len(_dets(c)), 1 << (c["N"] - 1).bit_length()
        L = nfft * c["fftpad"]
        sky = nifo * (4 * 5 * nfft * math.log2(nfft) + 250 * N)
        spin = 2 * 5 * L * math.log2(L) + 40 * nifo * N + 10 * (L // 2)
        return dict(bytes=32 * nifo * N + 64 * c["nsky"], flops=c["nsky"] * (sky + c["nspin"] * spin))
    if case["kind"] == "search":
        return search(case)
    if case["kind"] == "segments":
        mid = (case["nmin"] + case["nmax"]) // 2
        w = search(_search("", "H1L1", mid, fftpad=case["fftpad"], nsky=case["nsky"], nspin=case["nspin"]))
        return {k: v * case["nseg"] for k, v in w.items()}
    if case["kind"] == "coinc":
        n = case["frames"] * case["per_frame"]
        return dict(bytes=40 * n, flops=60 * n)
    nifo, n = len(_dets(case)), case["npts"]
    return dict(bytes=32 * nifo * case["N"] + 120 * n, flops=(60 if case["kind"] == "fstat" else 180) * nifo * case["N"] * n)


# ---------------------------------------------------------------------------
# the same in 64 bits, in plain torch

def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _resample(x, N, nfft, shftf):
    """x (2, N) at the times i - shftf: interpolation by two through the
    zero-padded spectrum, then a natural cubic spline through 2N points."""
    X = torch.fft.fft(x, n=nfft)
    q = nfft // 2 + 1
    Z = torch.zeros((2, 2 * nfft), dtype=X.dtype, device=X.device)
    Z[:, :q] = X[:, :q]
    Z[:, q + nfft:] = X[:, q:]
    y = torch.fft.ifft(Z)[:, :2 * N] * 2
    n = 2 * N
    # second derivatives: the tridiagonal (1, 4, 1) system with zero ends,
    # solved in the sine basis (odd extension)
    d = torch.zeros_like(y)
    d[:, 1:-1] = 6 * (y[:, :-2] - 2 * y[:, 1:-1] + y[:, 2:])
    e = torch.cat([d, -torch.flip(d[:, 1:-1], [1])], dim=1)
    k = torch.arange(e.shape[1], dtype=torch.float64, device=x.device)
    z = torch.fft.ifft(torch.fft.fft(e) / (4 + 2 * torch.cos(2 * math.pi * k / e.shape[1])))[:, :n]
    z[:, 0] = z[:, -1] = 0
    at = 2 * (torch.arange(N, dtype=torch.float64, device=x.device) - shftf)
    lo = at.floor().clamp(0, n - 1).long()
    hi = (lo + 1).clamp(max=n - 1)
    b = at - lo
    a = 1 - b
    v = a * y[:, lo] + b * y[:, hi] + ((a ** 3 - a) * z[:, lo] + (b ** 3 - b) * z[:, hi]) / 6
    return torch.where((at < 0) | (at > n - 1), torch.zeros_like(v), v)


def _exact_search(case, g, chunk=16):
    dev, N, L = _dev(), g["N"], g["nfft"] * g["fftpad"]
    i = torch.arange(N, dtype=torch.float64, device=dev)
    dets = [dict(x=torch.tensor(d["x"], device=dev), pos=torch.tensor(d["pos"], device=dev), **{k: d[k] for k in (
        "phir", "amod", "sig2")}) for d in g["dets"]]
    index, Fs, recs = [], [], []
    m5 = 0.0 if g["nospin"] else g["m5"]
    spins = [g["nspin"] - 1] if g["nospin"] else list(range(g["nspin"]))
    for pm, mm, nn in g["tasks"]:
        delta, alpha = _sky(pm, mm, nn, g["spacing"])
        src = torch.tensor(_source(delta, alpha), device=dev)
        aa = bb = 0.0
        xm, t1 = [], []
        for d in dets:
            a, b = _modulation(d["amod"], d["phir"], N, g["dt"], torch.tensor(delta, device=dev, dtype=torch.float64),
                               alpha, torch, i)
            sh = d["pos"] @ src
            ph = torch.exp(-1j * (g["oms"] * sh))
            xm.append(_resample(torch.stack([d["x"] * a * ph, d["x"] * b * ph]), N, g["nfft"], sh - sh[0]) / d["sig2"])
            t1.append(i * i + 2 * i * sh)
            aa, bb = aa + float((a * a).sum()) / d["sig2"], bb + float((b * b).sum()) / d["sig2"]
        for c0 in range(0, len(spins), chunk):
            ss = spins[c0:c0 + chunk]
            s1 = torch.tensor([k * m5 for k in ss], dtype=torch.float64, device=dev)[:, None]
            z = torch.zeros((2, len(ss), N), dtype=torch.complex128, device=dev)
            for x, t in zip(xm, t1):
                e = torch.exp(-1j * (s1 * t))
                z[0] += x[0] * e
                z[1] += x[1] * e
            Z = torch.fft.fft(z, n=L)[:, :, g["nmin"]:g["nmax"]]
            F = (Z[0].real ** 2 + Z[0].imag ** 2) / aa + (Z[1].real ** 2 + Z[1].imag ** 2) / bb
            nb = F.shape[1] // 4096
            if not g["white"] and nb:
                blk = F[:, :nb * 4096].reshape(len(ss), nb, 4096)
                F[:, :nb * 4096] = (blk / (blk.sum(dim=2, keepdim=True) / 8192)).reshape(len(ss), nb * 4096)
            hit = torch.nonzero(F > g["trl"]).cpu().numpy()
            val = F[F > g["trl"]].cpu().numpy()
            p = 0
            while p < len(hit):  # runs of bins: the largest value, the later one of equal ones
                q = p
                while q + 1 < len(hit) and hit[q + 1, 0] == hit[p, 0] and hit[q + 1, 1] == hit[q, 1] + 1:
                    q += 1
                best = max(range(p, q + 1), key=lambda t: (val[t], t))
                k, ii = ss[hit[best, 0]], int(hit[best, 1]) + g["nmin"]
                index.append((pm, mm, nn, k, ii))
                Fs.append(float(val[best]))
                recs.append((2 * math.pi * ii / L, k * m5, delta, alpha))
                p = q + 1
    to = {k: np.zeros(v.shape, v.dtype if v.dtype == np.int32 else np.float64) for k, v in _room(case).items()}
    n, F = len(Fs), np.array(Fs)
    to["F"][:n], to["snr"][:n] = F, np.sqrt(2 * (F - 2))
    if n:
        to["index"][:n], to["record"][:n] = np.array(index), np.array(recs)
    return dict(to, found=n, spindowns=len(g["tasks"]) * len(spins))


def _exact_points(case, g, chunk):
    dev, N = _dev(), g["N"]
    i = torch.arange(N, dtype=torch.float64, device=dev)
    dets = [dict(x=torch.tensor(d["x"], device=dev), pos=torch.tensor(d["pos"], device=dev), **{k: d[k] for k in (
        "phir", "amod", "sig2")}) for d in g["dets"]]
    grad = case["kind"] == "grad"
    sums, Fs, grads = [], [], []
    for c0 in range(0, len(g["points"]), chunk):
        p = torch.tensor(g["points"][c0:c0 + chunk], device=dev, requires_grad=grad)
        f, s, delta, alpha = (p[:, j:j + 1] for j in range(4))
        tot = [0.0] * 6
        for d in dets:
            a, b = _modulation(d["amod"], d["phir"], N, g["dt"], delta, alpha, torch, i[None])
            r = d["pos"]
            sh = torch.cos(alpha) * torch.cos(delta) * r[:, 0] + torch.sin(alpha) * torch.cos(delta) * r[:, 1] + \
                torch.sin(delta) * r[:, 2]
            ph = f * (i + sh) + s * i * i + (g["oms"] + 2 * s * i) * sh
            c, sn = d["x"] * torch.cos(ph), d["x"] * torch.sin(ph)
            for j, v in enumerate((a * c, -a * sn, b * c, -b * sn, a * a, b * b)):
                tot[j] = tot[j] + v.sum(dim=1) / d["sig2"]
        xr, xi, yr, yi, A, B = tot
        F = (xr * xr + xi * xi) / A + (yr * yr + yi * yi) / B
        if grad:
            grads.append(torch.autograd.grad(F.sum(), p)[0].cpu().numpy())
        Fs.append(F.detach().cpu().numpy())
        sums.append(torch.stack(tot, dim=1).detach().cpu().numpy())
    F, (xr, xi, yr, yi, A, B) = np.concatenate(Fs), np.concatenate(sums).T
    if grad:
        gr = np.concatenate(grads)
        return dict(F=F, dF=gr)
    with np.errstate(invalid="ignore"):
        snr = np.sqrt(2 * (F - 2))
    return dict(F=-F, amplitudes=np.stack([2 * xr / A, 2 * yr / B, -2 * xi / A, -2 * yi / B], axis=1), snr=snr,
                snr_amp=2 * np.sqrt(xr ** 2 + xi ** 2 + yr ** 2 + yi ** 2), point=g["points"])


def exact(case, seed):
    rng = np.random.default_rng([int(seed), 77])
    if case["kind"] == "search":
        return _exact_search(case, _segment(case, rng))
    if case["kind"] == "segments":
        return [_exact_search(case, _segment(c, rng)) for c in _segment_cases(case, rng)]
    if case["kind"] == "coinc":
        # whole numbers, and means of the records themselves: the order of the
        # sums, which FP64 already takes, is what the result is
        return None
    return _exact_points(case, _points(case, rng), 32 if case["kind"] == "fstat" else 16)
