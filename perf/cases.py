"""The timed cases of the trajectory framework, each one call that a program makes.

A case names an operation, a system, a precision and sizes.  The operations are the
public entry points of hawaiihybrid_b200:

  corr    C(t) of an ensemble: sampled initial conditions, both branches of every
          trajectory, the dipole at N sample times (correlation_iterations, or
          correlation_temperatures when several temperatures go in one call)
  moment  the Monte Carlo zeroth moment at nT temperatures (calculate_m0)
  prmu    one pass of the PR_MU spectral function (prmu_iteration)
  sf      C(t) -> spectral function (idct_cf_to_sf)

The physical settings (masses, surfaces, R ranges, tolerances, dt) are those of the
benchmark's workloads; the seed of a case draws its trajectories or samples.

exact() restates in numpy / torch, in 64 bits, what needs no fitted coefficient
tables: the He-Ar pair (analytic surface) and the transform.  The other surfaces are
tables of thousands of coefficients that only the repository holds, so they have no
independent value here.
"""
import math

import numpy as np
import torch

import hawaiihybrid_b200 as hh
from hawaiihybrid_b200 import hawaii

HTOCM = 2.1947463136320e5
# masses, moments of inertia, sampler ranges and sampling intervals of the workloads
SYSTEMS = {
    "hear": dict(mu=6.632039160324215e+03, pesmin=-9.424412560638486e-05, Rmin=4.0, dt=200.0),
    "co2ar": dict(mu=3.817083069753919e+04, II=2.819827114123505e+05, pesmin=-8.913727688689150e-04, Rmin=4.0,
                  dt=100.0),
    "n2ar": dict(mu=30016.287464295514, II=55141.90310147907, pesmin=-97.3 / HTOCM, Rmin=4.51, dt=100.0),
    "ch4co2": dict(mu=2.141790360592430e+04, II1=2.093840965876434e+04, II2=2.819827114123505e+05,
                   pesmin=-1.562522273622102e-03, Rmin=4.751, dt=200.0),
}
PREC = {"fp64": hh.PRECISION_FP64, "mixed": hh.PRECISION_MIXED}
# half-trajectory work of one trajectory on the benchmark's workloads: right-hand sides
# evaluated and dipole samples stored by both branches together (a sample count is
# bounded by 2 N), flops of one right-hand side (with its share of the step) and of one
# sample's dipole
TRAJ = {
    "hear": dict(rhs=1200, samples=1100, f_rhs=260, f_dip=70),
    "co2ar": dict(rhs=830, samples=3300, f_rhs=560, f_dip=300),
    "n2ar": dict(rhs=1100, samples=3500, f_rhs=3300, f_dip=600),
    "ch4co2": dict(rhs=300, samples=40, f_rhs=900, f_dip=70000),
}


def listed():
    return [
        # a quick look at a pair on a short grid: the smallest call of the ensemble path,
        # set by launches and latency (He-Ar, FP64, the default precision)
        dict(name="hear_fp64_64x1024", op="corr", system="hear", prec="fp64", n=64, N=1024, T=300.0, iters=1),
        # the He-Ar atom-atom workload: 10,240 trajectories, 65,536 samples
        dict(name="hear_fp64_10240x65536", op="corr", system="hear", prec="fp64", n=10240, N=65536, T=300.0, iters=1),
        # the headline CO2-Ar workload, four iterations per launch as
        # calculate_correlation_and_save groups them, batched mixed-precision path
        dict(name="co2ar_mixed_4x102400x32768", op="corr", system="co2ar", prec="mixed", n=102400, N=32768, T=300.0,
             iters=4),
        # one iteration of the same on the plain FP64 path (the drop-in)
        dict(name="co2ar_fp64_102400x32768", op="corr", system="co2ar", prec="fp64", n=102400, N=32768, T=300.0,
             iters=1),
        # N2-Ar with the PIP-NN surfaces, half of the benchmark's ensemble, mixed path
        dict(name="n2ar_mixed_131072x16384", op="corr", system="n2ar", prec="mixed", n=131072, N=16384, T=200.0,
             iters=1),
        # N2-Ar in FP64: an ensemble of an odd size on a grid that is no power of two
        dict(name="n2ar_fp64_20011x5000", op="corr", system="n2ar", prec="fp64", n=20011, N=5000, T=200.0, iters=1),
        # CH4-CO2 at 100, 200, 300 and 400 K in one call (the reference's example
        # settings: 21 samples), both precisions
        dict(name="ch4co2_mixed_4x65536x21", op="corr", system="ch4co2", prec="mixed", n=65536, N=21, T=100.0, nT=4),
        dict(name="ch4co2_fp64_4x25013x21", op="corr", system="ch4co2", prec="fp64", n=25013, N=21, T=100.0, nT=4),
        # CO2-Ar zeroth moment at 16 temperatures: the benchmark's 1e8 samples on the
        # mixed path, a fifth of it in FP64
        dict(name="m0_mixed_16T_1e8", op="moment", system="co2ar", prec="mixed", n=100_000_000, nT=16),
        dict(name="m0_fp64_16T_2e7", op="moment", system="co2ar", prec="fp64", n=20_000_000, nT=16),
        # the PR_MU spectrum of CO2-Ar, FP64
        dict(name="prmu_fp64_4096x4096", op="prmu", system="co2ar", prec="fp64", n=4096, N=4096, T=300.0),
        # the spectral function of one C(t) of the He-Ar workload's length
        dict(name="sf_65536", op="sf", N=65536),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["corr"] * 7 + ["moment", "moment", "prmu", "sf"])
    if op == "sf":
        return dict(op="sf", N=1 << rng.randint(8, 16), scale=round(rng.uniform(0.5, 2.0), 3))
    if op == "moment":
        return dict(op="moment", system=rng.choice(["hear", "co2ar", "co2ar"]), prec=rng.choice(["fp64", "mixed"]),
                    n=_log(rng, 10_000, 20_000_000), nT=rng.randint(1, 16))
    T = round(rng.uniform(120.0, 400.0), 1)
    if op == "prmu":
        return dict(op="prmu", system=rng.choice(["hear", "co2ar"]), prec=rng.choice(["fp64", "mixed"]),
                    n=_log(rng, 64, 4096), N=1 << rng.randint(9, 12), T=T)
    system = rng.choice(["hear", "co2ar", "co2ar", "n2ar", "ch4co2"])
    prec = rng.choice(["fp64", "mixed"])
    if system == "ch4co2":
        return dict(op="corr", system=system, prec=prec, n=_log(rng, 500, 60_000 if prec == "mixed" else 25_000),
                    N=rng.randint(9, 33), T=100.0, nT=rng.randint(2, 4))
    big = {("hear", "fp64"): 10_240, ("hear", "mixed"): 10_240, ("co2ar", "fp64"): 60_000,
           ("co2ar", "mixed"): 200_000, ("n2ar", "fp64"): 20_000, ("n2ar", "mixed"): 100_000}[system, prec]
    longest = {"hear": 65536, "co2ar": 32768, "n2ar": 5000 if prec == "fp64" else 16384}[system]
    return dict(op="corr", system=system, prec=prec, n=_log(rng, 64, big), N=_log(rng, 512, longest), T=T,
                iters=rng.choice([1, 1, 2]) if prec == "mixed" else 1)


def _ms(system, seed):
    s = SYSTEMS[system]
    if system == "hear":
        return hh.init_ms(s["mu"], hh.ATOM, hh.ATOM, None, None, seed)
    if system == "ch4co2":
        return hh.init_ms(s["mu"], hh.ROTOR, hh.LINEAR_MOLECULE, (s["II1"],) * 3, (s["II2"],) * 2, seed)
    sid = hh.SYSTEM_CO2_AR if system == "co2ar" else hh.SYSTEM_N2_AR
    return hh.init_ms(s["mu"], hh.LINEAR_MOLECULE, hh.ATOM, (s["II"],) * 2, None, seed, system_id=sid)


def _seed(seed):
    return 1 + (int(seed) * 2654435761 + 12345) % 0x7FFFFFF0


def _cf(case, seed):
    """A C(t) of the shape the path gives: a decaying, noisy correlation function."""
    N = case["N"]
    rng = np.random.default_rng(int(seed))
    t = np.arange(N) / N
    width = rng.uniform(0.02, 0.06)
    c = 1e-60 * case.get("scale", 1.0) * np.exp(-(t / width) ** 2) * np.cos(40.0 * t)
    return c + 1e-64 * rng.standard_normal(N)


def prepare(case, seed):
    op = case["op"]
    if op == "sf":
        # the device context that computed C(t), and C(t)
        _ms("hear", 1)
        dt = SYSTEMS["hear"]["dt"]
        return dict(op=op, t=dt * np.arange(case["N"]), cf=_cf(case, seed))
    s = SYSTEMS[case["system"]]
    sd = _seed(seed)
    p = hh.CalcParams(ps=1, sampler_Rmin=s["Rmin"], sampler_Rmax=40.0, pesmin=s["pesmin"], sampling_time=s["dt"],
                      MaxTrajectoryLength=case.get("N", 64), Rcut=40.0, cvode_tolerance=1e-12, mixed_tolerance=3e-8,
                      partial_partition_function_ratio=1.0)
    if op == "prmu":
        p.sampling_time = 200.0
    st = dict(op=op, ms=_ms(case["system"], sd), p=p, seed=sd, prec=PREC[case["prec"]], n=case["n"], T=case.get("T"),
              iters=case.get("iters", 1), nT=case.get("nT", 1), many="nT" in case and op == "corr")
    st["Ts"] = _temperatures(case)
    return st


def _temperatures(case):
    if case["op"] == "moment":
        return np.linspace(150.0, 400.0, case["nT"]) if case["nT"] > 1 else np.array([300.0])
    return np.array([100.0 * (i + 1) for i in range(case.get("nT", 1))])


def run(st):
    op = st["op"]
    if op == "sf":
        # the transform apodizes the C(t) it is given in place: a program hands it a copy
        # when it keeps its own
        cf = hh.CFnc(t=st["t"], data=st["cf"].copy(), ntraj=1.0, Temperature=300.0, normalized=True)
        sf = hh.idct_cf_to_sf(cf)
        return sf.nu, sf.data, cf.data
    if op == "moment":
        return hh.calculate_m0(st["ms"], st["p"], st["Ts"], st["n"], seed=st["seed"], precision=st["prec"])
    if op == "prmu":
        nu, sf, counted, _ = hh.prmu_iteration(st["ms"], st["p"], st["T"], 40.0, st["n"], 400.0, False, st["prec"],
                                               seed=st["seed"])
        return nu, sf, counted
    if st["many"]:
        crln, ntraj, _ = hh.correlation_temperatures(st["ms"], st["p"], st["Ts"], st["n"], st["prec"], seed=st["seed"])
    else:
        crln, ntraj, _ = hawaii.correlation_iterations(st["ms"], st["p"], st["T"], st["n"], st["iters"], st["prec"],
                                                       seed=st["seed"])
    return crln, ntraj


def work(case):
    op = case["op"]
    if op == "sf":
        N = case["N"]
        return {"bytes": 8.0 * 4 * N, "flops": 5.0 * 2 * N * math.log2(2 * N)}
    if op == "moment":
        # per sample the surface and dipole (about 320) and per temperature the weight
        # and its two sums (11)
        phys = 320 if case["system"] == "co2ar" else 150
        return {"bytes": 16.0 * case["nT"], "flops": float(case["n"]) * (phys + 11 * case["nT"])}
    t = TRAJ[case["system"]]
    sets = case.get("iters", 1) * case.get("nT", 1)
    n = case["n"] * sets
    qp = {"hear": 6, "co2ar": 10, "n2ar": 10, "ch4co2": 16}[case["system"]]
    half = 0.5 if op == "prmu" else 1.0
    samples = min(t["samples"], 2 * case["N"]) * half
    flops = n * (t["rhs"] * half * t["f_rhs"] + samples * t["f_dip"])
    nbytes = 8.0 * (n * qp + sets * case["N"])
    if op == "prmu":
        flops += n * 3 * 2.5 * case["N"] * math.log2(case["N"])
        nbytes += 8.0 * n * 3 * case["N"]
    return {"bytes": nbytes, "flops": float(flops)}


# ---- values in 64 bits, without the repository's code ----
ALU = 5.29177210903e-11
HKT = 4.3597447222071e-18 / 1.380649e-23
C_DISP = (0.940835513e1, 0.165523018e3, 0.379715796e4, 0.1165179999e6, 0.466258000e7, 0.236861000e9)


def _hear_V(R, want_dV=True):
    """He-Ar potential and its derivative: exponential repulsion and damped dispersion."""
    x = 1.62747925 * R
    ex = np.exp(-x)
    V = 0.2303058634e2 * np.exp(-0.163051044e1 * R - 0.4680016e-1 * R * R)
    dV = V * (-0.163051044e1 - 2.0 * 0.4680016e-1 * R)
    term = np.ones_like(R)
    S = np.ones_like(R)
    for m in range(1, 17):
        term = term * x / m
        S = S + term
        if m >= 6 and m % 2 == 0:
            c = C_DISP[m // 2 - 3] / R ** m
            f = 1.0 - ex * S
            V = V - c * f
            dV = dV - c * (1.62747925 * ex * term - m * f / R)
    return V, dV


def _hear_dip(R):
    return np.exp(0.47293181 - 0.40100613 * R - 0.10292726 * R * R) - 148.55391 / R ** 7


def _hear_sample(seed, T, n):
    """The first n accepted He-Ar phase points of the MT19937 stream of `seed` (ten words a
    candidate: R, Phi, Theta, three Box-Muller normals, the rejection's word)."""
    key = np.empty(624, dtype=np.uint32)
    v = seed & 0xFFFFFFFF
    for i in range(624):
        key[i] = v
        v = v * 69069 & 0xFFFFFFFF
    rs = np.random.RandomState()
    rs.set_state(("MT19937", key, 624))
    s = SYSTEMS["hear"]
    mu, kT = s["mu"], T / HKT
    got = []
    while sum(len(g) for g in got) < n:
        w = rs.randint(0, 1 << 32, size=(16384, 10), dtype=np.uint32).astype(np.float64) / 4294967296.0
        R = np.cbrt(w[:, 0] * (40.0 ** 3 - s["Rmin"] ** 3) + s["Rmin"] ** 3)
        Phi, Th = w[:, 1] * 2.0 * np.pi, np.arccos(2.0 * w[:, 2] - 1.0)
        x = [np.sqrt(-2.0 * np.log(w[:, k])) * np.cos(2.0 * np.pi * w[:, k + 1]) for k in (3, 5, 7)]
        pm = math.sqrt(mu * kT)
        K = 0.5 * kT * (x[0] ** 2 + x[1] ** 2 + x[2] ** 2)
        V = _hear_V(R)[0]
        ok = (np.exp(-(V - s["pesmin"]) / kT) / 1.5 >= w[:, 9]) & (K + V >= 0.0)
        # position and momentum in Cartesian coordinates
        sT, cT, sP, cP = np.sin(Th), np.cos(Th), np.sin(Phi), np.cos(Phi)
        e = np.stack([sT * cP, sT * sP, cT], 1)
        et = np.stack([cT * cP, cT * sP, -sT], 1)
        ep = np.stack([-sP, cP, np.zeros_like(sP)], 1)
        r = R[:, None] * e
        p = pm * (x[2][:, None] * e + x[1][:, None] * et + x[0][:, None] * ep)
        got.append(np.concatenate([r, p], 1)[ok])
    return np.concatenate(got)[:n]


def _hear_corr(case, seed):
    """sum_i (fwd + bwd) / 2 ALU^3 of mu0 . mu(t_k) by extrapolated midpoint steps (Gragg,
    six substep counts, error order 12) from sample to sample."""
    mu, dt, N = SYSTEMS["hear"]["mu"], SYSTEMS["hear"]["dt"], case["N"]
    y0 = _hear_sample(_seed(seed), case["T"], case["n"])
    y = np.concatenate([y0, y0 * np.array([1, 1, 1, -1, -1, -1.0])]).T.copy()
    counts = (4, 6, 8, 10, 12, 14)

    def f(y):
        R = np.sqrt((y[:3] ** 2).sum(0))
        return np.concatenate([y[3:] / mu, -_hear_V(R)[1] / R * y[:3]])

    def dip(y):
        R = np.sqrt((y[:3] ** 2).sum(0))
        return _hear_dip(R) / R * y[:3]

    out = np.zeros(N)
    d0 = dip(y)
    out[0] = (d0 * d0).sum()
    for k in range(1, N):
        table = []
        for j, m in enumerate(counts):
            h = dt / m
            a, b = y, y + h * f(y)
            for _ in range(m - 1):
                a, b = b, a + 2.0 * h * f(b)
            row = [0.5 * (a + b + h * f(b))]
            for q in range(1, j + 1):
                row.append(row[-1] + (row[-1] - table[-1][q - 1]) / ((m / counts[j - q]) ** 2 - 1.0))
            table.append(row)
        y = table[-1][-1]
        out[k] = (d0 * dip(y)).sum()
        inside = (y[:3] ** 2).sum(0) <= 40.0 ** 2
        if not inside.all():
            y, d0 = y[:, inside], d0[:, inside]
            if not y.shape[1]:
                break
    return 0.5 * ALU ** 3 * out


def _philox(ids, block, key):
    m32 = 0xFFFFFFFF
    c = [ids & m32, ids >> 32, torch.full_like(ids, block), torch.zeros_like(ids)]
    k0, k1 = key & m32, key >> 32

    def mul(a, x):  # 32 x 32 -> (high, low) in signed 64-bit words
        lo = (x & 0xFFFF) * a
        hi = (x >> 16) * a + (lo >> 16)
        return hi >> 16, ((hi & 0xFFFF) << 16) | (lo & 0xFFFF)

    for _ in range(10):
        h0, l0 = mul(0xD2511F53, c[0])
        h1, l1 = mul(0xCD9E8D57, c[2])
        c = [h1 ^ c[1] ^ k0, l1, h0 ^ c[3] ^ k1, l0]
        k0, k1 = (k0 + 0x9E3779B9) & m32, (k1 + 0xBB67AE85) & m32
    return c


def _hear_moment(case, seed):
    """<R^2 |mu|^2 exp(-V/kT) 1[H >= 0]> over the Philox samples, scaled, and its error."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    Ts, n, key = _temperatures(case), case["n"], _seed(seed)
    sw, sw2 = np.zeros(len(Ts)), np.zeros(len(Ts))
    for lo in range(0, n, 1 << 21):
        ids = torch.arange(lo, min(n, lo + (1 << 21)), dtype=torch.int64, device=dev)
        w = [_philox(ids, b, key) for b in range(3)]

        def u(i):
            return ((w[i // 4][i % 4] >> 8).double() + 0.5) / 16777216.0

        zc = torch.cos(2.0 * math.pi * u(8))
        kappa = -torch.log(u(5)) - torch.log(u(7)) * zc * zc
        R = 4.0 + 36.0 * u(0)
        x = 1.62747925 * R
        ex = torch.exp(-x)
        V = 0.2303058634e2 * torch.exp(-0.163051044e1 * R - 0.4680016e-1 * R * R)
        term, S = torch.ones_like(R), torch.ones_like(R)
        for m in range(1, 17):
            term = term * x / m
            S = S + term
            if m >= 6 and m % 2 == 0:
                V = V - C_DISP[m // 2 - 3] / R ** m * (1.0 - ex * S)
        d = torch.exp(0.47293181 - 0.40100613 * R - 0.10292726 * R * R) - 148.55391 / R ** 7
        base = R * R * d * d
        for i, T in enumerate(Ts):
            kT = T / HKT
            g = torch.where(kappa * kT + V >= 0.0, base * torch.exp(-V / kT), torch.zeros_like(base))
            sw[i] += float(g.sum())
            sw2[i] += float((g * g).sum())
    scale = 0.00361479637 * 36.0
    mean = sw / n
    return scale * mean, scale * np.sqrt(np.maximum(sw2 / n - mean * mean, 0.0) / n)


def _sf(case, seed):
    """Connes apodization, then SF(nu_i) from the cosine sum over the half-shifted samples."""
    N, dt = case["N"], SYSTEMS["hear"]["dt"]
    cf = _cf(case, seed)
    r = np.arange(N) / N
    c = cf * (1.0 - r * r) ** 2
    k = np.arange(2 * N)
    z = np.concatenate([c, [0.0], -c[:0:-1]]) * np.exp(1j * np.pi * k / (2 * N)) / (2 * N)
    X = np.fft.ifft(z).real[:N] * 2 * N
    atu, c_cm, tmax = 2.4188843265857e-17, 2.99792458e10, N * dt
    dip_au = 8.4783536255e-30
    nu = np.arange(N) * np.pi / tmax / c_cm / atu / 2.0 / np.pi
    return nu, X * tmax / np.pi * atu * dip_au ** 2 / (4.0 * np.pi * 8.8541878128e-12), c


def exact(case, seed):
    op = case["op"]
    if op == "sf":
        return _sf(case, seed)
    if case["system"] != "hear":
        return None  # fitted surfaces: their tables are in the repository alone
    if op == "moment":
        return _hear_moment(case, seed)
    if op == "corr" and case["prec"] == "fp64" and case["n"] * case["N"] <= 100_000:
        # a longer grid or ensemble takes minutes in numpy; on the mixed path the value is
        # the FP64 path's, which the mixed one approaches to its tolerance only
        return _hear_corr(case, seed)[None, :], np.array([float(case["n"])])
    return None
