"""What a host code has this library do, as cases that can be timed and checked.

``listed()`` names the cases, ``draw(rng)`` gives more of the same ranges, ``prepare``
makes what a host program has in hand before the call, ``run`` makes one pass through the
public entry points, ``work`` counts what the pass cannot do without, and ``exact``
restates the outputs in 64 bits with plain torch.

Kinds of case:

* ``delta_nu``   the integrator alone (``get_delta_nu_update``), as codes that bin their
                 own power spectrum call it every PM step;
* ``step``       the whole PM step on a grid in device memory
                 (``add_nu_power_to_rhogrid``).  The grid is corrected in place, so each
                 pass first writes the field into it, as the forward FFT of a PM code does;
* ``spectrum``   the power spectrum of a grid (``total_powerspectrum``), whole or the
                 first rank's slabs;
* ``gradient``   forward and backward of the differentiable step (``NeutrinoStep``);
* ``batch``      many independent integrators advanced by one call (``KspaceBatch``), some
                 of them bound to a grid;
* ``setup``      a new integrator up to its first delta_nu, the unit of work of a
                 parameter scan or of an emulator's training set.

Grids, bins, history lengths and masses are those of the repository's workloads and tests
(N = 64 ... 1024 with N/4 ... N bins, 16 ... 512 rows, one to three mass states, hybrid
neutrinos), with ragged sizes between them.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "kspace-neutrinos_gb300"))
import kspace_gpu as kg  # noqa: E402
import workloads as W  # noqa: E402

BOX = 512.0
LIGHT_KMS = 299792.458
A0 = 0.01

# ------------------------------------------------------------------ the cases


def _delta_nu(nk, rows, m, hybrid=False, a_end=1.0):
    return dict(kind="delta_nu", nk=nk, rows=rows, m1=m[0], m2=m[1], m3=m[2], hybrid=hybrid, a_end=a_end)


def _step(N, nbins, rows, m, a_end=1.0):
    return dict(kind="step", N=N, nbins=nbins, rows=rows, m1=m[0], m2=m[1], m3=m[2], a_end=a_end)


def _spectrum(N, nbins, nslab):
    return dict(kind="spectrum", N=N, nbins=nbins, nslab=nslab)


def _gradient(N, nbins, rows, m, recompute=False, a_end=1.0):
    return dict(kind="gradient", N=N, nbins=nbins, rows=rows, m1=m[0], m2=m[1], m3=m[2], recompute=recompute,
                a_end=a_end)


def _batch(M, grids, nk_max, rows_max, pick=0):
    return dict(kind="batch", M=M, grids=grids, nk_max=nk_max, rows_max=rows_max, pick=pick)


def _setup(nk, rows, m, a_end=1.0):
    return dict(kind="setup", nk=nk, rows=rows, m1=m[0], m2=m[1], m3=m[2], a_end=a_end)


EQUAL, SPLIT, LIGHT = (0.1, 0.1, 0.1), (0.02, 0.03, 0.06), (0.05, 0.05, 0.05)


def listed():
    return [
        # a coarse spectrum and a short history early in a run: launches and latency
        dict(_delta_nu(64, 16, EQUAL), name="delta_nu nk64 rows16"),
        # the bins and history of the N=1024 workload, three mass states
        dict(_delta_nu(407, 512, SPLIT), name="delta_nu nk407 rows512 split"),
        # hybrid neutrinos after the switch to particles: the truncated J series
        dict(_delta_nu(151, 100, EQUAL, hybrid=True), name="delta_nu nk151 rows100 hybrid"),
        # the smallest PM grid a host uses (tests, debugging runs, zoom boxes)
        dict(_step(64, 32, 24, EQUAL, a_end=0.5), name="step n64"),
        # a size that is no power of two, between the small and the large grids
        dict(_step(300, 150, 100, LIGHT), name="step n300"),
        # the N=512 workload
        dict(_step(512, 256, 256, EQUAL), name="step n512"),
        # the N=1024 precision workload, three mass states
        dict(_step(1024, 512, 512, SPLIT), name="step n1024"),
        # one rank's slabs of a decomposed grid
        dict(_spectrum(768, 384, 192), name="spectrum n768 192 slabs"),
        # a whole spectrum at a snapshot, the largest grid
        dict(_spectrum(1280, 640, 1280), name="spectrum n1280"),
        # the differentiation workload
        dict(_gradient(256, 128, 128, LIGHT), name="gradient n256"),
        # a parameter scan, four of its members with a grid
        dict(_batch(256, 4, 512, 512), name="batch 256"),
        # one more member of a scan
        dict(_setup(128, 64, EQUAL), name="setup nk128 rows64"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    m = rng.choice([EQUAL, SPLIT, LIGHT])
    rows = _log_int(rng, 12, 512)
    a_end = rng.choice([0.5, 1.0])
    kind = rng.choice(["delta_nu", "delta_nu", "step", "step", "spectrum", "gradient", "batch", "setup"])
    if kind == "delta_nu":
        hybrid = rng.random() < 0.2
        if hybrid:
            m, rows, a_end = EQUAL, min(rows, 120), 1.0
        return _delta_nu(_log_int(rng, 33, 512 if not hybrid else 200), rows, m, hybrid, a_end)
    if kind == "step":
        N = 2 * _log_int(rng, 16, 512)
        return _step(N, max(16, int(N * rng.uniform(0.4, 0.8))), rows, m, a_end)
    if kind == "spectrum":
        N = 2 * _log_int(rng, 32, 640)
        return _spectrum(N, max(16, int(N * rng.uniform(0.3, 0.8))), rng.choice([N, N, max(1, N // rng.randint(2, 9))]))
    if kind == "gradient":
        N = 2 * _log_int(rng, 16, 128)
        return _gradient(N, max(16, int(N * rng.uniform(0.4, 0.8))), min(rows, 256), m, rng.random() < 0.4, a_end)
    if kind == "batch":
        return _batch(_log_int(rng, 12, 256), rng.choice([0, 0, 2]), _log_int(rng, 80, 512), _log_int(rng, 24, 512),
                      rng.randint(0, 999))
    return _setup(_log_int(rng, 32, 512), rows, m, a_end)


# ------------------------------------------------------------------ inputs


def _rng(seed, salt=0):
    return np.random.default_rng(7919 * seed + salt)


def _masses(case):
    return (case["m1"], case["m2"], case["m3"])


def _transfer(masses, seed):
    """300 log-spaced k of T_nu / T_nonu with a seeded free-streaming scale."""
    logk = np.linspace(math.log(1e-4), math.log(50.0), 300)
    kfs = 0.05 * sum(masses) / 0.1 * (1 + 0.1 * _rng(seed, 1).uniform(-1, 1))
    return logk, 1.0 / (1.0 + (np.exp(logk) / kfs) ** 2)


def _history(delta, rows, a_end, seed):
    """(log a_j, delta_tot[nk][rows]): delta of every bin grown from A0 to a_end."""
    a = np.exp(np.linspace(math.log(A0), math.log(a_end), rows))
    sf = np.log(a)
    sf[0] = math.log(A0)
    g = 1 + 0.02 * _rng(seed, 2).uniform(-1, 1)
    return sf, np.ascontiguousarray(delta[:, None] * (a[None, :] / a_end) ** g)


def _bins(nk, seed):
    """Physical k of nk bins and their delta_cdm, with the scatter of finite mode counts."""
    k = np.exp(np.linspace(math.log(0.0125), math.log(8.0), nk))
    d = np.sqrt(W.spectrum(k)) * (1 + 0.05 * (0.0125 / k) * _rng(seed, 3).standard_normal(nk))
    return k, d


def _time_max(rows):
    return A0 + (rows + 12) / 100.0


def _instance(masses, nbins, rows, seed, hybrid=False, Omega0=0.3, h=0.7):
    logk, T = _transfer(masses, seed)
    if not hybrid:
        return kg.make_instance(masses, A0, h, Omega0, nbins, _time_max(rows), logk, T,
                                UnitLength_in_cm=W.UNIT_LENGTH_MPC)
    k = kg.KspaceNeutrinos()
    k.init_omega_nu(masses, A0, h)
    k.init_hybrid_nu(700.0, LIGHT_KMS, 0.5)
    k.set_hubble(Omega0)
    k.alloc_table(nbins, A0, _time_max(rows), Omega0, W.UNIT_TIME, W.UNIT_LENGTH_MPC)
    k.set_transfer(logk, T)
    return k


def _field(N, seed, nslab=None):
    """The r2c transform of a Gaussian random density field with the workloads' P(k):
    complex64 [nslab, N, N/2+1] in device memory, F(0) = BOX^1.5."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    white = torch.randn((N, N, N), generator=gen, device="cuda", dtype=torch.float32)
    n = min(N, nslab or N)
    g = torch.fft.rfftn(white)[:n].contiguous()
    del white
    kx = torch.as_tensor(W.kval(np.arange(N), N), dtype=torch.float32, device="cuda")
    kz = torch.arange(N // 2 + 1, dtype=torch.float32, device="cuda")
    step = max(1, (1 << 27) // (N * (N // 2 + 1)))
    for i in range(0, n, step):
        j = min(n, i + step)
        k = torch.sqrt(kx[i:j, None, None] ** 2 + kx[None, :, None] ** 2 + kz[None, None, :] ** 2)
        x = (2 * math.pi / BOX / 0.02) * k.clamp_(min=1.0)
        g[i:j] *= torch.sqrt(2e4 * x / (1.0 + x ** 2.8)) / N ** 1.5
    g[0, 0, 0] = complex(BOX ** 1.5, 0.0)
    return g


def _first_time(case):
    return case["a_end"] + 0.002


def _next_time(state):
    """The next PM step's scale factor: short steps, within one row of the history."""
    state["n"] += 1
    return state["a"] + 2e-7 * (state["n"] % 20000)


class _Owner(dict):
    """A state that closes the instances it holds (the batch before its members)."""

    def __del__(self):
        for key in ("batch", "k"):
            if key in self:
                self[key].close()
        for k in self.get("insts", ()):
            k.close()


def _grid_instance(case, seed, field):
    """An instance whose history belongs to this grid, past its first call."""
    masses, N = _masses(case), case["N"]
    k = _instance(masses, case["nbins"], case["rows"], seed)
    nk, power, count, keff = k.total_powerspectrum(N, field, case["nbins"])
    kphys, delta = keff * (2 * math.pi / BOX), np.sqrt(power * BOX ** 3)
    sf, dt = _history(delta, case["rows"], case["a_end"], seed)
    k.set_nu_state(sf, dt)
    k.delta_tot_init(kphys, delta, case["a_end"] + 0.001)
    return k, sf, dt


def _batch_members(case):
    """The scan's members (a property of the case) without the seeded inputs."""
    rng = np.random.default_rng(case["pick"])
    out = []
    for i in range(case["M"]):
        out.append(dict(m=float(rng.uniform(0.03, 0.6)) / 3, Omega0=float(rng.uniform(0.25, 0.35)),
                        h=float(rng.uniform(0.6, 0.75)), rows=int(rng.integers(16, case["rows_max"] + 1)),
                        nk=int(rng.integers(64, case["nk_max"] + 1)), N=0))
    for i in range(case["grids"]):
        out[i].update(N=(64, 96, 128, 192)[i % 4], nk=48)
    return out


def _prepare_batch(case, seed):
    members = _batch_members(case)
    insts, keff, delta, nks = [], [], [], []
    a_first = np.ones(case["M"]) * 1.001
    fields = []
    for i, p in enumerate(members):
        s = seed + 131 * i
        masses = (p["m"],) * 3
        k = _instance(masses, p["nk"], p["rows"], s, Omega0=p["Omega0"], h=p["h"])
        insts.append(k)
        if p["N"]:
            f = _field(p["N"], s)
            _, power, _, ke = k.total_powerspectrum(p["N"], f, p["nk"])
            d = np.sqrt(power * BOX ** 3)
            fields.append((i, f, f.clone(), p["N"], d))
            nks.append(0)
        else:
            ke, d = _bins(p["nk"], s)
            keff.append(ke)
            delta.append(d)
            nks.append(p["nk"])
        k.set_nu_state(*_history(d, p["rows"], 1.0, s))
    torch.cuda.synchronize()
    b = kg.KspaceBatch(insts)
    for i, f, work, N, _ in fields:
        b.bind_grid(i, work, N, BOX)
    b.init(a_first, nks, np.concatenate(keff) if keff else np.zeros(0), np.concatenate(delta) if delta else np.zeros(0))
    pool = np.zeros(int(b.offsets[-1]))
    free = iter(delta)
    for i, p in enumerate(members):
        if not p["N"]:
            pool[b.offsets[i]:b.offsets[i + 1]] = next(free)
    st = _Owner(kind="batch", batch=b, insts=insts, fields=fields, a=1.002, n=0, M=case["M"],
                pool=torch.as_tensor(pool).cuda(), dnu=torch.zeros(len(pool), dtype=torch.float64, device="cuda"))
    torch.cuda.synchronize()
    return st


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return _prepare_batch(case, seed)
    if kind == "delta_nu":
        k = _instance(_masses(case), case["nk"], case["rows"], seed, case["hybrid"])
        keff, delta = _bins(case["nk"], seed)
        k.set_nu_state(*_history(delta, case["rows"], case["a_end"], seed))
        k.delta_tot_init(keff, delta, case["a_end"] + 0.001)
        return _Owner(kind=kind, k=k, keff=keff, delta=delta, a=_first_time(case), n=0)
    if kind == "setup":
        keff, delta = _bins(case["nk"], seed)
        sf, dt = _history(delta, case["rows"], case["a_end"], seed)
        return dict(kind=kind, case=case, seed=seed, keff=keff, delta=delta, sf=sf, dt=dt, a=_first_time(case), n=0)
    if kind == "spectrum":
        k = _instance(EQUAL, case["nbins"], 16, seed)
        f = _field(case["N"], seed, case["nslab"])
        torch.cuda.synchronize()
        k.total_powerspectrum(case["N"], f, case["nbins"], 0, case["nslab"])  # the size's geometry
        return _Owner(kind=kind, k=k, grid=f, N=case["N"], nbins=case["nbins"], nslab=case["nslab"])
    field = _field(case["N"], seed)
    torch.cuda.synchronize()
    k, sf, dt = _grid_instance(case, seed, field)
    if kind == "step":
        stream = torch.cuda.Stream()
        k.set_stream(stream)
        st = _Owner(kind=kind, k=k, field=field, grid=torch.empty_like(field), stream=stream, N=case["N"],
                    a=_first_time(case), n=0)
        torch.cuda.synchronize()
        return st
    from autograd import NeutrinoStep
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed + 17)
    nk = dt.shape[0]
    gbar = torch.view_as_complex(torch.randn(field.shape + (2,), generator=gen, device="cuda") * 1e-3) + field
    pbar = torch.rand(nk, generator=gen, dtype=torch.float64, device="cuda")
    step = NeutrinoStep(k, sf, _first_time(case), BOX, recompute=case["recompute"])
    st = _Owner(kind=kind, k=k, step=step, grid=field.requires_grad_(True),
                hist=torch.as_tensor(dt).cuda().requires_grad_(True),
                masses=torch.tensor(_masses(case), dtype=torch.float64, requires_grad=True), gbar=gbar, pbar=pbar)
    torch.cuda.synchronize()
    return st


# ------------------------------------------------------------------ one pass


def run(state):
    kind = state["kind"]
    if kind == "delta_nu":
        return state["k"].get_delta_nu_update(_next_time(state), state["keff"], state["delta"])
    if kind == "step":
        with torch.cuda.stream(state["stream"]):
            state["grid"].copy_(state["field"])  # the forward FFT's output of this step
        state["k"].add_nu_power_to_rhogrid(_next_time(state), BOX, state["grid"], state["N"])
        return state["grid"]
    if kind == "spectrum":
        nk, power, count, keff = state["k"].total_powerspectrum(state["N"], state["grid"], state["nbins"], 0,
                                                                state["nslab"])
        return [nk, power, count, keff]
    if kind == "gradient":
        leaves = [state["grid"], state["hist"], state["masses"]]
        out, pnu = state["step"](*leaves)
        grads = torch.autograd.grad([out, pnu], leaves, [state["gbar"], state["pbar"]])
        return [out.detach(), pnu.detach()] + list(grads)
    if kind == "batch":
        for _, f, work, _, _ in state["fields"]:
            work.copy_(f)  # the members' FFTs
        if state["fields"]:
            torch.cuda.current_stream().synchronize()  # the batch runs on a stream of its own
        a = np.full(state["M"], _next_time(state))
        state["batch"].step(a, state["pool"], state["dnu"])
        return [state["dnu"]] + [work for _, _, work, _, _ in state["fields"]]
    # setup
    case = state["case"]
    k = _instance(_masses(case), case["nk"], case["rows"], state["seed"])
    k.set_nu_state(state["sf"], state["dt"])
    dnu = k.get_delta_nu_update(_next_time(state), state["keff"], state["delta"])
    om = np.array([k.OmegaNu(a) for a in (0.01, 0.1, 0.5, 1.0)])
    k.close()
    return [dnu, om]


def work(case):
    kind = case["kind"]

    def integrals(nk, rows, nspec, series=1):
        # the rule on the interval and on six bisections of it, J, the spline and the sums
        return nspec * nk * 13 * 61 * (30.0 if series == 1 else 600.0)

    if kind in ("delta_nu", "setup"):
        ns = len(set(_masses(case)))
        return {"bytes": 8.0 * case["nk"] * (case["rows"] + 4),
                "flops": integrals(case["nk"], case["rows"], ns, 19 if case.get("hybrid") else 1)}
    if kind == "batch":
        m = _batch_members(case)
        modes = sum(p["N"] ** 2 * (p["N"] // 2 + 1) for p in m)
        return {"bytes": sum(8.0 * p["nk"] * (p["rows"] + 4) for p in m) + 16.0 * modes,
                "flops": sum(integrals(p["nk"], p["rows"], 1) for p in m) + 40.0 * modes}
    N = case["N"]
    row = N * (N // 2 + 1)
    if kind == "spectrum":
        return {"bytes": 8.0 * case["nslab"] * row, "flops": 15.0 * case["nslab"] * row}
    ns = len(set(_masses(case)))
    f = integrals(0.8 * case["nbins"], case["rows"], ns)
    if kind == "step":
        return {"bytes": 16.0 * N * row, "flops": 30.0 * N * row + f}
    # gradient: grid and its cotangent in, corrected grid and the gradient out
    return {"bytes": 32.0 * N * row, "flops": 80.0 * N * row + 3 * f}


# ------------------------------------------------------------------ 64-bit values


def _gl(n):
    return np.polynomial.legendre.leggauss(n)


class _Background:
    """Omega_nu(a) from the Fermi-Dirac integrals, H(a) and the free-streaming length."""

    def __init__(self, masses, Omega0=0.3, h=0.7, hybrid=False):
        c, hub, G = 2.99792458e10, 3.24077929e-18, 6.67408e-8
        self.masses, self.Omega0 = np.asarray(masses), Omega0
        self.kT = 8.61734e-5 * ((4 / 11.) ** (1 / 3.) * 1.00328) * 2.7255
        self.rhocrit = 3 * (hub * h) ** 2 / (8 * math.pi * G)
        self.conv = 8 * math.pi / (2 * math.pi * c * 6.582119e-16) ** 3 * (1.60217646e-12 / c ** 2)
        self.omegag = 4 * 5.670373e-5 / c ** 3 * 2.7255 ** 4 / self.rhocrit
        x, w = _gl(64)
        edges = np.array([0, .5, 1, 2, 3, 5, 8, 12, 18, 27, 40, 60.])
        t = np.concatenate([0.5 * (b - a) * x + 0.5 * (a + b) for a, b in zip(edges, edges[1:])])
        wt = np.concatenate([0.5 * (b - a) * w for a, b in zip(edges, edges[1:])])
        self.lo, self.hi = math.log(0.008), math.log(1.2)
        self.kinds = sorted(set(masses))
        self.cheb = {}
        for m in self.kinds:
            def rho(la, m=m):
                y = np.exp(la) * m / self.kT
                s = (wt * t * t / (np.exp(t) + 1))[:, None] * np.sqrt(t[:, None] ** 2 + y[None, :] ** 2)
                return self.kT ** 4 * s.sum(0) * self.conv / np.exp(la)  # rho a^3
            self.cheb[m] = np.polynomial.chebyshev.Chebyshev.interpolate(rho, 90, domain=[self.lo, self.hi])
        self.hybrid = hybrid
        self.nufrac, self.vfrac = 0.0, 700.0 / LIGHT_KMS
        if hybrid:
            qc = self.masses[0] * self.vfrac / self.kT
            q = 0.5 * qc * (x + 1)
            self.nufrac = float(np.sum(0.5 * qc * w * q * q / (np.exp(q) + 1)) / (1.5 * 1.202056903159594))
        self.nonu = Omega0 - self.om(1.0)
        self.light = c * W.UNIT_TIME / W.UNIT_LENGTH_MPC
        self.hubble0 = hub * W.UNIT_TIME
        self.prefac = 1.5 * Omega0 * self.hubble0 ** 2 / self.light

    def om_one(self, m, a):
        a = np.asarray(a, dtype=np.float64)
        return self.cheb[m](np.log(a)) / a ** 3 / self.rhocrit

    def om(self, a):
        return sum(self.om_one(m, a) for m in self.masses)

    def part(self, a):
        return self.nufrac if self.hybrid and a > 0.5 else 0.0

    def nopart(self, a):
        return self.om(a) - self.om(1.0) * self.part(a) / a ** 3

    def H(self, a):
        a = np.asarray(a, dtype=np.float64)
        return self.hubble0 * np.sqrt(self.nonu / a ** 3 + 1 - self.Omega0 + self.om(a) + self.omegag / a ** 4)

    def quad(self, knots, end):
        """Nodes, weights and fslength(x, end) of a panel rule on [log A0, end]: panels end
        at every knot and shrink towards the end."""
        span = end - knots[0]
        geo = end - span * 0.8 ** np.arange(0, 110)
        e = np.unique(np.concatenate([knots, geo, np.arange(knots[0], end, 0.05), [end]]))
        e = e[(e >= knots[0]) & (e <= end)]
        e = e[np.concatenate([[True], np.diff(e) > 1e-13])]
        x, w = _gl(10)
        h, c = 0.5 * np.diff(e), 0.5 * (e[1:] + e[:-1])
        nodes = c[:, None] + h[:, None] * x
        f = lambda la: 1.0 / (np.exp(2 * la) * self.H(np.exp(la)))  # noqa: E731
        tot = (h[:, None] * w * f(nodes)).sum(1)
        after = np.concatenate([np.cumsum(tot[::-1])[::-1][1:], [0.0]])
        hh = 0.5 * (e[1:, None] - nodes)  # from the node to its panel's end
        inner = sum(wi * f(nodes + hh * (1 + xi)) for xi, wi in zip(x, w)) * hh
        fsl = self.light * (inner + after[:, None])
        return nodes.ravel(), (h[:, None] * w).ravel(), fsl.ravel(), self.light * tot.sum()


def _t(x):
    return torch.as_tensor(x, dtype=torch.float64, device="cuda")


def _spline_matrix(x):
    """c = S''/2 of a natural spline on knots x as a matrix on its values."""
    n = len(x)
    h = np.diff(x)
    A, R = np.eye(n), np.zeros((n, n))
    for i in range(1, n - 1):
        A[i, i - 1:i + 2] = h[i - 1], 2 * (h[i - 1] + h[i]), h[i]
        R[i, i - 1:i + 2] = 3 / h[i - 1], -3 / h[i - 1] - 3 / h[i], 3 / h[i]
    return np.linalg.solve(A, R)


def _spline(x, y, q):
    """Natural cubic spline of rows y[..., n] (torch) on knots x at the points q (numpy)."""
    C = y @ _t(_spline_matrix(x)).T
    j = np.clip(np.searchsorted(x, q, side="right") - 1, 0, len(x) - 2)
    h, d = _t((x[1:] - x[:-1])[j]), _t(q - x[j])
    j = torch.as_tensor(j, device="cuda")
    y0, y1, c0, c1 = y[..., j], y[..., j + 1], C[..., j], C[..., j + 1]
    return y0 + d * ((y1 - y0) / h - h * (c1 + 2 * c0) / 3 + d * (c0 + d * (c1 - c0) / (3 * h)))


def _J(x, qc=0.0, nufrac=0.0):
    if qc <= 0:
        x2 = x * x
        return (1 + 0.0168 * x2 + 0.0407 * x2 ** 2) / (1 + 2.1734 * x2 + 1.6787 * x ** 4.1811 + 0.1467 * x2 ** 4)
    s = 0
    for n in range(1, 20):
        term = (n * n + n ** 3 * qc + n * qc * x * x - x * x) * qc * torch.sinc(qc * x / math.pi) + \
            (2 * n + n * n * qc + qc * x * x) * torch.cos(qc * x)
        s = s + (1 if n % 2 else -1) * math.exp(-n * qc) / (n * n + x * x) ** 2 * term
    return s / (1.5 * 1.202056903159594 * (1 - nufrac))


def _dnu(B, k, sf, rows, a, nu_init, mJ=None):
    """The species-weighted delta_nu of bins k at a from history rows (torch) on knots sf."""
    part = B.part(a)
    loga = math.log(a)
    total = 0
    if loga <= sf[0]:
        nodes = None
        A0a = 0.0
    else:
        nodes, w, fsl, A0a = B.quad(np.asarray(sf), loga)
        S = _spline(np.asarray(sf), rows, nodes) if len(sf) > 2 else \
            rows[:, :1] + _t(nodes - sf[0]) * ((rows[:, 1:] - rows[:, :1]) / (sf[1] - sf[0]))
        kern = _t(w * fsl / (np.exp(nodes) * B.H(np.exp(nodes))))
    dp = A0 * float(B.H(A0)) / B.light * A0
    for i, m in enumerate(B.masses):
        first = list(B.masses).index(m)
        mk = (mJ[first] if mJ is not None else _t(m)) / B.kT
        v = _J(k * A0a / mk) * nu_init * (1 + dp * A0a)
        if nodes is not None:
            qc = B.vfrac * m / B.kT if part > 0 else 0.0
            v = v + B.prefac * ((kern * S) * _J(k[:, None] * _t(fsl) / mk, qc, B.nufrac)).sum(1)
        om = float(B.om_one(m, a)) - float(B.om_one(m, 1.0)) * part / a ** 3
        total = total + v * (om / float(B.nopart(a)))
    return total


def _delta_tot(B, a, dnu, dcdm):
    o3, o1 = float(B.nopart(a)) * a ** 3, float(B.om(1.0))
    return (1 - o3 / (B.nonu + o1)) * (dcdm + dnu * o3 / (B.nonu + o1 * B.part(a)))


def _init(B, masses, seed, k, sf, rows):
    """delta_nu_init and delta_nu_last of a resumed history."""
    lk, T = _transfer(masses, seed)
    t = _spline(lk, _t(T)[None, :], np.log(k.cpu().numpy()))[0]
    o3 = float(B.nopart(A0)) * A0 ** 3
    M = B.nonu + o3
    nu_init = rows[:, 0] * M / (M - o3 + t * o3) * t.abs()
    return nu_init, _dnu(B, k, sf, rows, math.exp(sf[-1]), nu_init)


def _update(B, masses, seed, k, sf, rows, dcdm, a, mJ=None, fixed=None):
    """get_delta_nu_update's first call after the initialisation, before the clamp."""
    nu_init, nu_last = fixed if fixed is not None else _init(B, masses, seed, k, sf, rows)
    new = _delta_tot(B, a, nu_last, dcdm)
    return _dnu(B, k, np.append(sf, math.log(a)), torch.cat([rows, new[:, None]], 1), a, nu_init, mJ)


def _modes(N, nbins, i, j):
    """Of slabs i..j: bin of every mode (-1 at k = 0), its weight times W^4, and k^2."""
    kx = torch.as_tensor(W.kval(np.arange(N), N), device="cuda")
    kz = torch.arange(N // 2 + 1, device="cuda")
    k2 = (kx[i:j, None, None] ** 2 + kx[None, :, None] ** 2 + kz[None, None, :] ** 2).reshape(-1)
    n = np.arange(1, 3 * (N // 2) ** 2 + 1, dtype=np.float64)
    bpu = (nbins - 1) / math.log(math.sqrt(3) * N / 2.0)
    table = np.concatenate([[-1], np.clip(np.floor(bpu * np.log(np.sqrt(n))), 0, nbins - 1)]).astype(np.int64)
    f = np.arange(N // 2 + 1) / N
    w1 = _t(1.0 / np.sinc(f) ** 4)
    wt = torch.full((N // 2 + 1,), 2.0, dtype=torch.float64, device="cuda")
    wt[0] = wt[-1] = 1.0
    w = (w1[kx.abs()[i:j]][:, None, None] * w1[kx.abs()][None, :, None] * (w1 * wt)[None, None, :]).reshape(-1)
    return torch.as_tensor(table, device="cuda")[k2], w, k2


def _chunks(N, n):
    step = max(1, (1 << 25) // (N * (N // 2 + 1)))
    return [(i, min(n, i + step)) for i in range(0, n, step)]


def _spectrum64(g, N, nbins, nslab):
    """Per non-empty bin of the whole grid: power, sum of modes, mean |k|."""
    S = torch.zeros(nbins, dtype=torch.float64, device="cuda")
    cnt, ks = torch.zeros_like(S), torch.zeros_like(S)
    nz = N // 2 + 1
    wz = torch.full((nz,), 2.0, dtype=torch.float64, device="cuda")
    wz[0] = wz[-1] = 1.0
    for i, j in _chunks(N, N):
        b, w, k2 = _modes(N, nbins, i, j)
        one = wz.repeat((j - i) * N)
        live = b >= 0
        cnt.index_add_(0, b[live], one[live])
        ks.index_add_(0, b[live], (one * k2.double().sqrt())[live])
        if i < nslab:
            n = (min(j, nslab) - i) * N * nz
            x = torch.view_as_real(g[i:min(j, nslab)]).double().square().sum(-1).reshape(-1)
            S = S.index_add(0, b[:n].clamp(min=0), torch.where(live[:n], x * w[:n], torch.zeros_like(x)))
    m = cnt > 0
    F0 = torch.view_as_real(g[0, 0, 0]).double().square().sum()
    return S[m] / F0 / cnt[m], cnt[m], ks[m] / cnt[m]


def _corrected64(g, N, nbins, kphys, ratio, norm):
    lk = torch.log(kphys)
    out = []
    for i, j in _chunks(N, N):
        _, _, k2 = _modes(N, nbins, i, j)
        q = torch.log(k2.clamp(min=1).double().sqrt() * (2 * math.pi / BOX)).clamp(lk[0].item(), lk[-1].item())
        s = (torch.searchsorted(lk, q, right=True) - 1).clamp(0, len(lk) - 2)
        y = ratio[s] + (q - lk[s]) * ((ratio[s + 1] - ratio[s]) / (lk[s + 1] - lk[s]))
        f = torch.where(k2 > 0, 1 + norm * y, torch.ones_like(y))
        out.append(g[i:j].to(torch.complex128) * f.reshape(j - i, N, -1))
    return torch.cat(out)


def _norm(B, a):
    nop = float(B.nopart(a))
    return nop / (B.nonu / a ** 3 + float(B.om(a)) - nop)


def exact(case, seed):
    kind = case["kind"]
    if kind == "spectrum":
        p, _, ke = _spectrum64(_field(case["N"], seed, case["nslab"]), case["N"], case["nbins"], case["nslab"])
        return [None, p.cpu().numpy(), None, ke.cpu().numpy()]
    if kind == "batch":
        out = []
        grids = [None] * case["grids"]
        for i, p in enumerate(_batch_members(case)):
            s = seed + 131 * i
            masses = (p["m"],) * 3
            B = _Background(masses, p["Omega0"], p["h"])
            if p["N"]:
                f = _field(p["N"], s)
                pw, _, ke = _spectrum64(f, p["N"], p["nk"], p["N"])
                k, d = ke * (2 * math.pi / BOX), torch.sqrt(pw * BOX ** 3)
            else:
                k, d = (_t(v) for v in _bins(p["nk"], s))
            sf, dt = _history(d.cpu().numpy(), p["rows"], 1.0, s)
            a = 1.002 + 2e-7
            v = _update(B, masses, s, k, sf, _t(dt), d, a).clamp(min=0)
            out.append(v)
            if p["N"]:
                grids[i] = _corrected64(f, p["N"], p["nk"], k, v / d, _norm(B, a))
        return [torch.cat(out)] + grids
    masses = _masses(case)
    B = _Background(masses, hybrid=case.get("hybrid", False))
    a = _first_time(case) + 2e-7
    if kind in ("delta_nu", "setup"):
        keff, delta = _bins(case["nk"], seed)
        sf, dt = _history(delta, case["rows"], case["a_end"], seed)
        v = _update(B, masses, seed, _t(keff), sf, _t(dt), _t(delta), a).clamp(min=0).cpu().numpy()
        return v if kind == "delta_nu" else [v, np.array([float(B.om(x)) for x in (0.01, 0.1, 0.5, 1.0)])]
    N, nb = case["N"], case["nbins"]
    g = _field(N, seed)
    if kind == "step":
        pw, _, ke = _spectrum64(g, N, nb, N)
        k, d = ke * (2 * math.pi / BOX), torch.sqrt(pw * BOX ** 3)
        sf, dt = _history(d.cpu().numpy(), case["rows"], case["a_end"], seed)
        v = _update(B, masses, seed, k, sf, _t(dt), d, a).clamp(min=0)
        return _corrected64(g, N, nb, k, v / d, _norm(B, a))
    # gradient: the same step in 64 bits, differentiated by torch
    a = _first_time(case)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed + 17)
    gbar = torch.view_as_complex(torch.randn(g.shape + (2,), generator=gen, device="cuda") * 1e-3) + g
    g64 = g.to(torch.complex128).requires_grad_(True)
    pw, _, ke = _spectrum64(g64, N, nb, N)
    k, d = ke * (2 * math.pi / BOX), torch.sqrt(pw * BOX ** 3)
    sf, dt = _history(d.detach().cpu().numpy(), case["rows"], case["a_end"], seed)
    pbar = torch.rand(len(k), generator=gen, dtype=torch.float64, device="cuda")
    D = _t(dt).requires_grad_(True)
    mJ = _t(masses).requires_grad_(True)
    with torch.no_grad():
        fixed = _init(B, masses, seed, k, sf, D)
    v = _update(B, masses, seed, k, sf, D, d, a, mJ, fixed).clamp(min=0)
    out = _corrected64(g64, N, nb, k, v / d, _norm(B, a))
    grads = torch.autograd.grad([out, v * v], [g64, D, mJ], [gbar.to(torch.complex128), pbar])
    return [out.detach(), (v * v).detach(), grads[0], grads[1], grads[2].cpu()]
