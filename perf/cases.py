"""The work that programs using turbchannel_b200 have it do, as measurable cases.

Every case goes through the Python mirror of the C ABI.  A time step is followed by the
diagnostics that the reference's driver reads after every step (bulk integral, CFL number
and plane profiles); the ring advances from pass to pass as in a run.  The kinds:

  step   one order-3 SBDF step (data::Step) of the staggered or collocated scheme and its
         diagnostics: DNS, and LES with the Smagorinsky or the learned closure
  solve  the pressure solve alone on device arrays (the Poisson microbenchmark)
  srk    one segregated IMEX Runge-Kutta step of the collocated scheme and its diagnostics
  train  one epoch of Adam on the learned closure's samples

exact() restates the steps and solves in 64 bits with plain torch.
"""
import math

import numpy as np
import torch

import turbchannel_b200 as tb
from turbchannel_b200 import imex

SCHEMES = {"hw2": tb.HW2, "vv4": tb.VV4, "coll": tb.COLLOC}


def _step(name, scheme, nx, ny, nz, precision, model="dns", stab=0, tau=0.0, re=0.0, gamma=2.0, lx=2 * math.pi, ly=math.pi):
    return {"name": name, "kind": "step", "scheme": scheme, "nx": nx, "ny": ny, "nz": nz, "precision": precision,
            "model": model, "stab": stab, "tau": tau, "re": re, "gamma": gamma, "lx": lx, "ly": ly}


def listed():
    return [
        # the smallest flow configuration: HW2 DNS at Re_b 5600, where launches and latency count
        _step("step hw2 64x64x64 f64", "hw2", 64, 64, 64, "f64", tau=0.002, re=5600.0, gamma=1.8, lx=4 * math.pi,
              ly=4 * math.pi / 3),
        # the headline DNS (Re_tau ~ 590) in the mixed form and in FP64
        _step("step vv4 384x384x256 mixed", "vv4", 384, 384, 256, "mixed", tau=0.0008, re=21900.0, gamma=2.2),
        _step("step vv4 384x384x256 f64", "vv4", 384, 384, 256, "f64", tau=0.0008, re=21900.0, gamma=2.2),
        # the collocated DNS at Re_b 13750
        _step("step coll 256x256x192 f64", "coll", 256, 256, 192, "f64", tau=0.001, re=13750.0, gamma=2.0),
        # the LES grid of the closure experiment: Smagorinsky-van Driest, and the learned closure
        _step("step les smag 96x96x64 f64", "hw2", 96, 96, 64, "f64", model="smag", tau=0.002, re=21900.0, gamma=2.2),
        _step("step les mlp 96x96x64 mixed", "hw2", 96, 96, 64, "mixed", model="mlp", tau=0.002, re=21900.0, gamma=2.2),
        # a DNS on sizes that are no powers of two and an odd number of planes
        _step("step vv4 216x108x95 mixed", "vv4", 216, 108, 95, "mixed", tau=0.001, re=11000.0, gamma=2.0),
        # the Poisson microbenchmark: a solve that fits the L2 cache, and a large one
        {"name": "solve hw2 128x128x128 f64", "kind": "solve", "scheme": "hw2", "nx": 128, "ny": 128, "nz": 128,
         "precision": "f64"},
        {"name": "solve vv4 512x512x256 mixed", "kind": "solve", "scheme": "vv4", "nx": 512, "ny": 512, "nz": 256,
         "precision": "mixed"},
        # collocated_SRK: the reference driver's own grid, and a DNS grid
        {"name": "srk 128x64x49 f64", "kind": "srk", "nx": 128, "ny": 64, "nz": 49, "precision": "f64"},
        {"name": "srk 384x384x257 mixed", "kind": "srk", "nx": 384, "ny": 384, "nz": 257, "precision": "mixed"},
        # training the closure: one snapshot's samples of the 96x64x96 LES grid at the default batch
        {"name": "train 589824 by 4096", "kind": "train", "samples": 589824, "batch": 4096},
    ]


def _lengths(lo, hi):
    """The even products of powers of 2 and 3 between lo and hi."""
    return sorted(2 ** a * 3 ** b for a in range(1, 11) for b in range(7) if lo <= 2 ** a * 3 ** b <= hi)


def draw(rng):
    def length(lo, hi):
        x = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        return min(_lengths(lo, hi), key=lambda n: abs(math.log(n / x)))

    def planes(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["step"] * 5 + ["solve"] * 2 + ["srk", "train"])
    prec = rng.choice(["f64", "mixed"])
    if kind == "train":
        return {"kind": "train", "samples": planes(30000, 589824), "batch": rng.choice([1024, 4096, 10000])}
    if kind == "solve":
        return {"kind": "solve", "scheme": rng.choice(sorted(SCHEMES)), "nx": length(32, 512), "ny": length(32, 512),
                "nz": planes(32, 256), "precision": prec}
    if kind == "srk":
        return {"kind": "srk", "nx": length(32, 256), "ny": length(32, 256), "nz": planes(32, 192), "precision": prec}
    scheme = rng.choice(["hw2", "vv4", "vv4", "coll"])
    model = rng.choice(["dns", "dns", "smag"]) if scheme != "coll" else "dns"
    c = _step("", scheme, length(32, 384), length(32, 384), planes(32, 256), prec, model=model,
              stab=rng.choice([0, 1]) if scheme == "coll" else 0, re=rng.choice([5600.0, 13750.0, 21900.0]),
              gamma=rng.choice([1.8, 2.0, 2.2]))
    del c["name"]
    return c


# ---- what a program has before the call ---------------------------------------------------


def _mesh(case):
    """Parameters and wall-normal coordinates of the case's channel, and the time step."""
    prec = tb.FP64 if case["precision"] == "f64" else tb.MIXED
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if case["kind"] == "srk":  # the channel of the reference's SRK driver, Re_tau 180
        lx, ly, visc = 4 * math.pi, 4 * math.pi / 3, 1.0 / 180.0
        zz = 1.0 + np.tanh(1.8 * (2.0 * np.arange(nz) / (nz - 1) - 1.0)) / np.tanh(1.8)
        p = dict(scheme=tb.COLLOC, visc_type=tb.VISC_CROSS, stab_type=1, fd_mode=1, NX=nx, NY=ny, NZ=nz, visc=visc,
                 sour_dpdx=1.0, inv_length_scale=180.0, xmin=0.0, ymin=0.0, hx=lx / nx, hy=ly / ny,
                 area=lx * ly * (zz[-1] - zz[0]), precision=prec, turb_model=0, device=0, low_modes=0)
        return p, zz, min(2e-3, 0.2 * float(np.min(np.diff(zz))) ** 2 / visc)
    scheme = SCHEMES[case["scheme"]]
    turb = 0 if case.get("model", "dns") == "dns" else tb.TURB_SMAGORINSKY
    p, zz = tb.channel_params(scheme, nx, ny, nz, case.get("lx", 2 * math.pi), case.get("ly", math.pi),
                              case.get("re", 13750.0), case.get("gamma", 2.0), precision=prec, turb=turb,
                              stab_type=case.get("stab", 0))
    tau = case.get("tau", 0.0)
    if not tau:  # within the convective and the wall-normal diffusion limits
        tau = min(0.002, 0.15 * min(p["hx"], p["hy"]), 0.08 * float(np.min(np.diff(zz))) ** 2 / p["visc"])
    return p, zz, tau


def _field(case, zz, seed):
    """A seeded channel field (z, y, x) in 64 bits: a flat mean profile, large eddies that vanish at the
    walls, and weak noise.  Staggered and collocated cases take the same values at their own points."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    r = np.random.RandomState(seed % (1 << 31))
    dev = dict(device="cuda", dtype=torch.float64)
    coll = case["kind"] == "srk" or case["scheme"] == "coll"
    zf = torch.tensor(zz[:nz] if coll else zz[:-1], **dev) - 1.0  # nodes, or the w faces
    zc = zf if coll else torch.tensor(0.5 * (zz[1:] + zz[:-1]), **dev) - 1.0
    x = torch.arange(nx, **dev) * (2 * math.pi / nx)
    y = torch.arange(ny, **dev) * (2 * math.pi / ny)
    out = []
    for c in range(3):
        z = (zf if c == 2 else zc).view(-1, 1, 1)
        wall = (1.0 - z ** 2).clamp(min=0.0)
        f = 0.02 * (2.0 * torch.rand((nz, ny, nx), generator=g, **dev) - 1.0) * wall
        for _ in range(5):
            kx, ky, kz = r.randint(0, 4), r.randint(1, 5), r.randint(1, 4)
            a, b, d = r.uniform(0, 2 * math.pi, 3)
            f += (0.08 * torch.cos(kx * x + a).view(1, 1, -1)) * torch.cos(ky * y + b).view(1, -1, 1) * (
                wall * torch.cos(kz * math.pi * z / 2 + d))
        if c == 0:
            f += 1.125 * (1.0 - z.abs() ** 8)
        if coll:
            f[0] = 0.0
            f[-1] = 0.0
        elif c == 2:
            f[0] = 0.0
        out.append(f)
    return out


class _Buffer:
    """A device buffer of a solver, for torch; the tensor made from it keeps the solver."""

    def __init__(self, owner, ptr, shape, f64):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": "<f8" if f64 else "<f4", "data": (ptr, False),
                                         "version": 3, "strides": None}


def _levels(S, case):
    """torch views of the solver's four ring levels (structure of arrays) and pressures."""
    f64 = case["precision"] == "f64"
    shape = (case["nz"], case["ny"], case["nx"])
    vel, prs = [], []
    for level in range(4):
        v, p = S.device_level(level)
        vel.append(torch.as_tensor(_Buffer(S, v, (3,) + shape, f64), device="cuda"))
        prs.append(torch.as_tensor(_Buffer(S, p, shape, f64), device="cuda"))
    return vel, prs


def _closure(seed):
    m = tb.Mlp(seed=int(seed) % (1 << 31))
    w = m.params
    m.close()
    return w


def prepare(case, seed):
    if case["kind"] == "train":
        return _prepare_train(case, seed)
    p, zz, tau = _mesh(case)
    S = tb.Solver(p, zz)
    st = {"case": dict(case), "S": S, "tau": tau, "t": 0.0}
    if case["kind"] == "solve":
        rhs = _rhs(case, seed).to(torch.float64 if case["precision"] == "f64" else torch.float32)
        st["rhs"], st["p"] = rhs, torch.empty_like(rhs)
        torch.cuda.synchronize()
        return st
    st["vel"], st["prs"] = _levels(S, case)
    for c, f in enumerate(_field(case, zz, seed)):
        st["vel"][0][c].copy_(f)
    torch.cuda.synchronize()
    if case["kind"] == "srk":
        S.srk_init(imex.ARS_343(), 1)
        S.srk_step(0.0, tau)
        S.sync()
        return st
    if case["model"] == "mlp":
        S.set_turb_model(tb.TURB_MLP, _closure(seed))
    S.set_forcing(1, 1.0)  # constant flow rate, bulk velocity 1
    # the first step projects the field; the BDF order is then ramped to 3
    for cur, order in ((0, 1), (1, 1), (2, 2)):
        S.Step(cur * tau, tau, cur, order)
    S.sync()
    st["cur"], st["t"] = 3, 3 * tau
    return st


def _rhs(case, seed):
    """N(0,1) right-hand side with zero mean (the solvable part of the pinned system)."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    r = torch.randn((case["nz"], case["ny"], case["nx"]), generator=g, device="cuda", dtype=torch.float64)
    return r - r.mean()


def _prepare_train(case, seed):
    """Closure samples as tc_les_samples gives them: asinh of the invariants, log(1+y+)/4, nu*/nu."""
    r = np.random.RandomState(seed % (1 << 31))
    n = case["samples"]
    x = np.arcsinh(r.standard_normal((n, 6)).astype(np.float32) * np.float32(2.0))
    x[:, 0] = np.abs(x[:, 0])
    x[:, 1] = -np.abs(x[:, 1])
    x[:, 5] = np.float32(0.25) * np.log1p(r.uniform(0.0, 590.0, n)).astype(np.float32)
    y = (0.3 * x[:, 0] * x[:, 5] + 0.2 * r.standard_normal(n)).astype(np.float32)
    m = tb.Mlp(seed=int(seed) % (1 << 31))
    m.set_data(x, y)
    return {"case": dict(case), "mlp": m}


# ---- one pass -------------------------------------------------------------------------------


def _diagnostics(st, level):
    integral, cfl, prof = st["S"].diagnostics(level, st["tau"])
    # a mixed solver's sums carry the accuracy of its 32-bit fields
    kind = np.float64 if st["case"]["precision"] == "f64" else np.float32
    return {"integral": integral.astype(kind), "cfl": np.array([cfl], dtype=kind), "profiles": prof.astype(kind)}


def _level(st, level):
    """What the program reads of the new level.  A mixed step's pressure is only defined to some 2e-4 of
    itself (the right-hand side of its Poisson problem is the divergence of a 32-bit v / tau: any other
    rounding of v moves p by that much, exact() shows it), so there the field is judged by the velocity that
    its gradient made divergence-free and by its plane statistics; the mixed solve cases return p whole."""
    if st["case"]["precision"] == "f64":
        return {"velocity": st["vel"][level], "pressure": st["prs"][level]}
    return {"velocity": st["vel"][level]}


def run(st):
    kind = st["case"]["kind"]
    if kind == "train":
        loss = st["mlp"].train(1, st["case"]["batch"], 1e-3)
        return {"loss": loss, "params": st["mlp"].params}
    S = st["S"]
    if kind == "solve":
        S.pressure_solve_device(st["rhs"].data_ptr(), st["p"].data_ptr())
        return {"p": st["p"]}
    if kind == "srk":
        S.srk_step(st["t"], st["tau"])
        st["t"] += st["tau"]
        return {**_level(st, 0), "dpdt": st["prs"][1], **_diagnostics(st, 0)}
    S.Step(st["t"], st["tau"], st["cur"], 3)
    st["t"] += st["tau"]
    st["cur"] = (st["cur"] + 1) % 4
    return {**_level(st, st["cur"]), **_diagnostics(st, st["cur"])}


def work(case):
    if case["kind"] == "train":
        n = case["samples"]  # forward and backward of 6-64-64-1, features and targets read once
        return {"bytes": 28.0 * n, "flops": 6.0 * n * (6 * 64 + 64 * 64 + 64)}
    N = float(case["nx"] * case["ny"] * case["nz"])
    w = 8 if case["precision"] == "f64" else 4
    if case["kind"] == "solve":  # read the right-hand side, write p; the FFTs and the banded sweeps
        return {"bytes": 2 * w * N, "flops": N * (5.0 * math.log2(case["nx"] * case["ny"]) + 30)}
    if case["kind"] == "srk":  # velocity, pressure and dp/dt read and written; 4 stages
        return {"bytes": 10 * w * N, "flops": 4 * N * (120 + 5.0 * math.log2(case["nx"] * case["ny"]))}
    # v_n, v_{n-1}, v_{n-2}, F_{n-1}, F_{n-2} read, F_n, v_{n+1} and p written
    words = 22 + (1 if case["stab"] else 0)
    per = {"hw2": 150, "vv4": 320, "coll": 120}[case["scheme"]]
    mlp = 2.0 * (6 * 64 + 64 * 64 + 64) if case["model"] == "mlp" else 0.0
    return {"bytes": words * w * N, "flops": N * (per + mlp + 5.0 * math.log2(case["nx"] * case["ny"]) + 30)}


# ---- the same in 64 bits with plain torch ---------------------------------------------------


def _sh(a, x=0, y=0):
    """a displaced: the value at (x + dx, y + dy), periodic."""
    if x:
        a = torch.roll(a, -x, 2)
    if y:
        a = torch.roll(a, -y, 1)
    return a


def _zs(a, k, lo=None, hi=None):
    """a at plane z + k; beyond the walls the planes given by lo / hi (lists, nearest first) or zero."""
    n = a.shape[0]
    out = torch.zeros_like(a)
    if k >= 0:
        out[: n - k] = a[k:]
        for j in range(k):  # z = n-k+j reads plane n + j
            if hi is not None:
                out[n - k + j] = hi[j]
    else:
        out[-k:] = a[:n + k]
        for j in range(-k):  # z = j reads plane j + k < 0: ghost -(j+k)
            if lo is not None:
                out[j] = lo[-(j + k) - 1]
    return out


class _Exact:
    """The SBDF and SRK steps of one channel in 64 bits (fields (z, y, x))."""

    def __init__(self, p, zz, scheme, srk=False):
        self.p, self.scheme, self.srk = p, scheme, srk
        d = dict(device="cuda", dtype=torch.float64)
        nz = p["NZ"]
        self.nx, self.ny, self.nz = p["NX"], p["NY"], nz
        self.hx, self.hy, self.nu = p["hx"], p["hy"], p["visc"]
        self.zz = zz
        dz = np.diff(zz)
        self.dzn = dz
        v = lambda a: torch.tensor(np.asarray(a, dtype=np.float64), **d).view(-1, 1, 1)  # noqa: E731
        if scheme == "coll":
            h = np.zeros(nz)
            h[0], h[-1] = 0.5 * dz[0], 0.5 * dz[-1]
            h[1:-1] = 0.5 * (dz[:-1] + dz[1:])
            self.hn, self.h, self.dz = h, v(h), v(np.append(dz, dz[-1]))
            self.dzm = v(np.append(dz[0], dz))
        else:
            self.hn, self.h = dz, v(dz)
            self.up = v(2.0 / (dz + np.append(dz[1:], 0.0)))
            self.dn = v(2.0 / (dz + np.append(0.0, dz[:-1])))
            self.hm = v(np.append(1.0, dz[:-1]))
        if scheme == "vv4":
            e = np.concatenate([dz[:1], dz, dz[-1:]])
            self.wn = (e[1:-1] + e[:-2] + e[2:]) / 3.0
            self.w = v(self.wn)
            self.g1 = v(dz / (dz - self.wn / 9.0))
            self.g2 = v(-(self.wn / 27.0) / (dz - self.wn / 9.0))
            gz = np.zeros(nz)
            for i in range(1, nz):
                gz[i] = 1.0 / (0.5 * (dz[i] + dz[i - 1]) - (dz[i] + dz[i - 1] + 0.5 * (
                    dz[i if i == nz - 1 else i + 1] + dz[0 if i == 1 else i - 2])) / 27.0)
            self.gzn, self.gz = gz, v(gz)
            T = np.zeros((nz, nz))  # the gradient's null vector
            for i in range(nz):
                T[i, i] = -1.0 if i in (0, nz - 1) else -1.0 + 1.0 / 27.0
                if i:
                    T[i, i - 1] = 1.0 / 27.0
                if i < nz - 1:
                    T[i, i + 1] = 1.0 / 27.0
            self.kergn = np.linalg.solve(T, np.ones(nz))
        self._bands()

    def _bands(self):
        """Symmetric band of each mode's wall-normal matrix: diag[z][mode], off[k][z] couples z and z + k."""
        nx, ny, nz = self.nx, self.ny, self.nz
        d = dict(device="cuda", dtype=torch.float64)
        kx = torch.arange(nx // 2 + 1, **d).view(1, -1)
        ky = torch.arange(ny, **d).view(-1, 1)
        one = torch.ones((ny, nx // 2 + 1), **d)
        dz = self.dzn
        if self.scheme == "vv4":
            gc = {-1: 1 / 27.0, 0: -1.0, 1: 1.0, 2: -1 / 27.0}
            M = np.zeros((nz, nz))
            for j in range(nz):
                for a, c1 in gc.items():
                    l = abs(j + a)
                    l = 2 * nz - l if l > nz else l
                    if l in (0, nz):
                        continue
                    for b, c2 in ((-2, 1 / 27.0), (-1, -1.0), (0, 1.0), (1, -1 / 27.0)):
                        m, c = l + b, c2
                        if m < 0:
                            m, c = -m - 1, -c
                        if m >= nz:
                            m, c = 2 * nz - m - 1, -c
                        if abs(m - j) <= 3:
                            M[j, m] += c1 * c * self.gzn[l]
            L = np.tril(M, -1)
            self.off = [None] + [np.append(np.diagonal(L, -k), np.zeros(k)) for k in (1, 2, 3)]
            base = -(L + L.T).sum(1)
            for i in (0, 1, 2, nz - 3, nz - 2, nz - 1):
                base[i] = M[i, i]
            sx, sy = torch.sin(math.pi * kx / nx), torch.sin(math.pi * ky / ny)
            s3x, s3y = 3 * sx - 4 * sx ** 3, 3 * sy - 4 * sy ** 3
            self.diag = []
            for i in range(nz):
                q = dz[i] - self.wn[i] / 9.0
                cx, cy = dz[i] * sx - self.wn[i] / 27.0 * s3x, dz[i] * sy - self.wn[i] / 27.0 * s3y
                self.diag.append(base[i] * one - 4 * cx ** 2 / (self.hx ** 2 * q) - 4 * cy ** 2 / (self.hy ** 2 * q))
        else:
            cx, cy = 1 - torch.cos(2 * math.pi * kx / nx), 1 - torch.cos(2 * math.pi * ky / ny)
            A = np.zeros(nz + 1)  # A[i] couples i - 1 and i
            if self.scheme == "hw2":
                A[1:nz] = 2.0 / (dz[:-1] + dz[1:])
                mm = 2 * (cx / self.hx ** 2 + cy / self.hy ** 2)
                self.diag = [-(A[i] + A[i + 1]) * one - dz[i] * mm for i in range(nz)]
            else:  # the horizontal part vanishes in the first and the last row, whose couplings are halved
                A[1:nz] = self.hx * self.hy / dz
                A[1] *= 0.5
                A[nz - 1] *= 0.5
                mm = cx * self.hy / self.hx + cy * self.hx / self.hy
                self.diag = []
                for i in range(nz):
                    inner = 0 < i < nz - 1
                    self.diag.append(-(A[i] + A[i + 1]) * one - ((dz[i - 1] + dz[i]) * mm if inner else 0.0 * mm))
            self.off = [None, A[1:]]
        self.diag[0][0, 0] *= 2  # the pinned mean mode

    def solve(self, rhs):
        """The pressure solve: 2-D FFT, one symmetric band per mode, inverse FFT, normalisation."""
        nz, nb = self.nz, len(self.off) - 1
        x = torch.fft.rfft2(rhs)
        y, inv, b = [None] * nz, [None] * nz, [None] * nz
        for i in range(nz):  # A = L D L^T: b[i][k] = L[i+k, i]
            dg, r = self.diag[i].clone(), x[i]
            for k in range(1, nb + 1):
                if i - k >= 0:
                    dg = dg - b[i - k][k] * b[i - k][k] / inv[i - k]
                    r = r - b[i - k][k] * y[i - k]
            inv[i], y[i] = 1.0 / dg, r
            b[i] = [None] * (nb + 1)
            for k in range(1, nb + 1):
                if i + k < nz:
                    o = torch.full_like(dg, float(self.off[k][i]))
                    for j in range(1, nb + 1 - k):  # rows i - j reach both i and i + k
                        if i - j >= 0:
                            o = o - b[i - j][j] * b[i - j][j + k] / inv[i - j]
                    b[i][k] = o * inv[i]
        for i in range(nz - 1, -1, -1):
            s = y[i] * inv[i]
            for k in range(1, nb + 1):
                if i + k < nz:
                    s = s - b[i][k] * x[i + k]
            x[i] = s
        q = torch.fft.irfft2(x, s=(self.ny, self.nx))
        mean = q.mean((1, 2)).cpu().numpy()
        if self.scheme == "vv4":
            c = (mean * self.kergn * self.dzn).sum() / (self.kergn ** 2 * self.dzn).sum() * self.kergn
            return q - torch.tensor(c, device=q.device).view(-1, 1, 1)
        if self.scheme == "hw2":
            return q - (mean * self.dzn).sum() / (self.zz[-1] - self.zz[0])
        s = (mean * self.hn).sum() * self.hx * self.hy * self.nx * self.ny / self.p["area"]
        return q - (s if self.srk else s * self.hx * self.hy)

    def div(self, v):
        U, V, W = v
        if self.scheme == "coll":
            up = _zs(W, 1)
            up[-1] = W[-1]
            dn = _zs(W, -1)
            dn[0] = W[0]
            return 0.5 * ((_sh(U, 1) - _sh(U, -1)) * self.hy * self.h + (_sh(V, 0, 1) - _sh(V, 0, -1)) * self.hx * self.h
                          + (up - dn) * self.hx * self.hy)
        if self.scheme == "hw2":
            return ((_sh(U, 1) - U) / self.hx + (_sh(V, 0, 1) - V) / self.hy) * self.h + _zs(W, 1) - W
        near = ((_sh(U, 1) - U) / self.hx + (_sh(V, 0, 1) - V) / self.hy) * self.h
        wide = ((_sh(U, 2) - _sh(U, -1)) / self.hx + (_sh(V, 0, 2) - _sh(V, 0, -1)) / self.hy) * self.w
        zero = torch.zeros_like(W[0])
        return near + _zs(W, 1) - W - (wide + _zs(W, 2, hi=[zero, W[-1]]) - _zs(W, -1, lo=[W[1]])) / 27.0

    def grad(self, q):
        if self.scheme == "coll":
            g = [0.5 * (_sh(q, 1) - _sh(q, -1)) / self.hx, 0.5 * (_sh(q, 0, 1) - _sh(q, 0, -1)) / self.hy,
                 0.5 * (_zs(q, 1) - _zs(q, -1)) / self.h]
            for a in g:
                a[0] = 0
                a[-1] = 0
            return g
        if self.scheme == "hw2":
            g = [(q - _sh(q, -1)) / self.hx, (q - _sh(q, 0, -1)) / self.hy, (q - _zs(q, -1)) * self.dn]
        else:
            g = [(self.g1 * (q - _sh(q, -1)) + self.g2 * (_sh(q, 1) - _sh(q, -2))) / self.hx,
                 (self.g1 * (q - _sh(q, 0, -1)) + self.g2 * (_sh(q, 0, 1) - _sh(q, 0, -2))) / self.hy,
                 ((q - _zs(q, -1)) - (_zs(q, 1, hi=[-q[-1]]) - _zs(q, -2, lo=[-q[0], -q[1]])) / 27.0) * self.gz]
        g[2][0] = 0
        return g

    def conv(self, v):
        return {"hw2": self._conv_hw2, "vv4": self._conv_vv4, "coll": self._conv_coll}[self.scheme](v)

    def _conv_hw2(self, v):
        U, V, W = v
        hx, hy, hz = self.hx, self.hy, self.h
        xl = (U + _sh(U, -1)) ** 2
        yl = (U + _sh(U, 0, -1)) * (V + _sh(V, -1))
        zl = (U + _zs(U, -1)) * (W + _sh(W, -1))
        zl[0] = 0
        s0 = -(_sh(xl, 1) - xl) / hx - (_sh(yl, 0, 1) - yl) / hy - (_zs(zl, 1) - zl) / hz
        xl = (V + _sh(V, -1)) * (U + _sh(U, 0, -1))
        yl = (V + _sh(V, 0, -1)) ** 2
        zl = (V + _zs(V, -1)) * (W + _sh(W, 0, -1))
        zl[0] = 0
        s1 = -(_sh(xl, 1) - xl) / hx - (_sh(yl, 0, 1) - yl) / hy - (_zs(zl, 1) - zl) / hz
        Uh, Vh = U * hz + _zs(U * hz, -1), V * hz + _zs(V * hz, -1)
        xl = (W + _sh(W, -1)) * Uh
        yl = (W + _sh(W, 0, -1)) * Vh
        zl = (W + _zs(W, -1)) ** 2
        s2 = -((_sh(xl, 1) - xl) / hx + (_sh(yl, 0, 1) - yl) / hy + (W + _zs(W, 1)) ** 2 - zl) * self.dn
        s2[0] = 0
        return [0.25 * s0, 0.25 * s1, 0.25 * s2]

    def _conv_vv4(self, v):
        U, V, W = v
        n, hx, hy, dz, dw, C = self.nz, self.hx, self.hy, self.h, self.w, 1.0 / 27.0
        zero = torch.zeros_like(U[0])
        s = []
        for q, a in ((U, 0), (V, 1)):
            e = dict(x=1, y=0) if a == 0 else dict(x=0, y=1)  # the component's own direction
            m = lambda f, k: _sh(f, k * e["x"], k * e["y"])  # noqa: E731,B023
            t = 0
            for f, ax, hh in ((U, 0, hy), (V, 1, hx)):
                d = lambda g, k: _sh(g, k if ax == 0 else 0, k if ax == 1 else 0)  # noqa: E731,B023
                if ax == a:  # own direction: faces between q and its neighbour
                    J = 9 * (d(f, -1) + f) - (d(f, -2) + d(f, 1))
                else:        # the other component interpolated along the own direction
                    J = 9 * (f + m(f, -1)) - (m(f, -2) + m(f, 1))
                t = t + hh * (dz * (d(J, 1) * (q + d(q, 1)) - J * (d(q, -1) + q))
                              - C * dw * (d(J, 2) * (q + d(q, 3)) - d(J, -1) * (d(q, -3) + q)))
            K = hx * hy * (9 * (W + m(W, -1)) - (m(W, -2) + m(W, 1)))
            r = q + _zs(q, 1)
            r[-1] = 0
            l = q + _zs(q, -1)
            l[0] = 0
            rr = q + _zs(q, 3, hi=[-q[-1], zero, q[n - 3]])
            ll = q + _zs(q, -3, lo=[-q[0], zero, q[2]])
            t = t + _zs(K, 1) * r - K * l - C * (_zs(K, 2, hi=[zero, K[-1]]) * rr - _zs(K, -1, lo=[K[1]]) * ll)
            s.append(-t / (32.0 * (dz - dw / 9.0) * hx * hy))
        t = 0
        for f, ax in ((U, 0), (V, 1)):
            d = lambda g, k: _sh(g, k if ax == 0 else 0, k if ax == 1 else 0)  # noqa: E731,B023

            def mass(E):
                return hy * (9 * (E + _zs(E, -1)) - (_zs(E, -2, lo=[-E[0], -E[1]]) + _zs(E, 1, hi=[-E[-1]])))

            M, Mw = mass(f * dz), mass(f * dw)
            t = t + d(M, 1) * (W + d(W, 1)) - M * (d(W, -1) + W) - C * (
                d(Mw, 2) * (W + d(W, 3)) - d(Mw, -1) * (d(W, -3) + W))
        lo, hi = [W[1], W[2], W[3]], [zero, W[-1], W[-2]]
        z = lambda k: _zs(W, k, lo=lo, hi=hi)  # noqa: E731
        hh = hx * hy
        bl, br = hh * (9 * (z(-1) + W) - (z(-2) + z(1))), hh * (9 * (W + z(1)) - (z(-1) + z(2)))
        bbl, bbr = hh * (9 * (z(-2) + z(-1)) - (z(-3) + W)), hh * (9 * (z(1) + z(2)) - (W + z(3)))
        r3, l3 = W + z(3), W + z(-3)
        r3[n - 2] = W[n - 2] - W[n - 1]
        l3[2] = W[2] - W[1]
        t = t + br * (W + z(1)) - bl * (z(-1) + W) - C * (bbr * r3 - bbl * l3)
        t = -t * self.gz / (32.0 * hx * hy)
        t[0] = 0
        return s + [t]

    def _conv_coll(self, v):
        s = [0, 0, 0]
        for d, h in enumerate((self.hx, self.hy, self.h)):
            m = (lambda f, k: _zs(f, k)) if d == 2 else (lambda f, k: _sh(f, k if d == 0 else 0, k if d == 1 else 0))  # noqa: B023
            for c in range(3):
                kc, jc, kd, jd = m(v[c], 1), m(v[c], -1), m(v[d], 1), m(v[d], -1)
                s[c] = s[c] - 0.25 * ((kc * kd - jc * jd) + v[d] * (kc - jc)) / h
        return s

    def visc(self, v, nut=None):
        nu, hx, hy = self.nu, self.hx, self.hy
        if nut is not None:
            return self._naive(v, nu + nut)
        s = []
        for c, q in enumerate(v):
            t = (_sh(q, 1) + _sh(q, -1) - 2 * q) / hx ** 2 + (_sh(q, 0, 1) + _sh(q, 0, -1) - 2 * q) / hy ** 2
            a, b = _zs(q, 1) - q, _zs(q, -1) - q
            if self.scheme == "coll":
                t = t + (a / self.dz + b / self.dzm) / self.h
            elif c < 2:
                t = t + (a * self.up + b * self.dn) / self.h
            else:
                t = t + (a / self.h + b / self.hm) * self.dn
            s.append(nu * t)
        return s

    def _shear(self, v, mu):
        """Twice the edge strains: xy at (x-1/2, y-1/2), xz and yz at the lower face, with wall values."""
        U, V, W = v
        xy = (U - _sh(U, 0, -1)) / self.hy + (V - _sh(V, -1)) / self.hx
        xz = (U - _zs(U, -1)) * self.dn + (W - _sh(W, -1)) / self.hx
        yz = (V - _zs(V, -1)) * self.dn + (W - _sh(W, 0, -1)) / self.hy
        return xy, xz, yz

    def _naive(self, v, mu):
        U, V, W = v
        hx, hy, hz = self.hx, self.hy, self.h
        xy, xz, yz = self._shear(v, mu)
        m4 = lambda a: a + _zs(a, -1)  # noqa: E731
        top = lambda q: -2 * q[-1] / hz[-1] * self.nu  # noqa: E731
        bot = lambda q: 2 * q[0] / hz[0] * self.nu  # noqa: E731
        sxy = 0.25 * xy * (mu + _sh(mu, -1) + _sh(mu, 0, -1) + _sh(mu, -1, -1))
        # the reference weights the right-hand xy stress of the v equation with mu(x+1, y+1)
        sxy_r = 0.25 * _sh(xy, 1) * (mu + _sh(mu, 1) + _sh(mu, 0, -1) + _sh(mu, 1, 1))
        sxz, syz = 0.25 * xz * m4(mu + _sh(mu, -1)), 0.25 * yz * m4(mu + _sh(mu, 0, -1))
        sxz[0], syz[0] = bot(U), bot(V)
        sxx, syy = 2 * (_sh(U, 1) - U) / hx * mu, 2 * (_sh(V, 0, 1) - V) / hy * mu
        szz = 2 * (_zs(W, 1) - W) / hz * mu
        s0 = (sxx - _sh(sxx, -1)) / hx + (_sh(sxy, 0, 1) - sxy) / hy + (_zs(sxz, 1, hi=[top(U)]) - sxz) / hz
        s1 = (sxy_r - sxy) / hx + (syy - _sh(syy, 0, -1)) / hy + (_zs(syz, 1, hi=[top(V)]) - syz) / hz
        s2 = (_sh(sxz, 1) - sxz) / hx + (_sh(syz, 0, 1) - syz) / hy + (szz - _zs(szz, -1)) * self.dn
        s2[0] = 0
        return [s0, s1, s2]

    def smagorinsky(self, v):
        U, V, W = v
        xy, xz, yz = self._shear(v, None)
        xz[0], yz[0] = 2 * U[0] / self.h[0], 2 * V[0] / self.h[0]
        S = ((_sh(U, 1) - U) / self.hx) ** 2 + ((_sh(V, 0, 1) - V) / self.hy) ** 2 + ((_zs(W, 1) - W) / self.h) ** 2
        up = lambda a, q: _zs(a, 1, hi=[-2 * q[-1] / self.h[-1]])  # noqa: E731
        xzu, yzu = up(xz, U), up(yz, V)
        for a, b in ((xy, _sh(xy, 0, 1)), (_sh(xy, 1), _sh(xy, 1, 1)), (xz, xzu), (_sh(xz, 1), _sh(xzu, 1)), (yz, yzu),
                     (_sh(yz, 0, 1), _sh(yzu, 0, 1))):
            S = S + 0.125 * (a * a + b * b)
        z = 0.5 * (self.zz[1:] + self.zz[:-1]) - self.zz[0]
        H = 0.5 * (self.zz[-1] - self.zz[0])
        dist = np.where(z < H, z, 2 * H - z)
        damp = 1 - np.exp(-(0.04 * dist * self.p["inv_length_scale"]) ** 3)
        ln = np.minimum(0.1 * np.cbrt(self.hx * self.hy * self.dzn), 0.41 * dist)
        return torch.tensor(damp * ln ** 2, device=U.device).view(-1, 1, 1) * torch.sqrt(2 * S)

    def explicit(self, v, nut=None):
        c, s = self.conv(v), self.visc(v, nut)
        f = [a + b for a, b in zip(c, s)]
        f[0] = f[0] + self.p["sour_dpdx"]
        for k, a in enumerate(f):
            if self.scheme == "coll":
                a[0] = 0
                a[-1] = 0
            elif k == 2:
                a[0] = 0
        return f

    def step(self, vs, fs, q, tau, order, smag):
        """vs: velocities, newest first; fs: their explicit fluxes from the second on.  The new velocity,
        pressure and the newest flux."""
        nut = self.smagorinsky(vs[0]) if smag else None
        f = self.explicit(vs[0], nut)
        a, b, d0 = {1: ([1.0], [1.0], 1.0), 2: ([2.0, -1.0], [2.0, -0.5], 1.5),
                    3: ([3.0, -3.0, 1.0], [3.0, -1.5, 1.0 / 3.0], 1.5 + 1.0 / 3.0)}[order]
        ff = [f] + fs
        r = [sum(a[j] * ff[j][c] + b[j] / tau * vs[j][c] for j in range(order)) for c in range(3)]
        st1 = self.scheme == "coll" and self.p["stab_type"] == 1
        if st1:
            r = [x - g for x, g in zip(r, self.grad(q))]
        dq = self.solve(self.div(r))
        v = [(x - g) * (tau / d0) for x, g in zip(r, self.grad(dq))]
        ub = self.bulk(v[0])
        if self.scheme == "coll":
            full = (self.zz[-1] - self.zz[0]) / self.hn[1:-1].sum()
            v[0][1:-1] += (1.0 - ub) * full
        else:
            v[0] += 1.0 - ub
        return v, (dq + q if st1 else dq), f, nut

    def bulk(self, u):
        return float((u.sum((1, 2)).cpu().numpy() * self.hn).sum()) * self.hx * self.hy / self.p["area"]

    def srk_step(self, v, q, dq, tau):
        """ARS(3,4,3) of Ascher, Ruuth and Spiteri with StabType 1 (empty implicit part)."""
        g = 0.435866521508458999416019451193556842529
        a42 = 0.5529291479
        b1, b2 = -1.5 * g * g + 4 * g - 0.25, 1.5 * g * g - 5 * g + 1.25
        x1, x2 = 1 - 4.5 * g + 1.5 * g * g, 2.75 - 10.5 * g + 3.75 * g * g
        a31 = x1 * a42 + x2 * a42 - 3.5 + 13 * g - 4.5 * g * g
        a32 = -x1 * a42 - x2 * a42 + 4 - 12.5 * g + 4.5 * g * g
        I = [[0, 0, 0, 0], [0, g, 0, 0], [0, (1 - g) / 2, g, 0], [0, b1, b2, g]]
        E = [[0, 0, 0, 0], [g, 0, 0, 0], [a31, a32, 0, 0], [1 - 2 * a42, a42, a42, 0], [0, b1, b2, g]]
        ts, alpha = tau * g, 1.0 / tau  # half the stability limit 2
        K = [[a - b for a, b in zip(self.explicit(v), self.grad(q))]]
        mu, qq = [None], [None]
        for i in range(1, 4):
            u = [v[c] + tau * sum(E[i][j] * K[j][c] for j in range(i)) for c in range(3)]
            k = self.explicit(u)
            muj = ts * dq + sum(I[i][j] / g * mu[j] for j in range(1, i))
            hat = q + sum(tau * I[i][j] * qq[j] for j in range(1, i))
            buf = muj + hat - alpha * ts * ts * dq
            w = [a - b + alpha * c for a, b, c in zip(k, self.grad(buf), v)]
            m = self.solve(self.div(w))
            pj = m + buf
            mu.append(m - alpha * ts * ts * dq)
            qq.append((pj - hat) / ts)
            K.append([a - b for a, b in zip(k, self.grad(pj))])
        return [v[c] + tau * sum(E[4][j] * K[j][c] for j in range(4)) for c in range(3)], pj, qq[3]

    def diagnostics(self, v, q, tau, nut=None):
        U, V, W = v
        coll = self.scheme == "coll"
        Wc = W if coll else 0.5 * (W + _zs(W, 1))
        zero = torch.zeros_like(U)
        n = zero if nut is None else nut
        cols = [U, V, Wc, U * U, V * V, Wc * Wc, U * V, U * Wc, V * Wc, n, q, q * q]
        prof = torch.stack([a.mean((1, 2)) for a in cols], 1).cpu().numpy()
        h = self.hn
        hw = h if coll else np.append(0.0, 0.5 * (h[1:] + h[:-1]))
        s = lambda a, w: float((a.sum((1, 2)).cpu().numpy() * w).sum()) * self.hx * self.hy  # noqa: E731
        kv = 1.0 if nut is None else 2.0
        lap = 1 / self.hx ** 2 + 1 / self.hy ** 2 + 1 / self.h ** 2
        cc = tau * (U.abs() / self.hx + V.abs() / self.hy + W.abs() / self.h) + 4 * kv * tau * (self.nu + n) * lap
        return {"integral": np.array([s(U, h), s(V, h), s(W, hw)]), "cfl": np.array([float(cc.max())]), "profiles": prof}


def exact(case, seed):
    if case["kind"] == "train" or case.get("model") == "mlp":
        return None  # BF16 activations: the network has no 64-bit result of its own
    p, zz, tau = _mesh(case)
    kind = torch.float64 if case["precision"] == "f64" else torch.float32
    if case["kind"] == "solve":
        return {"p": _Exact(p, zz, case["scheme"]).solve(_rhs(case, seed).to(kind).double())}
    v = [f.to(kind).double() for f in _field(case, zz, seed)]
    if case["kind"] == "srk":
        X = _Exact(p, zz, "coll", srk=True)
        q, dq = torch.zeros_like(v[0]), torch.zeros_like(v[0])
        for _ in range(2):
            v, q, dq = X.srk_step(v, q, dq, tau)
        level = {"velocity": torch.stack(v), "pressure": q}
        if case["precision"] != "f64":
            del level["pressure"]
        return {**level, "dpdt": dq, **X.diagnostics(v, q, tau)}
    X = _Exact(p, zz, case["scheme"])
    smag = case["model"] == "smag"
    q = torch.zeros_like(v[0])
    vs, fs = [v], []
    for order in (1, 1, 2, 3):
        w, q, f, nut = X.step(vs[:order], fs[:order - 1], q, tau, order, smag)
        vs, fs = [w] + vs[:2], [f] + fs[:2]
    level = {"velocity": torch.stack(vs[0]), "pressure": q}
    if case["precision"] != "f64":
        del level["pressure"]
    return {**level, **X.diagnostics(vs[0], q, tau, nut)}
