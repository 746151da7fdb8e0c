"""Performance cases of the AFQMC engine, through its public Python binding.

A case is one pass of what a user's program does with a walker population that lives on the GPU:

  block    the body of the projection drivers (afqmclab_b200.driver): a mixed measurement, then `steps` steps with
           Gram-Schmidt and population control at their cadence, the estimator sums read back and cleared, and the
           walkers handed over in the library's transfer format (a device buffer, afqmc_pack_walkers)
  measure  a mixed measurement alone, its sums (and, for a molecule, the sums per Cholesky vector) read back
  adjoint  mixed local energy, mean log-overlap and their gradients
  batch    one step of several lattices of different size and filling, as one graph launch

Kinds: "cp" is the constrained-path Hubbard model, "pl" the phaseless molecule with real Cholesky vectors; "fp64" and
"mixed" are the two precision forms.  The Hamiltonian of a case is fixed by its sizes, the walkers and the random
stream come from the seed.  The mixed form carries its walkers and overlaps in single precision, so its outputs are
returned as single-precision numbers; the FP64 form's are returned as doubles.
"""
import functools
import math
import types

import numpy as np
import torch

from afqmclab_b200 import capi, inputs

DEV = "cuda"
# the uneven batch: lattices, fillings and couplings (as the engine's benchmark)
LATTICES = ((6, 6, 16, 4.0), (8, 8, 28, 8.0), (10, 10, 40, 4.0), (12, 12, 60, 8.0))
MGS = {"cp": 10, "pl": 10}
POP = {"cp": 40, "pl": 10}


def listed():
    return [
        # the tutorial's lattice and population: latency and launches are what it costs
        dict(name="hubbard4x4_fp64", op="block", kind="cp", prec="fp64", nx=4, ny=4, nup=7, ndn=7, U=4.0, decomp="densitySpin", W=100, steps=5),
        # an ordinary production lattice in the form that is used where the energy criterion matters
        dict(name="hubbard8x8_fp64", op="block", kind="cp", prec="fp64", nx=8, ny=8, nup=28, ndn=28, U=4.0, decomp="densitySpin", W=1024, steps=5),
        # the same lattice on the tensor cores
        dict(name="hubbard8x8_mixed", op="block", kind="cp", prec="mixed", nx=8, ny=8, nup=28, ndn=28, U=4.0, decomp="densitySpin", W=1024, steps=1),
        # odd sizes, unequal filling, a decomposition that mixes the spins and an odd population
        dict(name="hubbard5x7_hop_fp64", op="block", kind="cp", prec="fp64", nx=5, ny=7, nup=13, ndn=10, U=6.0, decomp="hopCharge", W=333, steps=5),
        # several lattices advanced together
        dict(name="uneven_batch_fp64", op="batch", kind="cp", prec="fp64", W=1024),
        # small molecule (the size at which the gradients are checked)
        dict(name="molecule64_fp64", op="block", kind="pl", prec="fp64", n=64, nup=16, ndn=16, G=320, W=512, steps=5),
        dict(name="molecule64_mixed", op="block", kind="pl", prec="mixed", n=64, nup=16, ndn=16, G=320, W=512, steps=5),
        # the benchmark's molecule, in both forms
        dict(name="molecule128_mixed", op="block", kind="pl", prec="mixed", n=128, nup=32, ndn=32, G=640, W=2048, steps=5),
        dict(name="molecule128_fp64", op="block", kind="pl", prec="fp64", n=128, nup=32, ndn=32, G=640, W=2048, steps=5),
        # open shell with ragged sizes: two spin blocks of different width
        dict(name="molecule90_open_fp64", op="block", kind="pl", prec="fp64", n=90, nup=21, ndn=14, G=277, W=300, steps=5),
        # the largest molecule, which only the FP64 form takes
        dict(name="molecule256_fp64", op="block", kind="pl", prec="fp64", n=256, nup=64, ndn=64, G=1280, W=512, steps=2),
        # gradients with respect to the Hamiltonian and the trial
        dict(name="adjoint128", op="adjoint", kind="pl", prec="fp64", n=128, nup=32, ndn=32, G=640, W=512),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(("cp", "cp", "pl", "pl", "pl", "cp_mixed", "pl_mixed", "measure", "adjoint"))
    if what.startswith("cp"):
        prec = "mixed" if what == "cp_mixed" else "fp64"
        nx, ny = rng.randint(3, 12), rng.randint(3, 12)
        sites = nx * ny
        if prec == "mixed":     # the sizes that this form takes
            nx, ny = rng.choice(((4, 4), (8, 4), (8, 8), (8, 6)))
            sites = nx * ny
        nup = rng.randint(max(1, sites // 6), max(1, min(60, (3 * sites) // 5)))
        ndn = rng.randint(max(1, sites // 6), max(1, min(60, (3 * sites) // 5)))
        decomp = "densitySpin" if prec == "mixed" else rng.choice(("densitySpin", "densitySpin", "hopSpin", "densityCharge", "hopCharge"))
        return dict(op="block", kind="cp", prec=prec, nx=nx, ny=ny, nup=nup, ndn=ndn, U=rng.choice((2.0, 4.0, 8.0)), decomp=decomp,
                    W=_log(rng, 32, 1024), steps=1 if prec == "mixed" else 5)
    if what == "pl_mixed":
        n, ns = rng.choice(((64, 16), (64, 32), (128, 16), (128, 32)))
        return dict(op="block", kind="pl", prec="mixed", n=n, nup=ns, ndn=ns, G=64 * rng.randint(2, 10), W=4 * _log(rng, 32, 512), steps=5)
    n = rng.randint(24, 160)
    nup = rng.randint(max(2, n // 8), n // 3)
    ndn = nup if rng.random() < 0.5 else rng.randint(max(1, n // 8), nup)
    op = {"pl": "block"}.get(what, what)
    case = dict(op=op, kind="pl", prec="fp64", n=n, nup=nup, ndn=ndn, G=rng.randint(2 * n, 5 * n), W=_log(rng, 48, 1024 if op == "block" else 512))
    return dict(case, steps=5) if op == "block" else case


# ----------------------------------------------------------------- inputs
@functools.lru_cache(maxsize=4)
def _hubbard(nx, ny, nup, ndn, U, decomp):
    uhf = nup <= 28 and nx * ny == 64 and decomp == "densitySpin" and U == 4.0
    m = inputs.hubbard_inputs(nx, ny, nup, ndn, 1.0, -0.2 if uhf else 0.0, U, 0.005 if uhf else 0.01, decomp, "uhf" if uhf else "free")
    m.ET = inputs.hubbard_trial_energy(m)
    return m


@functools.lru_cache(maxsize=1)
def _molecule(n, nup, ndn, G):
    """Real symmetric Cholesky vectors of unit Frobenius norm, scaled by exp(-g/60) (the spectrum of the engine's
    synthetic molecule), h1 with eigenvalues on [-5, 5], the trial from its lowest orbitals."""
    gen = torch.Generator(device=DEV).manual_seed(20240502 + 1000 * n + G)
    X = torch.randn(G, n, n, generator=gen, dtype=torch.float64, device=DEV)
    X = X + X.transpose(1, 2)
    lam = torch.exp(-torch.arange(G, dtype=torch.float64, device=DEV) / 60.0)
    X *= (lam.sqrt() / X.flatten(1).norm(dim=1))[:, None, None]
    q, _ = torch.linalg.qr(torch.randn(n, n, generator=gen, dtype=torch.float64, device=DEV))
    h1 = (q * torch.linspace(-5.0, 5.0, n, dtype=torch.float64, device=DEV)) @ q.T
    h1 = 0.5 * (h1 + h1.T)
    flat = X.permute(1, 0, 2).reshape(n, G * n)
    K = h1 - 0.5 * flat @ flat.T
    V = torch.linalg.eigh(h1)[1].cpu().numpy()
    # chol[i, j, g] in Fortran order is (g, j, i) in C order; every L_g is symmetric
    chol = X.cpu().numpy().transpose(2, 1, 0)
    m = types.SimpleNamespace(
        n=n, nup=nup, ndn=ndn, G=G, dt=0.005, t=np.asfortranarray(h1.cpu().numpy()), K=np.asfortranarray(K.cpu().numpy()), chol=chol,
        bg=np.zeros(G), phiTUp=np.asfortranarray(V[:, :nup].astype(np.complex128)), phiTDn=np.asfortranarray(V[:, :ndn].astype(np.complex128)),
        logwT=0j, logwDt=0.0, logwHalf=0.0, force_cap=1.5)
    lam, U = np.linalg.eigh(m.K)
    ex = lambda a: np.asfortranarray(((U * np.exp(-a * lam)) @ U.T).astype(np.complex128))  # noqa: E731
    m.expMinusDtK, m.expHalfDtK, m.expMinusHalfDtK = ex(m.dt), ex(-0.5 * m.dt), ex(0.5 * m.dt)
    pu, pd = (torch.from_numpy(V[:, :k] @ V[:, :k].T).to(DEV) for k in (nup, ndn))
    e = (h1 * (pu + pd)).sum() + 0.5 * ((X * (pu + pd)).sum((1, 2)) ** 2).sum()
    for p in (pu, pd):
        for g0 in range(0, G, 64):
            y = X[g0:g0 + 64] @ p
            e -= 0.5 * (y * y.transpose(1, 2)).sum()
    m.ET = float(e)
    return m


def _model(c):
    if c["kind"] == "cp":
        return _hubbard(c["nx"], c["ny"], c["nup"], c["ndn"], c["U"], c["decomp"])
    return _molecule(c["n"], c["nup"], c["ndn"], c["G"])


def _lattices(c):
    return [dict(op="block", kind="cp", prec=c["prec"], nx=x, ny=y, nup=k, ndn=k, U=u, decomp="densitySpin", W=c["W"], steps=1) for x, y, k, u in LATTICES]


def _walkers(c, m, seed):
    """The trial's orbitals, each walker with a perturbation of its own.  A Hubbard walker whose fields keep the spins
    apart and real is real and keeps its spin blocks; the others are complex and full.  (n, ncol, W), on the GPU."""
    phi = torch.from_numpy(np.ascontiguousarray(m.phiT if c["kind"] == "cp" else m.phiTUp)).to(DEV)
    n, N = phi.shape
    gen = torch.Generator(device=DEV).manual_seed(int(seed))
    x = torch.randn(c["W"], N, n, 2, generator=gen, dtype=torch.float64, device=DEV) * (0.25 / math.sqrt(2 * n))
    if c["kind"] == "cp" and c["decomp"] == "densitySpin":
        x[..., 1] = 0.0
        x[:, :c["nup"], n // 2:] = 0.0
        x[:, c["nup"]:, :n // 2] = 0.0
    return (phi.T[None] + torch.view_as_complex(x)).permute(2, 1, 0)


def _engine(c, seed):
    m = _model(c)
    prec = capi.AFQMC_MIXED if c["prec"] == "mixed" else capi.AFQMC_FP64
    make = capi.cp_engine if c["kind"] == "cp" else capi.pl_engine
    e = make(m, c["W"], 1000 + int(seed), MGS[c["kind"]], POP[c["kind"]], precision=prec)
    w = _walkers(c, m, seed).permute(2, 1, 0).contiguous().cpu().numpy().transpose(2, 1, 0)
    e.set_walkers(w, np.zeros(c["W"], np.complex128), np.ones(c["W"], np.int32))
    e.reset_measurement()
    # the last step of the first pass stabilises and controls the population
    steps = c.get("steps", 1)
    e.set_cadence(MGS[c["kind"]] - steps, POP[c["kind"]] - steps)
    if c["op"] == "block":
        e.set_graphs(True)
    e.synchronize()
    return e


def prepare(case, seed):
    cs = _lattices(case) if case["op"] == "batch" else [case]
    es = [_engine(c, seed + 7919 * k) for k, c in enumerate(cs)]
    s = types.SimpleNamespace(case=case, cases=cs, engines=es, batch=None, chol=None)
    s.idx = [np.arange(e.W, dtype=np.int32) for e in es]
    s.buf = [torch.empty(e.W, e.n * e.ncol + 1, dtype=torch.complex128, device=DEV) if case["op"] in ("block", "batch") else None for e in es]
    if case["op"] == "batch":
        s.batch = capi.Batch(es)
    if case["op"] == "adjoint":
        s.chol = torch.empty(es[0].n ** 2 * es[0].G, dtype=torch.complex128, device=DEV)
    return s


def _population(s):
    """Every walker's matrix and log-weight; the log-weight's imaginary part, an angle, as cos and sin."""
    out = []
    for c, e, i, b in zip(s.cases, s.engines, s.idx, s.buf):
        e.pack_walkers(i, b.data_ptr())
        out.append(_handed(c, b[:, :-1], b[:, -1]))
    return out


def _handed(c, wf, logw):
    if c["prec"] == "mixed":
        wf, logw = wf.to(torch.complex64), logw.to(torch.complex64)
    return {"wf": wf, "logw": logw.real, "phase": torch.stack((torch.cos(logw.imag), torch.sin(logw.imag)))}


def _sums(c, v):
    return v.astype(np.complex64) if c["prec"] == "mixed" else v


def run(s):
    c, e = s.case, s.engines[0]
    if c["op"] == "adjoint":
        r = e.adjoint(chol_out=s.chol)
        return {"E": r["E"], "logov": r["mean_logov"].real, "t": r["dE_dt"], "chol": s.chol, "phiT": list(r["dE_dconj_phiT"]), "ov": list(r["dlogov_dconj_phiT"])}
    if c["op"] == "batch":
        s.batch.step(1)
        s.batch.synchronize()
        return _population(s)
    e.add_mixed_measurement()
    if c["op"] == "block":
        e.step(c["steps"])
    sums = [e.measurement()] + (list(e.cholesky_nums()) if c["kind"] == "pl" and c["op"] == "measure" else [])
    e.reset_measurement()
    out = {"sums": [_sums(c, v) for v in sums]}
    if c["op"] == "block":
        out["walkers"] = _population(s)
    return out


# ------------------------------------------------------------------- work
def _step_work(c):
    """Real operations and bytes of one step and of one measurement of the whole population (complex products: 8
    operations, real with complex: 4).  The walkers are read and written once; the operators are read once."""
    W, size = c["W"], 8 if c["prec"] == "mixed" else 16
    if c["kind"] == "cp":
        n, N = 2 * c["nx"] * c["ny"], c["nup"] + c["ndn"]
        step = W * (16.0 * n * N * N + 8.0 * N ** 3 + 8.0 * n * n * N + 24.0 * n * N)
        meas = W * (16.0 * n * N * N + 8.0 * N ** 3 + 8.0 * n * n * N + 32.0 * n * N)
        ops = 16.0 * n * (n + N)
        return step, meas, 2.0 * size * W * n * N + ops, 1.0 * size * W * n * N + ops
    n, nu, nd, G = c["n"], c["nup"], c["ndn"], c["G"]
    blocks = [nu] if nu == nd else [k for k in (nu, nd) if k]
    N = max(nu, nd)
    ov = sum(16.0 * n * k * k + 8.0 * k ** 3 for k in blocks)
    force = sum(4.0 * G * k * n for k in blocks)
    step = W * (ov + force + 4.0 * n * n * G + 8.0 * n * n * N * 6)
    ex = sum((k * n) ** 2 * (8.0 * W + 4.0 * G) for k in blocks)
    meas = W * (ov + force + 8.0 * n * n * N) + ex
    ops = 8.0 * n * n * G + 16.0 * n * n
    return step, meas, 2.0 * size * W * n * N + ops, 1.0 * size * W * n * N + ops


def work(case):
    if case["op"] == "batch":
        w = [_step_work(c) for c in _lattices(case)]
        size = sum(c["W"] * 2 * c["nx"] * c["ny"] * (c["nup"] + c["ndn"]) for c in _lattices(case))
        return {"bytes": sum(x[2] for x in w) + 16.0 * size, "flops": sum(x[0] for x in w)}
    step, meas, bs, bm = _step_work(case)
    if case["op"] == "measure":
        return {"bytes": bm, "flops": meas}
    if case["op"] == "adjoint":
        n, G, W = case["n"], case["G"], case["W"]
        K = [k * n for k in ({case["nup"]} if case["nup"] == case["ndn"] else (case["nup"], case["ndn"]))]
        return {"bytes": 16.0 * n * n * G + bm, "flops": sum(k * k * (8.0 * W + 4.0 * G) + 12.0 * k * G * W for k in K) + 16.0 * n * n * G * case["nup"]}
    k = case["steps"]
    out = 32.0 * case["W"] * (2 * case["nx"] * case["ny"] * (case["nup"] + case["ndn"]) if case["kind"] == "cp" else case["n"] * max(case["nup"], case["ndn"]))
    return {"bytes": k * bs + bm + out, "flops": k * step + meas}


# --------------------------------------------- the same in 64 bits, in torch
def _mix(z):
    """SplitMix64's output function on int64 tensors (products wrap, shifts are made logical)."""
    z = (z ^ ((z >> 30) & (2 ** 34 - 1))) * (0xBF58476D1CE4E5B9 - 2 ** 64)
    z = (z ^ ((z >> 27) & (2 ** 37 - 1))) * (0x94D049BB133111EB - 2 ** 64)
    return z ^ ((z >> 31) & (2 ** 33 - 1))


def _uniform(seed, k):
    """Draws number k of the stream: uniform on [0, 1)."""
    s = _mix(torch.tensor(seed, dtype=torch.int64, device=k.device))
    b = _mix(s + (k + 1) * (0x9E3779B97F4A7C15 - 2 ** 64))
    return ((b >> 11) & (2 ** 53 - 1)).to(torch.float64) * 2.0 ** -53


def _z(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(DEV).to(torch.complex128)


class _Population:
    """Walkers phi (W, n, ncol), log-weights, alive flags and the position in the random stream."""

    def __init__(self, c, seed):
        self.c, self.m = c, _model(c)
        m = self.m
        self.phi = _walkers(c, m, seed).permute(2, 0, 1).contiguous()
        W = c["W"]
        self.logw = torch.zeros(W, dtype=torch.complex128, device=DEV)
        self.alive = torch.ones(W, dtype=torch.bool, device=DEV)
        self.seed, self.counter = 1000 + int(seed), 0
        self.trials = [_z(m.phiT)] if c["kind"] == "cp" else [_z(t) for t in (m.phiTUp, m.phiTDn) if t.shape[1]]
        self.E = _z(m.expMinusDtK)
        self.half = _z(m.expHalfDtK)
        self.s = -math.sqrt(m.dt)       # sqrt(-dt) = i s
        if c["kind"] == "pl":
            self.chol = torch.from_numpy(np.ascontiguousarray(m.chol.transpose(2, 0, 1))).to(DEV)    # (G, n, n)
        else:
            self.consts()

    def consts(self):
        m, c = self.m, self.c
        y = m.dt * m.U * 0.5 * (-1.0 if c["decomp"] == "densityCharge" else 1.0)
        ey = np.exp(y).astype(np.complex128)
        if c["decomp"] == "hopSpin":      # cos(g) = e^y
            g = np.where(ey.real <= 1.0, np.arccos(np.minimum(ey.real, 1.0)) + 0j, -1j * np.arccosh(np.maximum(ey.real, 1.0)))
        else:                             # cosh(g) = e^y
            g = np.where(ey.real >= 1.0, -np.arccosh(np.maximum(ey.real, 1.0)) + 0j, -1j * np.arccos(np.minimum(ey.real, 1.0)))
        self.gamma = _z(g)
        self.site = _z(np.exp(-m.dt * m.U * 0.5))     # mu = h = 0: the constant on-site factor is diagonal

    def overlap(self, phi):
        """log of the determinants (an angle up to multiples of 2 pi) and theta = phi S^-1 of every spin block."""
        logdet, thetas = 0.0, []
        for t in self.trials:
            a = phi[:, :, :t.shape[1]]
            S = t.mH @ a
            sign, ld = torch.linalg.slogdet(S)
            logdet = logdet + ld + 1j * torch.angle(sign)
            thetas.append(torch.linalg.solve(S, a, left=False))
        return self.logw + logdet, thetas

    def xbar(self, thetas):
        """sum over the blocks of tr(A_g theta), A_g = phiT^H L_g (real): (W, G)."""
        x = 0.0
        for t, th in zip(self.trials, thetas):
            A = (t.real.T @ self.chol).reshape(self.c["G"], -1)           # (G, Ns n): A_g(b, i)
            x = x + _realmul(th.transpose(1, 2).reshape(th.shape[0], -1), A.T)
        return x

    def offsets(self, surv, draws):
        k = torch.cumsum(surv.to(torch.int64), 0)
        offs = self.counter + (k - surv.to(torch.int64)) * draws
        self.counter += int(k[-1]) * draws
        return offs

    def step(self):
        m, c = self.m, self.c
        lo, thetas = self.overlap(self.phi)
        cs = torch.cos(lo.imag)
        surv = self.alive & (cs > 0)
        self.alive = surv.clone()
        lw = self.logw + torch.where(surv, torch.log(cs.clamp_min(1e-300)), 0.0) - 1j * lo.imag
        new, lw = self.step_cp(thetas[0], surv, lw) if c["kind"] == "cp" else self.step_pl(thetas, surv, lw)
        keep = surv if c["kind"] == "cp" else self.alive
        self.phi = torch.where(keep[:, None, None], self.E @ new, self.phi)
        self.logw = torch.where(surv, lw, self.logw)

    def step_cp(self, th, surv, lw):
        m, c = self.m, self.c
        L, t = m.L, self.trials[0]
        P = lambda a, b: torch.einsum("ij,wij->wi", t[a].conj(), th[:, b])  # noqa: E731
        up, dn = slice(0, L), slice(L, 2 * L)
        if c["decomp"].startswith("density"):
            a, b = P(up, up), P(dn, dn)
        else:
            a, b = P(up, dn), P(dn, up)
        g = {"densityCharge": a + b - 1, "densitySpin": a - b, "hopCharge": a + b, "hopSpin": a - b}[c["decomp"]]
        f = (self.gamma * g).real.clamp(-m.force_cap, m.force_cap)
        offs = self.offsets(surv, L)
        u = _uniform(self.seed, offs[:, None] + torch.arange(L, device=DEV))
        em, ep = torch.exp(-f), torch.exp(f)
        x = torch.where(u < em / (em + ep), -1.0, 1.0)
        lw = lw + L * math.log(0.5) - (x * f - torch.log(em + ep)).sum(1) + m.dt * m.ET
        ga = self.gamma * x
        if c["decomp"] == "densityCharge":
            lw = lw + 0.5 * m.dt * m.U.sum() - ga.sum(1)
        s = self.site
        A, B = self.phi[:, :L], self.phi[:, L:]
        if c["decomp"].startswith("density"):
            ea = torch.exp(ga)
            eb = ea if c["decomp"] == "densityCharge" else torch.exp(-ga)
            A, B = (s * ea)[:, :, None] * A, (s * eb)[:, :, None] * B
        else:
            cc, ss = (torch.cosh(ga), torch.sinh(ga)) if c["decomp"] == "hopCharge" else (torch.cos(ga), torch.sin(ga))
            sgn = 1.0 if c["decomp"] == "hopCharge" else -1.0
            cc, ss = (s * cc)[:, :, None], (s * ss)[:, :, None]
            A, B = cc * A + ss * B, sgn * ss * A + cc * B
        return torch.cat((A, B), 1), lw

    def step_pl(self, thetas, surv, lw):
        m, c = self.m, self.c
        f = 1j * self.s * self.xbar(thetas)
        f = f * torch.clamp(m.force_cap / f.abs().clamp_min(1e-300), max=1.0)
        offs = self.offsets(surv, 2 * m.G)
        k = offs[:, None] + 2 * torch.arange(m.G, device=DEV)
        u1, u2 = _uniform(self.seed, k), _uniform(self.seed, k + 1)
        x = torch.sqrt(-2.0 * torch.log(torch.where(u1 == 0, 1e-300, u1))) * torch.cos(2.0 * math.pi * u2) + f
        xf = (x * f).sum(1)
        cs = torch.cos(xf.imag)
        self.alive = surv & (cs > 0)
        lw = lw + torch.where(cs > 0, torch.log(cs.clamp_min(1e-300)), 0.0) + 0.5 * (f * f).sum(1) - xf + m.dt * m.ET
        flat = self.chol.reshape(m.G, -1)
        new = torch.empty_like(self.phi)
        for w in range(0, c["W"], 256):
            M = (1j * self.s * _realmul(x[w:w + 256], flat)).reshape(-1, m.n, m.n)
            term = total = self.phi[w:w + 256]
            for order in range(1, 31):
                term = M @ term / order
                total = total + term
                if order > 3 and float(torch.view_as_real(term).abs().max()) < 1e-15:
                    break
            new[w:w + 256] = total
        return new, torch.where(self.alive, lw, self.logw)

    def stabilize(self):
        q, r = torch.linalg.qr(self.phi)
        d = torch.diagonal(r, dim1=1, dim2=2)
        q = q * (d / d.abs())[:, None, :]
        lr = torch.log(d.abs())
        add = lr.sum(1)
        if self.c["kind"] == "pl":
            add = add + lr[:, :min(self.c["nup"], self.c["ndn"])].sum(1)
        self.phi = torch.where(self.alive[:, None, None], q, self.phi)
        self.logw = torch.where(self.alive, self.logw + add, self.logw)

    def control(self):
        lo, _ = self.overlap(self.phi)
        wt = torch.where(self.alive, torch.exp(lo).real, 0.0)
        good = wt > 0
        self.logw = torch.where(good, self.logw - lo, self.logw)
        self.alive[:] = True
        W = self.c["W"]
        u = _uniform(self.seed, self.counter + torch.arange(W, device=DEV)).cpu().numpy()
        self.counter += W
        wt = torch.where(good, wt, 0.0).cpu().numpy()
        total = np.cumsum(wt)[-1]
        P = np.cumsum(wt / total)
        at = np.minimum(np.searchsorted(P, (np.arange(W) + u) / W, side="left"), W - 1)
        count = np.bincount(at, minlength=W)
        table = np.arange(W)
        table[count == 0] = np.repeat(np.arange(W), np.maximum(count - 1, 0))[:int((count == 0).sum())]
        t = torch.from_numpy(table).to(DEV)
        self.phi, self.logw = self.phi[t], self.logw[t]

    def measure(self):
        lo, thetas = self.overlap(self.half @ self.phi)
        den = torch.where(self.alive, torch.exp(lo), 0.0)
        sums = self.energy_cp(thetas[0]) if self.c["kind"] == "cp" else self.energy_pl(thetas, den)
        out = torch.zeros(5, dtype=torch.complex128, device=DEV)
        out[0] = den.sum()
        for k, v in enumerate(sums["each"]):
            out[1 + k] = (v * den).sum()
        return [out.cpu().numpy()] + [v.cpu().numpy() for v in sums["vectors"]]

    def energy_cp(self, th):
        m, t, L = self.m, self.trials[0], self.m.L
        K = torch.einsum("ji,wij->w", t.mH @ _z(m.K), th)
        P = lambda a, b: torch.einsum("ij,wij->wi", t[a].conj(), th[:, b])  # noqa: E731
        up, dn = slice(0, L), slice(L, 2 * L)
        V = ((P(up, up) * P(dn, dn) - P(up, dn) * P(dn, up)) * _z(m.U)).sum(1)
        return {"each": [K + V, K, V], "vectors": []}

    def energy_pl(self, thetas, den):
        """(xbar^2 - ex)/2 + T; the exchange through sum_g A_g x A_g and sum_w den theta x theta."""
        m = self.m
        x = self.xbar(thetas)
        T, ext, exg = 0.0, 0.0, 0.0
        for t, th in zip(self.trials, thetas):
            T = T + torch.einsum("ai,wia->w", t.real.T.to(torch.complex128) @ _z(m.t), th)
            N, n = t.shape[1], m.n
            A = (t.real.T @ self.chol).reshape(m.G, N * n)                # A_g(a, i)
            u = th.transpose(1, 2).reshape(-1, N * n)                     # u(a, i) = theta(i, a)
            for a0 in range(0, N, max(1, 4096 // n)):                     # rows (a, i) of the pair matrices
                a1 = min(N, a0 + max(1, 4096 // n))
                C = (A[:, a0 * n:a1 * n].T @ A).reshape(a1 - a0, n, N, n)             # sum_g A_g(a,i) A_g(b,j)
                Cx = C.permute(1, 0, 2, 3)                                            # index (i, a, b, j)
                V = Cx.permute(0, 2, 1, 3).reshape(n * N, (a1 - a0) * n)              # rows (i, b), columns (a, j)
                y = _realmul(u.reshape(-1, N, n).transpose(1, 2).reshape(-1, n * N), V)
                ext = ext + (y * u[:, a0 * n:a1 * n]).sum(1)
                M = ((u * den[:, None])[:, a0 * n:a1 * n].T @ u).reshape(a1 - a0, n, N, n)   # sum_w den u(a,i) u(b,j)
                R = M.permute(1, 2, 0, 3).reshape(n * N, (a1 - a0) * n)
                y = _realmul(R.T, A.reshape(-1, N, n).transpose(1, 2).reshape(-1, n * N).T)  # ((a,j), g)
                exg = exg + (y * A[:, a0 * n:a1 * n].T).sum(0)
        e = 0.5 * ((x * x).sum(1) - ext) + T
        return {"each": [e, T], "vectors": [(x * den[:, None]).sum(0), exg]}

    def handed(self):
        wf = self.phi.transpose(1, 2).reshape(self.c["W"], -1)
        h = _handed(dict(self.c, prec="fp64"), wf, self.logw)
        return {k: v.cpu() for k, v in h.items()}


def _realmul(z, r):
    """complex @ real without making the real one complex."""
    y = torch.cat((z.real, z.imag), 0) @ r
    k = z.shape[0]
    return torch.complex(y[:k], y[k:])


def _exact_adjoint(case, seed):
    p = _Population(case, seed)
    m = p.m
    lo, thetas = p.overlap(p.phi)
    den = torch.exp(lo)
    e = p.energy_pl(thetas, den)["each"][0]
    x, c = p.xbar(thetas), den / den.sum()
    E = (c * e).sum()
    dt_ = torch.zeros(m.n, m.n, dtype=torch.complex128, device=DEV)
    dL = torch.zeros(m.G, m.n, m.n, dtype=torch.complex128, device=DEV)
    grads, ovs = [], []
    W, n, G = case["W"], m.n, m.G
    for t, th in zip(p.trials, thetas):
        N = t.shape[1]
        R = (c[:, None, None] * th).sum(0)
        dt_ += (R @ t.mH).T
        # V = t theta + sum_g L_g theta Z_g, Z_g = xbar_g - A_g theta;  Y_g = sum_w c_w theta Z_g
        V = _z(m.t) @ th
        flat = th.permute(1, 0, 2).reshape(n, W * N)
        for g in range(G):
            D = ((t.real.T @ p.chol[g]).to(torch.complex128) @ flat).reshape(N, W, N).transpose(0, 1)
            Z = -D
            Z.diagonal(dim1=1, dim2=2).add_(x[:, g, None])
            Y = th @ Z
            dL[g] += ((c[:, None, None] * Y).sum(0) @ t.mH).T
            V += (p.chol[g].to(torch.complex128) @ Y.permute(1, 0, 2).reshape(n, W * N)).reshape(n, W, N).permute(1, 0, 2)
        grad = V - th @ (t.mH @ V) + (e - E)[:, None, None] * th
        grads.append((c[:, None, None] * grad).sum(0).cpu().numpy())
        ovs.append(th.mean(0).cpu().numpy())
    return {"E": E.cpu().numpy()[()], "logov": lo.mean().real.cpu().numpy()[()], "t": dt_.cpu().numpy(),
            "chol": dL.transpose(1, 2).reshape(-1), "phiT": grads, "ov": ovs}


def exact(case, seed):
    if case["op"] == "adjoint":
        return _exact_adjoint(case, seed)
    if case["op"] == "batch":
        out = []
        for k, c in enumerate(_lattices(case)):
            p = _Population(c, seed + 7919 * k)
            p.step()
            p.stabilize()
            p.control()
            out.append(p.handed())
        return out
    p = _Population(case, seed)
    sums = p.measure()
    if case["op"] == "measure":
        return {"sums": sums}
    for _ in range(case["steps"]):
        p.step()
    p.stabilize()
    p.control()
    return {"sums": sums[:1], "walkers": [p.handed()]}
