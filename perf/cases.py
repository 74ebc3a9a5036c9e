"""The work that is timed: the calls that an AFQMC program makes of this framework.

Two kinds of program use it.  One keeps the walker loop of its own and calls the operations (the
mixed density matrix, the force bias, the Hubbard-Stratonovich potential, the propagation, the
orthogonalization, the local energy) on device tensors in the reference's layouts; the other keeps a
whole system resident (``AfqmcEngine``) and advances it step by step or block by block, in FP64 or
from int8 slices (INT8X3).  Systems follow ``safire_b200.synthetic``'s distributions: hcore with
diagonal -2 + 0.25 i and off-diagonal N(0, 0.05^2), symmetric Cholesky vectors of N(0, 1) entries
times exp(-n / decay) / sqrt(M), the lowest eigenvectors of hcore as the trial.  Walkers are the
trial plus noise, as they are some steps into a run.

Sizes run from M = 24 orbitals, 6 electrons and 96 Cholesky vectors to the benchmark's M = 400,
N = 100, Nc = 2400, with 16 to 256 walkers.
"""
import math

import numpy as np
import torch

from safire_b200 import afqmc, capi, synthetic

DEV = "cuda"
C128 = torch.complex128
F64 = torch.float64


def listed():
    return [
        # a program's overlap check on a few walkers of a small molecule: launches and latency only
        dict(name="overlap_small", kind="overlap", W=16, M=24, N=6, Nc=96, cplx=False),
        # mixed density matrix against a complex trial, sizes that divide by no tile
        dict(name="green_odd", kind="green", W=90, M=129, N=33, Nc=640, cplx=True),
        # the benchmark's system, one call each: force bias, potential, propagation, orthogonalization
        dict(name="vbias_large", kind="vbias", W=256, M=400, N=100, Nc=2400, cplx=False),
        dict(name="vhs_large", kind="vhs", W=256, M=400, N=100, Nc=2400, cplx=False),
        dict(name="propagate_odd", kind="propagate", W=100, M=131, N=37, Nc=640, cplx=False),
        dict(name="propagate_large", kind="propagate", W=256, M=400, N=100, Nc=2400, cplx=False),
        dict(name="ortho_large", kind="ortho", W=256, M=400, N=100, Nc=2400, cplx=False),
        # the local energy of a measurement
        dict(name="energy_medium", kind="energy", W=128, M=200, N=50, Nc=1200, cplx=False),
        # the walker loop on the device, FP64: a small system's blocks, replayed from a graph
        dict(name="block_small_fp64", kind="block", W=64, M=24, N=6, Nc=96, steps=20, precision="fp64", ndn=-1),
        # the FP64 drop-in on a larger system, five steps and the orthogonalization
        dict(name="steps_fp64", kind="steps", W=128, M=256, N=64, Nc=1536, steps=5, precision="fp64", ndn=-1),
        # unrestricted walkers of a mid-sized system in INT8X3, with the energy measured
        dict(name="measured_int8_uhf", kind="measured", W=128, M=160, N=44, Nc=800, steps=2, precision="int8x3",
             ndn=20),
        # the benchmark's own loop: INT8X3, five steps and the orthogonalization
        dict(name="steps_int8_large", kind="steps", W=256, M=400, N=100, Nc=2400, steps=5, precision="int8x3",
             ndn=-1),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["overlap", "green", "vbias", "vhs", "propagate", "ortho", "energy", "block", "steps",
                       "measured"])
    while True:
        M = _log_uniform(rng, 24, 400)
        N = max(4, min(100, int(M * rng.uniform(0.12, 0.35))))
        c = dict(kind=kind, W=_log_uniform(rng, 16, 256), M=M, N=N, Nc=int(M * rng.uniform(4.0, 6.0)))
        if kind in ("block", "steps", "measured"):
            c["steps"] = {"block": 10, "steps": rng.choice([1, 5]), "measured": 1}[kind]
            c["precision"] = "int8x3" if kind != "block" and rng.random() < 0.5 else "fp64"
            c["ndn"] = N // 2 - rng.randint(0, 2) if rng.random() < 0.3 else -1
        else:
            c["cplx"] = kind in ("overlap", "green", "vbias", "energy") and rng.random() < 0.4
        # half of the largest listed case's cost at most (an engine's system is also made on the host)
        if work(c)["flops"] <= (2e12 if c.get("precision") == "int8x3" else 2.5e11) and (
                "precision" not in c or c["M"] <= 256):
            return c


# ---- inputs -----------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 17)


def _rn(g, *shape):
    return torch.randn(*shape, generator=g, device=DEV, dtype=F64)


def _cn(g, *shape):
    return torch.complex(_rn(g, *shape), _rn(g, *shape))


def _dt(M):
    """The timestep of the framework's serving loop: vHS grows with M, and larger ones lose the walkers."""
    return 5e-5 * 256 / M


def _decay(c):
    return c["Nc"] / 6.0


def _trial(g, M, N, cplx):
    """PsiT (N, M): orthonormal rows."""
    A = _cn(g, M, N) if cplx else _rn(g, M, N)
    return torch.conj_physical(torch.linalg.qr(A)[0]).T.contiguous()


def _walkers(g, PsiT, W):
    N, M = PsiT.shape
    return (PsiT.conj().T.to(C128)[None] + 0.3 / math.sqrt(M) * _cn(g, W, M, N)).contiguous()


def _chol_scale(c):
    return torch.exp(-torch.arange(c["Nc"], device=DEV, dtype=F64) / _decay(c)) / math.sqrt(c["M"])


def _likn(g, c):
    """Symmetric Cholesky vectors (M, M, Nc), n fastest."""
    M, Nc = c["M"], c["Nc"]
    L = torch.empty(M, M, Nc, device=DEV, dtype=F64)
    s = _chol_scale(c)
    for n0 in range(0, Nc, 128):
        n1 = min(Nc, n0 + 128)
        A = torch.triu(_rn(g, n1 - n0, M, M))
        A = A + torch.triu(A, 1).transpose(1, 2)
        L[:, :, n0:n1] = (A * s[n0:n1, None, None]).permute(1, 2, 0)
    return L


def _lnak(g, c):
    """Lnak (Nc, N, M): the half-rotated vectors of an orthonormal trial, their entries again normal."""
    Nc, N, M = c["Nc"], c["N"], c["M"]
    L = _cn(g, Nc, N, M) * math.sqrt(0.5) if c["cplx"] else _rn(g, Nc, N, M)
    return (L * _chol_scale(c)[:, None, None]).contiguous()


def _green(g, PsiT, W):
    """Mixed density matrices (W, N, M) near the trial's own."""
    N, M = PsiT.shape
    return (PsiT.conj().to(C128)[None] + 0.3 / math.sqrt(M) * _cn(g, W, N, M)).contiguous()


class _DeviceArray:
    """A resident engine array, seen as a tensor; the tensor holds this object, and so its engine, alive."""

    def __init__(self, engine, address, shape):
        self.engine = engine
        self.__cuda_array_interface__ = dict(shape=shape, typestr="<c16", data=(int(address), False), version=3)


def _system(seed, c):
    """hcore, L and the trial of an engine: (synthetic.System on the host, L on the device)."""
    g = _gen(seed)
    M, N, ndn = c["M"], c["N"], c["ndn"]
    h = torch.triu(0.05 * _rn(g, M, M), 1)
    h = h + h.T + torch.diag(-2.0 + 0.25 * torch.arange(M, device=DEV, dtype=F64))
    h = h.cpu().numpy()
    psi = np.linalg.eigh(h)[1]
    rows = [psi[:, :N].T] if ndn < 0 else [psi[:, :N - ndn].T, psi[:, :ndn].T]
    PsiT = np.ascontiguousarray(np.concatenate(rows)).astype(np.complex128)
    L = _likn(g, c)
    spec = synthetic.SystemSpec(M=M, N=N, Nc=c["Nc"], decay=_decay(c), seed=seed)
    walkers = _walkers(g, torch.from_numpy(PsiT).to(DEV), c["W"])
    uni = torch.rand(c["steps"], c["W"], c["Nc"], generator=g, device=DEV, dtype=F64).clamp_(1e-12, 1 - 1e-12)
    return spec, h, L, PsiT, walkers, uni


def prepare(case, seed):
    c = dict(case)
    k = c["kind"]
    if k in ("block", "steps", "measured"):
        spec, h, L, PsiT, walkers, uni = _system(seed, c)
        s = synthetic.System(spec=spec, hcore=h, Likn=L.cpu().numpy(), PsiT=PsiT, nel_dn=c["ndn"])
        del L
        e = afqmc.AfqmcEngine(s, c["W"], dt=_dt(c["M"]), seed=int(seed) & 0xFFFFFFFF,
                              precision=capi.PRECISION_INT8X3 if c["precision"] == "int8x3" else capi.PRECISION_FP64)
        e.set_walkers(walkers.cpu().numpy())
        info = e.info()
        return dict(kind=k, engine=e, Eshift=e.init(), step=0, steps=c["steps"], uniforms=uni,
                    SM=torch.as_tensor(_DeviceArray(e, info.SM, (c["W"], c["M"], c["N"])), device=DEV),
                    props=torch.as_tensor(_DeviceArray(e, info.props, (len(capi.PROPS), c["W"])), device=DEV))
    g = _gen(seed)
    W, M, N, Nc = c["W"], c["M"], c["N"], c["Nc"]
    if k in ("overlap", "green", "ortho"):
        PsiT = _trial(g, M, N, c["cplx"])
        SM = _walkers(g, PsiT, W)
        return dict(kind=k, PsiT=PsiT, SM0=SM, SM=torch.empty_like(SM) if k == "ortho" else SM)
    if k == "vbias":
        return dict(kind=k, G=_green(g, _trial(g, M, N, c["cplx"]), W), Lnak=_lnak(g, c), dt=_dt(M))
    if k == "vhs":
        return dict(kind=k, L=_likn(g, c), X=torch.complex(_rn(g, W, Nc), 0.3 * _rn(g, W, Nc)), dt=_dt(M))
    if k == "propagate":
        PsiT = _trial(g, M, N, False)
        SM = _walkers(g, PsiT, W)
        A = torch.complex(_rn(g, W, M, M), 0.2 * _rn(g, W, M, M)) * (0.25 / math.sqrt(M))
        V = (A + A.transpose(1, 2)).contiguous()
        A = torch.triu(1e-4 * _rn(g, M, M), 1)
        P1 = A + A.T + torch.diag(torch.exp(-0.5 * _dt(M) * (-2 + 0.25 * torch.arange(M, device=DEV, dtype=F64))))
        return dict(kind=k, SM0=SM, SM=torch.empty_like(SM), V=V, P1=P1.contiguous())
    if k == "energy":
        PsiT = _trial(g, M, N, c["cplx"])
        h = _rn(g, M, M) * 0.05
        h = h + h.T + torch.diag(-2.0 + 0.25 * torch.arange(M, device=DEV, dtype=F64))
        return dict(kind=k, G=_green(g, PsiT, W), haj=(PsiT.to(C128) @ h.to(C128)).contiguous(), Lnak=_lnak(g, c))
    raise ValueError(k)


# ---- one pass -----------------------------------------------------------------------------------
def run(s):
    k = s["kind"]
    if k == "overlap":
        return afqmc.Log_Overlap(s["PsiT"], s["SM"])
    if k == "green":
        return afqmc.MixedDensityMatrix(s["PsiT"], s["SM"])
    if k == "vbias":
        return afqmc.vbias(s["G"], s["Lnak"], s["dt"])
    if k == "vhs":
        return afqmc.vHS(s["L"], s["X"], s["dt"])
    if k == "propagate":  # in place: a step's walkers are new ones every time
        s["SM"].copy_(s["SM0"])
        return afqmc.Propagate(s["SM"], s["P1"], s["V"])
    if k == "ortho":
        s["SM"].copy_(s["SM0"])
        return afqmc.orthogonalize(s["SM"])
    if k == "energy":
        return afqmc.energy(s["G"], s["haj"], s["Lnak"])
    e, n = s["engine"], s["steps"]
    out = {}
    if k == "block":  # the loop between two returns to the host, with everything a run's block has in it
        s["Eshift"], meas = e.run_block(n, s["Eshift"], ortho_interval=5, pop_interval=10, equilibration_steps=0,
                                        measure_interval=10, relax=0.1, step0=s["step"], steer=True)
        out["meas"] = meas
    else:  # run_afqmc's loop with the program's own field stream; Eshift steered once per pass
        for i in range(n):
            e.propagate(s["Eshift"], s["step"] + i, uniforms=s["uniforms"][i])
        e.orthogonalize()
        if k == "measured":
            m = e.measure()
            out["meas"] = np.array([m[q] for q in ("Energy", "OnebodyEnergy", "ExchangeEnergy", "CoulombEnergy",
                                                   "TotalWeight")])
        s["Eshift"] = e.averages()[0]
    s["step"] += n
    p = s["props"]
    out.update(Eshift=s["Eshift"], SM=s["SM"], weight=p[0], phase=p[1], pseudo_eloc=p[2], overlap=p[6])
    return out


# ---- what one pass cannot do without ----------------------------------------------------------
def work(case):
    c = dict(case)
    k, W, M, N, Nc = c["kind"], c["W"], c["M"], c["N"], c["Nc"]
    le = 16 if c.get("cplx") else 8            # bytes of a trial / Lnak element
    lf = 8 if c.get("cplx") else 4             # flops of an element of it times a complex one, added up
    SM = 16 * W * M * N
    lu = 8.0 / 3.0 * N ** 3
    if k == "overlap":
        return dict(bytes=SM + le * M * N + 16 * W, flops=W * (lf * N * N * M + lu))
    if k == "green":
        return dict(bytes=2 * SM + le * M * N + 16 * W, flops=W * (lf * N * N * M + 8 * N ** 3 + 8 * N * N * M))
    if k == "vbias":
        return dict(bytes=SM + le * Nc * N * M + 16 * W * Nc, flops=lf * W * N * M * Nc)
    if k == "vhs":
        return dict(bytes=8 * M * M * Nc + 16 * W * Nc + 16 * W * M * M, flops=4 * W * M * M * Nc)
    if k == "propagate":
        return dict(bytes=2 * SM + 16 * W * M * M + 8 * M * M, flops=W * (8 + 48) * M * M * N)
    if k == "ortho":
        return dict(bytes=2 * SM, flops=W * (4 * N * N * M + 4 * N * N * M + 8.0 / 3.0 * N ** 3))
    if k == "energy":
        return dict(bytes=SM + le * Nc * N * M + 16 * N * M + 48 * W, flops=W * (lf * N * N * M * Nc + 8 * N * N * Nc))
    # engine steps: Green's function, force bias, vHS on the symmetric half, P1 and six Taylor terms, overlap
    step = (8 * N * N * M + 4 * N * M * Nc + 2 * M * (M + 1) * Nc + (8 + 48) * M * M * N + 4 * N * N * M + 8 * N ** 3)
    by = 8 * (M * (M + 1) // 2) * Nc + 8 * Nc * N * M + 2 * SM  # L and Lnak as FP64, the walkers in and out
    n = c["steps"]
    north = {"block": n // 5, "steps": 1, "measured": 1}[k]
    nmeas = {"block": n // 10, "steps": 0, "measured": 1}[k]
    npair = N * N if c["ndn"] < 0 else (N - c["ndn"]) ** 2 + c["ndn"] ** 2
    fl = W * (n * step + north * (8 * N * N * M + 8.0 / 3.0 * N ** 3) +
              nmeas * (4 * npair * M * Nc + 8 * npair * Nc + 8 * N * N * M))
    return dict(bytes=n * by + north * 2 * SM + nmeas * 8 * Nc * N * M, flops=fl)


def tolerance(case):
    """About four times what one pass differs by from exact() over the drawn sizes."""
    k = case["kind"]
    if k in ("steps", "measured", "block"):
        if case["precision"] == "int8x3":
            # 24-bit slices: 1e-6 in the walkers, more in the pseudo energy, which divides the
            # overlaps' difference by dt
            return {"rel": 1.5e-4, "max": 3e-3}
        # FP64: the rounding of one step grows through those that follow
        return {"rel": 1e-10, "max": 1e-9} if k == "block" else {"rel": 4e-12, "max": 1e-10}
    return {"rel": 1e-13, "max": 4e-12}


# ---- the same in 64 bits, plainly ---------------------------------------------------------------
def _fold(x):
    return x - 2 * math.pi * torch.round(x / (2 * math.pi))


def _logdet(T):
    sign, la = torch.linalg.slogdet(T)
    return torch.complex(la, torch.angle(sign))


def _qr(SM):
    Q, R = torch.linalg.qr(SM)
    d = torch.diagonal(R, dim1=1, dim2=2).real
    return Q * torch.where(d < 0, -1.0, 1.0).to(C128)[:, None, :]


def _propagate(SM, P1, V, order=6):
    S = P1.to(C128) @ SM
    T = S
    S = S.clone()
    for n in range(1, order + 1):
        T = (V @ T) * (1j / n)
        S += T
    return P1.to(C128) @ S


def _energy(G, haj, Lnak, scl, blocks):
    """(W, 3): one-body, exchange and Coulomb; `blocks`: the row ranges of the spins."""
    W, Nc = G.shape[0], Lnak.shape[0]
    E = torch.zeros(W, 3, device=DEV, dtype=C128)
    E[:, 0] = scl * torch.einsum("waj,aj->w", G, haj)
    K = torch.zeros(W, Nc, device=DEV, dtype=C128)
    for a, b in blocks:
        n, M = b - a, G.shape[2]
        step = max(1, int(1e8 // max(1, W * n * n)))
        for n0 in range(0, Nc, step):
            L = Lnak[n0:n0 + step, a:b].to(C128)
            T = (G[:, a:b].reshape(W * n, M) @ L.reshape(-1, M).T).reshape(W, n, -1, n)  # T[w, b, n, a]
            E[:, 1] += -0.5 * scl * (T * T.permute(0, 3, 2, 1)).sum((1, 2, 3))
            K[:, n0:n0 + step] += torch.diagonal(T, dim1=1, dim2=3).sum(2)
    E[:, 2] = 0.5 * scl * scl * (K * K).sum(1)
    return E


_PA = (-3.969683028665376e+01, 2.209460984245205e+02, -2.759285104469687e+02, 1.383577518672690e+02,
       -3.066479806614716e+01, 2.506628277459239e+00)
_PB = (-5.447609879822406e+01, 1.615858368580409e+02, -1.556989798598866e+02, 6.680131188771972e+01,
       -1.328068155288572e+01, 1.0)
_PC = (-7.784894002430293e-03, -3.223964580411365e-01, -2.400758277161838e+00, -2.549732539343734e+00,
       4.374664141464968e+00, 2.938163982698783e+00)
_PD = (7.784695709041462e-03, 3.224671290700398e-01, 2.445134137142996e+00, 3.754408661907416e+00, 1.0)


def _probit(p):
    """Acklam's rational approximation of the inverse normal distribution, which the method's fields use."""
    def poly(cs, x):
        v = torch.zeros_like(x)
        for q in cs:
            v = v * x + q
        return v
    q = p - 0.5
    r = q * q
    out = poly(_PA, r) * q / poly(_PB, r)
    for lo, tail, sgn in ((True, p, 1.0), (False, 1 - p, -1.0)):
        t = torch.sqrt(-2 * torch.log(tail.clamp(max=0.5)))
        m = p < 0.02425 if lo else p > 0.97575
        out = torch.where(m, sgn * poly(_PC, t) / poly(_PD, t), out)
    return out


def _exact_steps(c, seed):
    spec, h, L, PsiT, SM, uni = _system(seed, c)
    h, PsiT = torch.from_numpy(h).to(DEV), torch.from_numpy(PsiT).to(DEV)
    W, M, N, Nc, ndn = c["W"], c["M"], c["N"], c["Nc"], c["ndn"]
    dt, closed = _dt(M), c["ndn"] < 0
    blocks = [(0, N)] if closed else [(0, N - ndn)] + ([(N - ndn, N)] if ndn else [])
    scl = 2.0 if closed else 1.0
    Psi_r = PsiT.real.contiguous()  # the lowest eigenvectors: real
    Lnak = (Psi_r @ L.reshape(M, M * Nc)).reshape(N * M, Nc).T.reshape(Nc, N, M).contiguous()
    haj = PsiT @ h.to(C128)
    v0 = -0.5 * (L.reshape(M, M * Nc) @ L.reshape(M, M * Nc).T)

    def green(S):
        G, ov = torch.empty(S.shape[0], N, M, device=DEV, dtype=C128), 0
        for a, b in blocks:
            T = PsiT[a:b] @ S[:, :, a:b]
            G[:, a:b] = torch.linalg.solve(T.transpose(1, 2), S[:, :, a:b].transpose(1, 2))
            ov = ov + _logdet(T)
        return G, (2.0 if closed else 1.0) * ov

    def times_real(A, B):  # complex A against a real matrix
        return torch.complex(A.real @ B, A.imag @ B)

    def vbias(G):
        return scl * math.sqrt(dt) * times_real(G.reshape(G.shape[0], N * M), Lnak.reshape(Nc, N * M).T)

    def vhs(X):
        return math.sqrt(dt) * times_real(X, L.reshape(M * M, Nc).T).reshape(-1, M, M)

    vmf = vbias(green(PsiT.conj().T[None].contiguous())[0])[0].real
    H1 = dt * h + dt * v0 + vhs(vmf.to(C128)[None])[0].real
    w, U = torch.linalg.eigh(-0.25 * (H1 + H1.T))
    P1 = (U * torch.exp(w)) @ U.T
    P1 = torch.where(P1.abs() < 1e-8, torch.zeros_like(P1), P1)

    G, ov = green(SM)
    E = _energy(G, haj, Lnak, scl, blocks).sum(1)
    Eshift = E.mean().real
    eloc = E.clone()
    weight = torch.ones(W, device=DEV, dtype=C128)
    phase = weight.clone()
    vm = vmf.clamp(-50, 50)
    for i in range(c["steps"]):
        vb = vbias(green(SM)[0])
        a = vb.abs()
        vd = 1j * (torch.where(a > 50, vb / a * 50, vb) - vm)
        X = _probit(uni[i]) + vd
        hw = (-vd * (X - 0.5 * vd)).sum(1)
        mf = -0.5 * (vmf @ vmf) + 1j * (X @ vmf.to(C128))
        SM = _propagate(SM, P1, vhs(X))
        new = green(SM)[1]
        th = new.imag - ov.imag - mf.imag
        cut = math.sqrt(2.0 / dt)
        el = (mf - hw - (new - ov)) / dt
        el = torch.complex(torch.maximum(torch.minimum(el.real, Eshift + 10 * cut), Eshift - cut), el.imag)
        f = torch.exp(-dt * (el - Eshift))
        weight = weight * torch.clamp(torch.cos(th), min=0.0) * f.abs()
        weight = torch.where(weight.abs() > 100.0, weight * (100.0 / weight.abs()), weight)
        phase = phase * f / f.abs()
        eloc, ov = el, new
    SM = _qr(SM) if closed else torch.cat([_qr(SM[:, :, a:b]) for a, b in blocks], 2)
    G, ov = green(SM)
    out = {}
    if c["kind"] == "measured":
        E = _energy(G, haj, Lnak, scl, blocks)
        ws = weight.sum()
        parts = (weight @ E) / ws
        out["meas"] = torch.stack([parts.sum(), *parts, ws])
    es = torch.log(((weight * torch.exp(dt * eloc)).sum() / weight.sum()).real) / dt
    out.update(Eshift=float(es), SM=SM, weight=weight, phase=phase, pseudo_eloc=eloc, overlap=ov)
    return out


def exact(case, seed):
    c = dict(case)
    k = c["kind"]
    if k == "block":  # its fields and its comb come from the framework's own random streams
        return None
    if k in ("steps", "measured"):
        return _exact_steps(c, seed)
    s = prepare(c, seed)
    if k == "overlap":
        return _logdet(s["PsiT"].to(C128) @ s["SM"])
    if k == "green":
        T = s["PsiT"].to(C128) @ s["SM"]
        return torch.linalg.solve(T.transpose(1, 2), s["SM"].transpose(1, 2)), _logdet(T)
    if k == "vbias":
        G, L = s["G"].reshape(c["W"], -1), s["Lnak"].reshape(c["Nc"], -1)
        v = G @ L.T if c["cplx"] else torch.complex(G.real @ L.T, G.imag @ L.T)
        return 2.0 * math.sqrt(s["dt"]) * v
    if k == "vhs":
        L = s["L"].reshape(-1, c["Nc"]).T
        V = torch.complex(s["X"].real @ L, s["X"].imag @ L)
        return math.sqrt(s["dt"]) * V.reshape(c["W"], c["M"], c["M"])
    if k == "propagate":
        return _propagate(s["SM0"], s["P1"], s["V"])
    if k == "ortho":
        return _qr(s["SM0"])
    return _energy(s["G"], s["haj"], s["Lnak"], 2.0, [(0, c["N"])])
