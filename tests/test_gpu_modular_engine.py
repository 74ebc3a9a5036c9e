"""FP64 engines on the int8 tensor cores (residue planes made at setup) against the same engines on the FP64 tensor
pipe: every walker type, complex trials, Cholesky vectors that are not symmetric, blocks replayed from a graph; and what
becomes of them where device memory is short."""
import dataclasses

import numpy as np
import pytest

from oracle import afqmc_oracle as O
from safire_b200 import afqmc, synthetic
from safire_b200.serve import Server

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

# every product of an engine of these sizes is on the int8 path (vHS from 32 walkers, the energy from 40 electrons, the
# propagation from 250 orbitals and 48 electrons)
M, N, NC, W = 256, 48, 300, 80
DT = 1e-4


def _system(kind, seed=3):
    s = synthetic.make_system(synthetic.SystemSpec(M=M, N=N, Nc=NC, decay=NC / 6.0, seed=seed))
    rng = np.random.default_rng(seed)
    if kind == "complex":
        q = np.linalg.qr(rng.standard_normal((M, N)) + 1j * rng.standard_normal((M, N)))[0]
        return dataclasses.replace(s, PsiT=np.ascontiguousarray(q.T))
    if kind == "asymmetric":
        return dataclasses.replace(s, Likn=s.Likn * (1.0 + 1e-3 * rng.standard_normal((M, M, 1))))
    if kind == "collinear":
        psi = np.linalg.eigh(s.hcore)[1]
        return dataclasses.replace(s, PsiT=np.concatenate([psi[:, :28].T, psi[:, :20].T]).astype(np.complex128),
                                   nel_dn=20)
    if kind == "noncollinear":
        q = np.linalg.qr(rng.standard_normal((2 * M, N)) + 1j * rng.standard_normal((2 * M, N)))[0]
        return dataclasses.replace(s, PsiT=np.ascontiguousarray(q.T), npol=2)
    return s


def _engine(s, modular, walkers):
    e = afqmc.AfqmcEngine(s, W, dt=DT, seed=7, modular=modular)
    e.set_walkers(walkers)
    return e


def _walkers(s, seed=5):
    rng = np.random.default_rng(seed)
    x = s.initial_walkers(W)
    return x + 0.3 / np.sqrt(M) * (rng.standard_normal(x.shape) + 1j * rng.standard_normal(x.shape))


def _close(a, b, tol):
    assert np.abs(a - b).max() <= tol * np.abs(b).max(), np.abs(a - b).max() / np.abs(b).max()


@pytest.mark.parametrize("kind", ["closed", "complex", "asymmetric", "collinear", "noncollinear"])
def test_planes_against_the_pipe(kind):
    s = _system(kind)
    x = _walkers(s)
    a, b = _engine(s, True, x), _engine(s, False, x)
    assert a.footprint() > b.footprint()
    Ea, Eb = a.init(), b.init()
    # FP64 sums of a few hundred to 11520 terms, each side rounded in its own order, through divisions by the overlap
    assert abs(Ea - Eb) <= 1e-12 * abs(Eb)
    _close(a.energy(), b.energy(), 1e-12)
    uni = np.random.default_rng(9).uniform(1e-12, 1 - 1e-12, (3, W, NC))
    for i in range(3):
        u = torch.from_numpy(uni[i]).cuda()
        a.propagate(Ea, i, uniforms=u)
        b.propagate(Ea, i, uniforms=u)
        torch.cuda.synchronize()
    (xa, pa), (xb, pb) = a.walkers(), b.walkers()
    _close(xa, xb, 1e-12)
    assert not np.array_equal(xa, xb)  # they are two paths
    for k in ("WEIGHT", "OVLP", "PHASE"):
        _close(pa[k], pb[k], 1e-10)  # the overlaps' difference over dt
    a.orthogonalize()
    b.orthogonalize()
    _close(a.energy(), b.energy(), 1e-11)
    a.close()
    b.close()


def test_planes_against_the_oracle():
    """Two steps, the orthogonalization and the energy of walkers that the planes hold, at the bar of the FP64 engine."""
    s = _system("closed")
    x = _walkers(s)
    e = _engine(s, True, x)
    ham = O.Hamiltonian(s.hcore, s.Likn, s.PsiT)
    prop = O.Propagator(ham, DT, seed=7)
    wo = O.Walkers(x.copy())
    Eo = O.init_walkers(ham, wo)
    assert abs(e.init() - Eo) < 1e-10 * abs(Eo)
    for step in range(2):
        prop.propagate(wo, Eo, step)
        e.propagate(Eo, step)
    prop.orthogonalize(wo)
    e.orthogonalize()
    SM, pr = e.walkers()
    _close(SM, wo.SM, 1e-10)
    _close(pr["WEIGHT"], wo.weight, 1e-10)
    _close(pr["OVLP"], wo.ovlp, 1e-10)
    _close(e.energy(), O.wfn_energy_noupdate(ham, wo)[0], 1e-10)
    e.close()


def test_blocks_replayed_from_a_graph():
    """The flags that send walkers to the FP64 pipe are part of the graph: a block whose walkers the planes cannot all
    hold, then one where they can."""
    s = _system("closed")
    x = _walkers(s)
    kw = dict(ortho_interval=5, pop_interval=100, equilibration_steps=0, measure_interval=5)
    y = s.initial_walkers(W)  # unit vectors and little else
    for first in (x, y):
        a, b = _engine(s, True, first), _engine(s, False, first)
        Ea = Eb = a.init()
        b.init()
        for blk in range(2):
            Ea, ma = a.run_block(5, Ea, step0=5 * blk, **kw)
            Eb, mb = b.run_block(5, Eb, step0=5 * blk, **kw)
            _close(np.asarray(ma), np.asarray(mb), 1e-9)
            _close(a.walkers()[0], b.walkers()[0], 1e-10)
            for e in (a, b):
                e.set_walkers(x)
                e.init()
        a.close()
        b.close()


def test_short_memory_declines_the_planes():
    """An engine is built wherever the FP64 pipe's is, and leaves at least half of the memory that was free."""
    s = _system("closed")
    b = _engine(s, False, _walkers(s))
    arena = b.footprint()
    b.close()
    a = _engine(s, True, _walkers(s))
    extra = a.footprint() - arena
    assert extra > 0
    a.close()
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    hog = torch.empty(int(free - arena - 1.8 * extra), dtype=torch.uint8, device="cuda")  # half of what is left: 0.9 extra
    try:
        a = _engine(s, True, _walkers(s))
        assert arena <= a.footprint() < arena + extra
        a.init()
        a.propagate(0.0, 0)
        a.synchronize()
        a.close()
    finally:
        del hog
        torch.cuda.empty_cache()


def test_server_builds_what_fits_the_budget():
    s = _system("closed")
    sizes = []
    for modular in (False, True):
        e = _engine(s, modular, _walkers(s))
        sizes.append(e.footprint())
        e.close()
    budget = (sizes[0] + sizes[1]) / 2  # the FP64 pipe's engine fits, the planes do not
    srv = Server(hbm_budget_gb=budget / 1e9, max_inflight=1)
    sid = srv.add_system(s, W, dt=DT, seed=7)
    r = srv.submit(sid, steps=2, ortho_interval=2, pop_interval=100, equilibration_steps=0, measure_interval=2)
    srv.drain([r])
    assert srv.request(r)["status"] == 0
    srv.close()
