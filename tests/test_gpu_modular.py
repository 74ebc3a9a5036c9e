"""FP64 products from int8 residues (crt.cuh): the tensor-core path of the large force-bias, vHS, propagation
and energy calls against extended or plain FP64 references, at the edges of its tiles and ranges, and the
operands that it hands to the FP64 tensor pipe."""
import ctypes
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def _modular(A, B):
    from safire_b200.capi import check, lib, ptr
    M, K = A.shape
    N = B.shape[0]
    C = torch.full((M, N), float("nan"), dtype=torch.float64, device="cuda")
    check(lib().sfq_gemm_f64_modular(ptr(A), ptr(B), ptr(C), M, N, K, _stream()))
    torch.cuda.synchronize()
    return C


def _rn(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)


def _cn(g, *shape):
    return torch.complex(_rn(g, *shape), _rn(g, *shape))


# K edges: one MMA step, the K slices' edges, both reductions of the int32 sums (K > 8192); M, N edges:
# single rows, tile and column-tile edges, columns that divide by nothing
@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (3, 17, 31), (128, 256, 32), (129, 257, 128), (127, 255, 129),
                                   (64, 300, 400), (200, 513, 1023), (16, 33, 8192), (17, 30, 8193), (5, 40, 90000)])
@pytest.mark.parametrize("spread", [0.0, 12.0])
def test_product_against_extended_precision(M, N, K, spread):
    """Error relative to the rows' norms: the operands' rounding is at most 2^-59 of their row's norm per
    element, sqrt(K) / 2 of it per row in the 2-norm at most, plus the result's own roundings."""
    g = torch.Generator(device="cuda").manual_seed(M * 7 + N * 3 + K)
    A, B = _rn(g, M, K), _rn(g, N, K)
    if spread:  # rows and columns over 24 decades, entries over 6
        A = A * 10.0 ** (spread * (2 * torch.rand(M, 1, generator=g, device="cuda", dtype=torch.float64) - 1))
        B = B * 10.0 ** (6 * (torch.rand(N, K, generator=g, device="cuda", dtype=torch.float64) - 0.5))
    C = _modular(A, B).cpu().numpy().astype(np.longdouble)
    a, b = A.cpu().numpy().astype(np.longdouble), B.cpu().numpy().astype(np.longdouble)
    R = a @ b.T
    norms = np.sqrt((a * a).sum(1))[:, None] * np.sqrt((b * b).sum(1))[None]
    # two operands, each element off by at most half of 2^(1 - 58) of its norm; four roundings of the result
    bound = 2.0 ** -57 * math.sqrt(K) * norms + 4 * 2.0 ** -53 * np.abs(R)
    assert (np.abs(C - R) <= bound).all()


def test_exact_on_integers_and_zeros():
    g = torch.Generator(device="cuda").manual_seed(5)
    A = torch.randint(-2**20, 2**20, (70, 333), generator=g, device="cuda").double()
    B = torch.randint(-2**20, 2**20, (45, 333), generator=g, device="cuda").double()
    A[3], B[7] = 0.0, 0.0
    C = _modular(A, B)
    R = A.cpu().numpy().astype(np.int64) @ B.cpu().numpy().astype(np.int64).T
    # the operands are held exactly; the sum is rounded to 2^-64 of the residues' range P < 2^118, which is
    # at most 2^(54 - 116) of the rows' scales 2^(e + 58) <= 2 |row| each: 2^-61 of the norms' product at
    # most, then four roundings to FP64
    norms = (A.norm(dim=1)[:, None] * B.norm(dim=1)[None]).cpu().numpy()
    assert (np.abs(C.cpu().numpy() - R) <= 2.0 ** -61 * norms + 2.0 ** -51 * np.abs(R)).all()
    assert (C[3] == 0).all() and (C[:, 7] == 0).all()


@pytest.mark.parametrize("value", [float("inf"), float("nan"), 1e200, 1e-200])
def test_operands_outside_the_range(value):
    """Rows that the residues cannot hold: the result is the FP64 tensor pipe's."""
    g = torch.Generator(device="cuda").manual_seed(6)
    A, B = _rn(g, 40, 150), _rn(g, 50, 150)
    A[5] = 0.0
    A[5, 9] = value
    C, R = _modular(A, B).cpu(), (A.cpu() @ B.cpu().T)
    assert torch.equal(torch.isnan(C), torch.isnan(R)) and torch.equal(torch.isinf(C), torch.isinf(R))
    ok = torch.isfinite(R)
    # the FP64 chain's own bound
    bound = 150 * 2.0 ** -53 * (A.cpu().abs().nan_to_num(0, 0, 0) @ B.cpu().abs().T)
    assert ((C - R).abs()[ok] <= 2 * bound[ok]).all()


@pytest.mark.parametrize("fa,fb", [(1e118, 1e118), (1e-118, 1e-118), (1e118, 1e-118)])
def test_edges_of_the_range(fa, fb):
    """Rows whose norms are just inside the range: both scales at their largest or smallest."""
    g = torch.Generator(device="cuda").manual_seed(8)
    A, B = _rn(g, 20, 60) * fa, _rn(g, 30, 60) * fb
    C = _modular(A, B).cpu().numpy().astype(np.longdouble)
    R = A.cpu().numpy().astype(np.longdouble) @ B.cpu().numpy().astype(np.longdouble).T
    assert float(np.abs(C - R).max() / np.abs(R).max()) < 4 * 2.0 ** -53


def _workspace_path(op, *sizes):
    from safire_b200.capi import lib
    return lib().sfq_workspace_size(op, *sizes)


@pytest.mark.parametrize("W,M,N", [(44, 331, 49),    # one row tile of [re; im], odd sizes
                                   (36, 320, 64),    # [re; im] exactly 128 rows
                                   (36, 321, 65),    # two row tiles
                                   (18, 330, 128),   # the widest electron block
                                   (17, 333, 129),   # two chunks of electrons
                                   (5, 1030, 48),    # K slices that leave room for few electrons
                                   (3, 900, 100)])   # fewer units than SMs: split columns
@pytest.mark.parametrize("order", [1, 6])
def test_propagate(W, M, N, order):
    from safire_b200 import afqmc, capi
    f64 = 3 * ((16 * W * M * N + 255) // 256 * 256)
    assert _workspace_path(capi.OP_PROPAGATE, W, M, N, 0) > f64  # the int8 path runs
    g = torch.Generator(device="cuda").manual_seed(W + M + N)
    SM = _cn(g, W, M, N)
    V = _cn(g, W, M, M) * (0.3 / math.sqrt(M))
    P1 = torch.eye(M, device="cuda", dtype=torch.float64) + 1e-2 * _rn(g, M, M)
    P = P1.to(torch.complex128)
    T = P @ SM
    S = T.clone()
    for k in range(1, order + 1):
        T = (V @ T) * (1j / k)
        S += T
    R = P @ S
    out = afqmc.Propagate(SM.clone(), P1, V, order=order)
    assert float((out - R).norm() / R.norm()) < 2e-15  # both within a few roundings of the exact chain
    SM[0, 0, 0] = float("nan")  # a walker that the residues cannot hold: the FP64 tensor pipe's chain
    bad = afqmc.Propagate(SM.clone(), P1, V, order=order)
    assert torch.isnan(bad[0, :, 0].real).all() and not torch.isnan(bad[0, :, 1:].real).any()
    assert W == 1 or float((bad[1:] - R[1:]).norm() / R[1:].norm()) < 1e-14


@pytest.mark.parametrize("W,M,N,Nc,cplx", [(150, 100, 30, 1200, False), (8, 101, 23, 613, True),
                                           (300, 103, 10, 65, False)])
def test_vbias(W, M, N, Nc, cplx):
    from safire_b200 import afqmc, capi
    assert _workspace_path(capi.OP_VBIAS_COMPLEX if cplx else capi.OP_VBIAS, W, M, N, Nc) > 0
    g = torch.Generator(device="cuda").manual_seed(W)
    G, L = _cn(g, W, N, M), (_cn(g, Nc, N, M) if cplx else _rn(g, Nc, N, M))
    R = 2 * math.sqrt(0.01) * (G.reshape(W, -1) @ L.to(torch.complex128).reshape(Nc, -1).T)
    assert float((afqmc.vbias(G, L, 0.01) - R).norm() / R.norm()) < 1e-14
    L[3, 2, 1] = float("inf")
    bad = afqmc.vbias(G, L, 0.01)
    assert not torch.isfinite(bad[:, 3].real).any() and torch.isfinite(bad[:, :3].real).all()


@pytest.mark.parametrize("W,M,Nc", [(100, 160, 401), (200, 61, 1400), (97, 130, 700)])
def test_vhs(W, M, Nc):
    from safire_b200 import afqmc, capi
    assert _workspace_path(capi.OP_VHS, W, M, 0, Nc) > 0
    g = torch.Generator(device="cuda").manual_seed(W)
    L, X = _rn(g, M, M, Nc), _cn(g, W, Nc)
    R = 0.1 * (X @ L.to(torch.complex128).reshape(M * M, Nc).T).reshape(W, M, M)
    V = afqmc.vHS(L, X, 0.01)
    assert float((V - R).norm() / R.norm()) < 1e-14
    X[1, 5] = float("nan")
    bad = afqmc.vHS(L, X, 0.01)
    assert torch.isnan(bad[1].real).all() and float((bad[2:] - R[2:]).norm() / R[2:].norm()) < 1e-14


@pytest.mark.parametrize("W,M,N,Nc,cplx", [(20, 120, 45, 1100, False),   # padded columns of a vector
                                           (16, 90, 70, 800, True),      # complex Lnak, two row tiles
                                           (10, 130, 116, 300, False)])  # the largest block in shared memory
def test_energy(W, M, N, Nc, cplx):
    from safire_b200 import afqmc, capi
    nv = min(Nc, 2**27 // (W * N * N))
    assert _workspace_path(capi.OP_ENERGY, W, M, N, Nc) > 16 * W * (N * nv * N + 2 * Nc) + 4096  # the int8 path's
    g = torch.Generator(device="cuda").manual_seed(N)
    G, haj = _cn(g, W, N, M), _cn(g, N, M)
    L = _cn(g, Nc, N, M) if cplx else _rn(g, Nc, N, M)
    Lc = L.to(torch.complex128)
    R = torch.zeros(W, 3, device="cuda", dtype=torch.complex128)
    R[:, 0] = 0.25 + 2.0 * torch.einsum("waj,aj->w", G, haj)
    K = torch.empty(W, Nc, device="cuda", dtype=torch.complex128)
    for n in range(Nc):
        T = G @ Lc[n].T  # (W, b, a)
        R[:, 1] -= (T * T.transpose(1, 2)).sum((1, 2))
        K[:, n] = torch.diagonal(T, dim1=1, dim2=2).sum(1)
    R[:, 2] = 2.0 * (K * K).sum(1)
    scale = R.abs().max(dim=0).values
    E = afqmc.energy(G, haj, L, E0=0.25)
    assert float(((E - R).abs() / scale).max()) < 1e-12
    L[5, 2, 3] = float("nan")  # the FP64 tensor pipe's sums
    bad = afqmc.energy(G, haj, L, E0=0.25)
    assert torch.isnan(bad[:, 1].real).all() and float((bad[:, 0] - R[:, 0]).abs().max()) < 1e-9


# the loads stop before the first slice, within the first tile (or unit) and, in the walker kernel, after a tile
# whose rows stay; K = 300 has three 128-byte slices a tile and five 64-byte ones
@pytest.mark.parametrize("walker,hold_at,N", [(0, 0, 600), (0, 2, 600), (1, 0, 600), (1, 3, 600), (1, 5, 12000),
                                              (1, 7, 12000)])  # 12000: two column tiles a unit
def test_bounded_waits_expire(walker, hold_at, N):
    """Every wait limited to 1 ms: the kernel gives up with nothing in flight, the expiry is counted, the FP64
    product replaces the result, and the next product on the same context is right."""
    from safire_b200.capi import check, lib, ptr
    g = torch.Generator(device="cuda").manual_seed(hold_at)
    M, K = 64, 300
    A, B = _rn(g, M, K), _rn(g, N, K)
    R = A @ B.T
    n0, n1 = ctypes.c_ulonglong(), ctypes.c_ulonglong()
    check(lib().sfq_modular_expiries(ctypes.byref(n0)))
    C = torch.full((M, N), float("nan"), dtype=torch.float64, device="cuda")
    assert lib().sfq_selftest_modular_expiry(ptr(A), ptr(B), ptr(C), M, N, K, walker, hold_at, 1_000_000,
                                             _stream()) == 8  # SFQ_ERR_TIMEOUT
    check(lib().sfq_modular_expiries(ctypes.byref(n1)))
    assert n1.value == n0.value + 1
    # two FP64 sums of K terms
    bound = 2 * K * 2.0 ** -53 * (A.abs() @ B.abs().T)
    assert ((C - R).abs() <= bound).all()
    C.fill_(float("nan"))
    assert lib().sfq_selftest_modular_expiry(ptr(A), ptr(B), ptr(C), M, N, K, walker, 10**6, 1_000_000_000,
                                             _stream()) == 0
    assert ((C - R).abs() <= bound).all()
    assert ((_modular(A, B) - R).abs() <= bound).all()


@pytest.mark.parametrize("value", [float("nan"), 1e200])
def test_one_walker_outside_the_range_leaves_the_others(value):
    """A walker that the residues cannot hold goes through the FP64 tensor pipe on its own: the others' results are
    the same bits as without it."""
    from safire_b200 import afqmc
    g = torch.Generator(device="cuda").manual_seed(12)
    W, M, N, Nc = 97, 250, 50, 700
    G, haj, L = _cn(g, W, N, M), _cn(g, N, M), _rn(g, Nc, N, M)
    SM, X = _cn(g, W, M, N), _cn(g, W, Nc)
    V = _cn(g, W, M, M) * (0.3 / math.sqrt(M))
    Lik, P1 = _rn(g, M, M, Nc), torch.eye(M, device="cuda", dtype=torch.float64) + 1e-2 * _rn(g, M, M)
    bad = 35

    def put(t, at):
        t = t.clone()
        t[at] = value
        return t

    pairs = [(afqmc.vbias(G, L, 0.01), afqmc.vbias(put(G, (bad, 3, 5)), L, 0.01)),
             (afqmc.vHS(Lik, X, 0.01), afqmc.vHS(Lik, put(X, (bad, 7)), 0.01)),
             (afqmc.energy(G, haj, L), afqmc.energy(put(G, (bad, 3, 5)), haj, L)),
             (afqmc.Propagate(SM.clone(), P1, V), afqmc.Propagate(put(SM, (bad, 3, 5)), P1, V)),
             (afqmc.Propagate(SM.clone(), P1, V), afqmc.Propagate(SM.clone(), P1, put(V, (bad, 3, 5))))]
    for clean, with_bad in pairs:
        rest = [w for w in range(W) if w != bad]
        assert torch.equal(torch.view_as_real(clean)[rest], torch.view_as_real(with_bad)[rest])
        assert not torch.equal(clean[bad], with_bad[bad])


U = 2.0 ** -53


def _ld(t):
    a = t.cpu().numpy()
    return a.astype(np.clongdouble if np.iscomplexobj(a) else np.longdouble)


def _graded(g, rows, K, decades, rising):
    """Rows whose entries fall (or rise) over so many decades."""
    e = torch.arange(K, device="cuda", dtype=torch.float64) / max(1, K - 1) * decades
    return _rn(g, rows, K) * 10.0 ** (e - decades if rising else -e)


@pytest.mark.parametrize("decades", [0, 1, 2, 3, 6, 12, 18, 40])
@pytest.mark.parametrize("W,Nc,K", [(40, 70, 2400), (130, 300, 1026), (8, 64, 40000)])
def test_graded_rows_keep_the_fp64_bound(W, Nc, K, decades):
    """Rows graded in opposite directions: every output within the FP64 chain's own bound K u sum_k |a_k| |b_k|."""
    from safire_b200 import afqmc, capi
    assert _workspace_path(capi.OP_VBIAS, W, K // 2, 2, Nc) > 0
    g = torch.Generator(device="cuda").manual_seed(decades + K)
    A = torch.complex(_graded(g, W, K, decades, False), _graded(g, W, K, decades, False))
    B = _graded(g, Nc, K, decades, True)
    C = _ld(afqmc.vbias(A.reshape(W, 2, K // 2), B.reshape(Nc, 2, K // 2), 0.25))  # 2 sqrt(dt) = 1
    a, b = _ld(A), _ld(B)
    for part in ("real", "imag"):
        p = getattr(a, part)
        assert (np.abs(getattr(C, part) - p @ b.T) <= (K + 2) * U * (np.abs(p) @ np.abs(b).T)).all()


def test_graded_operands_of_the_calls():
    """The same through the public calls (sizes on the int8 path): graded operands, and imaginary parts far below the
    real ones, which are sums of their own."""
    from safire_b200 import afqmc
    g = torch.Generator(device="cuda").manual_seed(2)
    W, M, Nc = 97, 130, 700
    s = math.sqrt(0.01)
    L = _graded(g, M * M, Nc, 10, False).reshape(M, M, Nc)
    for X in (torch.complex(_graded(g, W, Nc, 10, True), _graded(g, W, Nc, 10, True)),
              torch.complex(_rn(g, W, Nc), 1e-9 * _rn(g, W, Nc))):
        V, x, l = _ld(afqmc.vHS(L, X, 0.01)).reshape(W, M * M)[:4], _ld(X)[:4], _ld(L.reshape(M * M, Nc))
        for part in ("real", "imag"):
            p = getattr(x, part)
            err = np.abs(getattr(V, part) - s * (p @ l.T))
            assert (err <= (Nc + 4) * U * s * (np.abs(p) @ np.abs(l).T)).all()
    N, Nc = 23, 613
    K = N * M
    for Lc in (_graded(g, Nc, K, 10, False), torch.complex(_graded(g, Nc, K, 10, False), _graded(g, Nc, K, 10, False))):
        G = torch.complex(_graded(g, W, K, 10, True), 1e-6 * _graded(g, W, K, 10, True))
        v = _ld(afqmc.vbias(G.reshape(W, N, M), Lc.reshape(Nc, N, M), 0.01))[:3]
        x, l = _ld(G)[:3], _ld(Lc)
        R = 2 * s * (x @ l.T)
        # the four real products' sums of moduli, each part on its own
        re = np.abs(x.real) @ np.abs(l.real).T + np.abs(x.imag) @ np.abs(l.imag).T
        im = np.abs(x.imag) @ np.abs(l.real).T + np.abs(x.real) @ np.abs(l.imag).T
        assert (np.abs(v.real - R.real) <= (2 * K + 4) * U * 2 * s * re).all()
        assert (np.abs(v.imag - R.imag) <= (2 * K + 4) * U * 2 * s * im).all()


@pytest.mark.parametrize("kind", ["unit", "near", "graded"])
def test_propagate_keeps_small_elements(kind):
    """Walkers of unit vectors, of unit vectors and little else, and graded V: every element within the FP64 chain's
    bound, the same recursion on the moduli times its number of roundings."""
    from safire_b200 import afqmc
    g = torch.Generator(device="cuda").manual_seed(4)
    W, M, N, order = 90, 250, 48, 6
    SM = torch.zeros(W, M, N, dtype=torch.complex128, device="cuda")
    SM[:, torch.arange(N), torch.arange(N)] = 1.0
    V = torch.complex(_rn(g, W, M, M), 0.2 * _rn(g, W, M, M)) * (0.25 / math.sqrt(M))
    if kind == "near":
        SM += 1e-7 * _cn(g, W, M, N)
    if kind == "graded":  # rows of V fall over the orbitals, the walkers rise
        f = 10.0 ** (-8.0 * torch.arange(M, device="cuda", dtype=torch.float64) / M)
        SM = _cn(g, W, M, N) / f[None, :, None] * 1e-8
        V = V * f[None, None, :]
    P1 = torch.diag(1.0 + 1e-3 * _rn(g, M)) + 1e-6 * _rn(g, M, M)
    out = _ld(afqmc.Propagate(SM.clone(), P1, V, order=order))
    p = _ld(P1)
    for w in range(2):
        v, x = _ld(V[w]), _ld(SM[w])

        def chain(p, v, x, i):
            t = p @ x
            s = t
            for k in range(1, order + 1):
                t = i * (v @ t) / k
                s = s + t
            return p @ s

        R = chain(p, v, x, np.clongdouble(1j))
        am = lambda z: np.abs(z.real) + np.abs(z.imag)  # noqa: E731 - bounds both parts of the complex products
        B = chain(np.abs(p), am(v), am(x), 1)
        assert (np.abs(out[w] - R) <= (2 * M * (order + 2)) * U * B).all()


def test_scratch_is_bounded():
    """The walkers' planes come in parts too: what the int8 path takes does not grow with the walkers without end."""
    from safire_b200 import capi
    gib = 1 << 30
    for W in (4096, 16384, 60000):
        # 16 bytes a plane element: 2 W x 40000 of them for all walkers at once would be 5 to 77 GB
        assert 0 < _workspace_path(capi.OP_VBIAS, W, 400, 100, 2400) < 4 * gib
        assert 0 < _workspace_path(capi.OP_VBIAS_COMPLEX, W, 400, 100, 2400) < 4 * gib
        assert 0 < _workspace_path(capi.OP_VHS, W, 400, 0, 2400) < 4 * gib
        vec = 2 * 16 * W * 2400  # the energy's sums per walker and vector
        chunk = max(16 * W * 100 * 100, 2 * gib)  # the FP64 path's exchange chunk
        assert _workspace_path(capi.OP_ENERGY, W, 400, 100, 2400) < max(4 * gib, chunk) + vec + gib // 8


def _rel(x, y):
    return float((x - y).norm() / y.norm())


# uneven last parts of the shared rows and of the walkers (1.5 GiB of planes at a time); a row that cannot be held in the
# last part only
def test_parts_of_vbias():
    from safire_b200 import afqmc
    g = torch.Generator(device="cuda").manual_seed(21)
    for W, M, N, Nc, cplx in ((9, 400, 100, 2501, False), (1301, 400, 100, 67, False), (701, 400, 100, 65, True)):
        G = torch.randn(W, N, M, generator=g, device="cuda", dtype=torch.complex128)
        L = _rn(g, Nc, N, M) if not cplx else torch.randn(Nc, N, M, generator=g, device="cuda", dtype=torch.complex128)
        Lc = L.to(torch.complex128).reshape(Nc, -1).T
        out = afqmc.vbias(G, L, 0.25)
        assert _rel(out, G.reshape(W, -1) @ Lc) < 1e-14
        G[W - 1, 3, 5] = float("nan")
        bad = afqmc.vbias(G, L, 0.25)
        assert torch.isnan(bad[W - 1].real).all()
        assert torch.equal(torch.view_as_real(bad[:-1]), torch.view_as_real(out[:-1]))
        G[W - 1, 3, 5] = 0.0
        L[Nc - 1, 3, 5] = float("inf")
        bad = afqmc.vbias(G, L, 0.25)
        assert not torch.isfinite(bad[:W - 1, Nc - 1].real).any()
        # an FP64 sum of 2 K random terms: u sqrt(2 K) at most
        assert _rel(bad[:W - 1, :Nc - 1], out[:W - 1, :Nc - 1]) < U * math.sqrt(2 * N * M)
        del G, L, Lc, out, bad


def test_parts_of_vhs():
    from safire_b200 import afqmc
    g = torch.Generator(device="cuda").manual_seed(22)
    for W, M, Nc in ((101, 250, 3001), (17001, 9, 3000)):  # three parts of the rows; two of the walkers
        L, X = _rn(g, M, M, Nc), _cn(g, W, Nc)
        out = afqmc.vHS(L, X, 0.01)
        R = 0.1 * (X @ L.to(torch.complex128).reshape(M * M, Nc).T).reshape(W, M, M)
        assert _rel(out, R) < 1e-14
        X[W - 1, 5] = float("nan")
        bad = afqmc.vHS(L, X, 0.01)
        assert torch.isnan(bad[W - 1].real).all()
        assert torch.equal(torch.view_as_real(bad[:-1]), torch.view_as_real(out[:-1]))
        X[W - 1, 5] = 0.0
        L[M - 1, M - 1, Nc - 1] = 1e200
        bad = afqmc.vHS(L, X, 0.01)
        assert float(bad[:W - 1, M - 1, M - 1].abs().median()) > 1e198
        bad[:, M - 1, M - 1] = out[:, M - 1, M - 1] = 0.0
        assert _rel(bad[:-1], out[:-1]) < 1e-14


def test_parts_of_propagate():
    from safire_b200 import afqmc
    g = torch.Generator(device="cuda").manual_seed(23)
    W, M, N = 161, 400, 100  # two parts of the walkers, 81 and 80
    SM, V = _cn(g, W, M, N), _cn(g, W, M, M) * (0.3 / math.sqrt(M))
    P1 = torch.eye(M, device="cuda", dtype=torch.float64) + 1e-2 * _rn(g, M, M)
    T = P1.to(torch.complex128) @ SM
    S = T.clone()
    for k in range(1, 7):
        T = (V @ T) * (1j / k)
        S += T
    out = afqmc.Propagate(SM.clone(), P1, V)
    assert _rel(out, P1.to(torch.complex128) @ S) < 2e-15
    V[W - 1, 7, 8] = float("inf")
    bad = afqmc.Propagate(SM.clone(), P1, V)
    assert not torch.isfinite(bad[W - 1].real).any()
    assert torch.equal(torch.view_as_real(bad[:-1]), torch.view_as_real(out[:-1]))


def test_parts_of_energy():
    from safire_b200 import afqmc
    g = torch.Generator(device="cuda").manual_seed(24)
    for W, M, N, Nc in ((30, 60, 70, 997), (1300, 400, 90, 7)):  # parts of the vectors; of the walkers
        G, haj, L = _cn(g, W, N, M), _cn(g, N, M), _rn(g, Nc, N, M)
        out = afqmc.energy(G, haj, L)
        E = torch.zeros(W, 2, device="cuda", dtype=torch.complex128)
        K = torch.empty(W, Nc, device="cuda", dtype=torch.complex128)
        for n in range(Nc):
            T = G @ L[n].to(torch.complex128).T
            E[:, 0] -= (T * T.transpose(1, 2)).sum((1, 2))
            K[:, n] = torch.diagonal(T, dim1=1, dim2=2).sum(1)
        E[:, 1] = 2.0 * (K * K).sum(1)
        scale = E.abs().max(dim=0).values
        assert float(((out[:, 1:] - E).abs() / scale).max()) < 1e-12
        G[W - 1, 3, 5] = float("nan")
        bad = afqmc.energy(G, haj, L)
        assert torch.isnan(bad[W - 1].real).all()
        assert torch.equal(torch.view_as_real(bad[:-1]), torch.view_as_real(out[:-1]))
        G[W - 1, 3, 5] = 0.0
        L[Nc - 1, N - 1, M - 1] = float("nan")
        bad = afqmc.energy(G, haj, L)
        assert torch.isnan(bad[:, 1].real).all()


def test_no_room_for_the_workspace(monkeypatch):
    """Where the device has no room for the int8 path's workspace (an allocator that refuses it) the calls run on the
    FP64 tensor pipe, in its own; where there is none for that either, they raise as before."""
    from safire_b200 import afqmc, capi
    g = torch.Generator(device="cuda").manual_seed(31)
    W, M, N, Nc = 90, 250, 48, 700
    G, L, Lik = _cn(g, W, N, M), _rn(g, Nc, N, M), _rn(g, M, M, Nc)
    Ge, haj, Le = _cn(g, 20, 45, 190), _cn(g, 45, 190), _rn(g, 1100, 45, 190)
    SM, X, V = _cn(g, W, M, N), _cn(g, 100, Nc), _cn(g, W, M, M) * (0.3 / math.sqrt(M))
    P1 = torch.eye(M, device="cuda", dtype=torch.float64) + 1e-2 * _rn(g, M, M)
    calls = [(lambda: afqmc.vbias(G, L, 0.01), 0, _workspace_path(capi.OP_VBIAS, W, M, N, Nc)),
             (lambda: afqmc.vHS(Lik, X, 0.01), 0, _workspace_path(capi.OP_VHS, 100, M, 0, Nc)),
             (lambda: afqmc.Propagate(SM.clone(), P1, V), _workspace_path(capi.OP_PROPAGATE_PIPE, W, M, N, 0),
              _workspace_path(capi.OP_PROPAGATE, W, M, N, 0)),
             (lambda: afqmc.energy(Ge, haj, Le), _workspace_path(capi.OP_ENERGY_PIPE, 20, 190, 45, 1100),
              _workspace_path(capi.OP_ENERGY, 20, 190, 45, 1100))]
    empty = torch.empty
    for call, pipe, full in calls:
        assert full > pipe
        want = call()

        def refuse(most):
            def alloc(*size, **kw):
                if kw.get("dtype") is torch.uint8 and size[0] > most:
                    raise torch.OutOfMemoryError("no room")
                return empty(*size, **kw)
            monkeypatch.setattr(afqmc.torch, "empty", alloc)

        refuse(full - 1)
        got = call()
        if pipe:
            refuse(pipe - 1)
            with pytest.raises(torch.OutOfMemoryError):
                call()
        monkeypatch.undo()
        # each side rounds its sums of up to 12000 terms in its own order
        assert _rel(got, want) < U * math.sqrt(2 * N * M) and not torch.equal(got, want)


def test_int8_path_where_it_does_not_gain():
    """Sizes that the int8 path takes without being the faster one: the calls leave them to the FP64 tensor pipe, and a
    C caller's full workspace still chooses it."""
    from safire_b200 import afqmc, capi
    from safire_b200.capi import check, lib, ptr
    g = torch.Generator(device="cuda").manual_seed(41)
    W, M, N, Nc = 300, 103, 10, 65
    assert not lib().sfq_int8_gains(capi.OP_VBIAS, W, M, N, Nc, 0)
    G, L = _cn(g, W, N, M), _rn(g, Nc, N, M)
    ws = torch.empty(_workspace_path(capi.OP_VBIAS, W, M, N, Nc), dtype=torch.uint8, device="cuda")
    v = torch.empty(W, Nc, dtype=torch.complex128, device="cuda")
    check(lib().sfq_vbias_ws(ptr(G), ptr(L), 0, ptr(v), W, N, M, Nc, 0.25, 1, ptr(ws), ws.numel(), _stream()))
    pipe = afqmc.vbias(G, L, 0.25)
    R = G.reshape(W, -1) @ L.to(torch.complex128).reshape(Nc, -1).T
    assert _rel(v, R) < 1e-14 and _rel(pipe, R) < 1e-14 and not torch.equal(v, pipe)
    for W, M, N, Nc in ((20, 120, 45, 1100), (10, 130, 116, 300)):  # padded columns; the largest block in shared memory
        assert not lib().sfq_int8_gains(capi.OP_ENERGY, W, M, N, Nc, 0)
        G, haj, L = _cn(g, W, N, M), _cn(g, N, M), _rn(g, Nc, N, M)
        ws = torch.empty(_workspace_path(capi.OP_ENERGY, W, M, N, Nc), dtype=torch.uint8, device="cuda")
        E = torch.empty(W, 3, dtype=torch.complex128, device="cuda")
        check(lib().sfq_energy(ptr(E), ptr(G), ptr(haj), ptr(L), 0, 0.0, W, N, M, Nc, 1, 1, 1, ptr(ws), ws.numel(),
                               _stream()))
        pipe = afqmc.energy(G, haj, L)
        scale = pipe.abs().max(dim=0).values
        # two FP64 evaluations of sums of up to 1.2e6 products of sums of M terms
        assert float(((E - pipe).abs() / scale).max()) < 1e-12 and not torch.equal(E, pipe)
        L[5, 2, 3] = float("nan")
        check(lib().sfq_energy(ptr(E), ptr(G), ptr(haj), ptr(L), 0, 0.0, W, N, M, Nc, 1, 1, 1, ptr(ws), ws.numel(),
                               _stream()))
        assert torch.isnan(E[:, 1].real).all() and torch.equal(E[:, 0], pipe[:, 0])
    # a pipe's workspace that would hold the int8 path's too
    W, M, N, Nc = 128, 120, 44, 700
    assert _workspace_path(capi.OP_ENERGY_PIPE, W, M, N, Nc) == _workspace_path(capi.OP_ENERGY, W, M, N, Nc)
    G, haj, L = _cn(g, W, N, M), _cn(g, N, M), _rn(g, Nc, N, M)
    n = _workspace_path(capi.OP_ENERGY, W, M, N, Nc) + 512
    ws = torch.empty(n, dtype=torch.uint8, device="cuda")
    E = torch.empty(W, 3, dtype=torch.complex128, device="cuda")
    check(lib().sfq_energy(ptr(E), ptr(G), ptr(haj), ptr(L), 0, 0.0, W, N, M, Nc, 1, 1, 1, ptr(ws), n, _stream()))
    pipe = afqmc.energy(G, haj, L)
    assert float(((E - pipe).abs() / pipe.abs().max(dim=0).values).max()) < 1e-12 and not torch.equal(E, pipe)
