"""The exchange reductions on both sides of the sizes that go through shared memory."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("N", [1, 5, 23, 24, 32, 33, 60])
def test_fp64(N):
    from safire_b200 import afqmc
    g = torch.Generator(device="cuda").manual_seed(N)
    W, M, Nc = 3, N + 5, 7
    G, haj = (torch.randn(*s, generator=g, device="cuda", dtype=torch.complex128) for s in ((W, N, M), (N, M)))
    L = torch.randn(Nc, N, M, generator=g, device="cuda", dtype=torch.float64)
    T = torch.einsum("wbk,nak->wnba", G, L.to(torch.complex128))
    E = afqmc.energy(G, haj, L)
    # sums of Nc N^2 products of sums of M terms; the moduli's sums bound both
    A = torch.einsum("wbk,nak->wnba", G.abs(), L.abs())
    u = 2.0 ** -53 * 2 * (2 * M + Nc * N * N)
    assert ((E[:, 1] + (T * T.transpose(2, 3)).sum((1, 2, 3))).abs() <= u * (A * A.transpose(2, 3)).sum((1, 2, 3))).all()
    K, KA = (torch.diagonal(X, dim1=2, dim2=3).sum(2) for X in (T, A))
    assert ((E[:, 2] - 2 * (K * K).sum(1)).abs() <= u * 2 * (KA * KA).sum(1)).all()


# rows of N Nc floats: multiples of 16 and not, on both sides of the sizes that go through shared memory; odd ones, whose
# chunks and rows start anywhere
@pytest.mark.parametrize("N,Nc", [(19, 64), (20, 64), (20, 50), (45, 51), (51, 51), (52, 51), (80, 51), (81, 51), (100, 52),
                                  (101, 64)])
def test_int8_slices(N, Nc):
    """Against the FP64 engine on the same walkers: 24-bit slices of G and L."""
    from safire_b200 import afqmc, capi, synthetic
    M, W = max(40, N + 6), 4
    s = synthetic.make_system(synthetic.SystemSpec(M=M, N=N, Nc=Nc, decay=20.0, seed=N))
    rng = np.random.default_rng(N)
    x = s.initial_walkers(W)
    x = x + 0.1 / np.sqrt(M) * (rng.standard_normal(x.shape) + 1j * rng.standard_normal(x.shape))
    out = []
    for p in (capi.PRECISION_INT8X3, capi.PRECISION_FP64):
        e = afqmc.AfqmcEngine(s, W, dt=1e-4, seed=1, precision=p)
        e.set_walkers(x)
        e.init()
        out.append(e.energy())
        e.close()
    assert np.abs(out[0] - out[1]).max() < 2e-6 * np.abs(out[1]).max()
