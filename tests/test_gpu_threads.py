"""Two host threads on one GPU with systems of different sizes: what one call sets on a kernel must not refuse the
other's launch."""
import threading

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _run_together(jobs, calls):
    """Each job on a thread and stream of its own; the errors raised."""
    errors = []
    start = threading.Barrier(len(jobs))

    def work(job):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                start.wait()
                for _ in range(calls):
                    job()
        except Exception as e:  # noqa: BLE001 - reported below
            errors.append(e)

    ts = [threading.Thread(target=work, args=(j,)) for j in jobs]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    torch.cuda.synchronize()
    return errors


@pytest.mark.parametrize("kind", ["energy", "orthogonalize", "inverse"])
def test_sizes_that_take_different_shared_memory(kind):
    from safire_b200 import afqmc
    g = torch.Generator(device="cuda").manual_seed(3)

    def cn(*s):
        return torch.randn(*s, generator=g, device="cuda", dtype=torch.complex128)

    # the larger of the two takes more than the 48 KB that a kernel has without being asked for more
    small, large = {"energy": (40, 100), "orthogonalize": (20, 100), "inverse": (105, 118)}[kind]
    jobs = []
    for n in (small, large):
        if kind == "energy":
            G, haj = cn(1, n, n + 4), cn(n, n + 4)
            L = torch.randn(1, n, n + 4, generator=g, device="cuda", dtype=torch.float64)
            jobs.append(lambda G=G, haj=haj, L=L: afqmc.energy(G, haj, L))
        elif kind == "orthogonalize":
            jobs.append(lambda S=cn(1, n + 30, n): afqmc.orthogonalize(S))
        else:
            jobs.append(lambda A=cn(1, n, n): afqmc.inverse_logdet(A))
    torch.cuda.synchronize()
    assert _run_together(jobs, 1500) == []


def test_group_of_members_with_different_shared_memory():
    """Members whose exchange blocks need more than 48 KB of shared memory beside smaller ones, captured into one graph
    before any of it runs: every member's block is the one it gets alone."""
    import numpy as np

    from safire_b200 import afqmc, capi, synthetic
    blk = dict(ortho_interval=2, pop_interval=4, equilibration_steps=0, measure_interval=2, relax=0.1, steer=True)
    members = [(120, 80, 240, capi.PRECISION_INT8X3), (48, 12, 96, capi.PRECISION_INT8X3),
               (80, 60, 160, capi.PRECISION_FP64), (24, 6, 96, capi.PRECISION_FP64)]

    def engines():
        return [afqmc.AfqmcEngine(synthetic.make_system(synthetic.SystemSpec(M=M, N=N, Nc=Nc, decay=float(M), seed=50 + i)),
                                  6, dt=1e-4, seed=i, precision=p) for i, (M, N, Nc, p) in enumerate(members)]

    grouped, alone = engines(), engines()
    grp = afqmc.EngineGroup(grouped)
    E0 = np.array([e.init() for e in grouped])
    Eg, st, mg = grp.run_block(4, E0, step0=0, **blk)
    assert not st.any()
    for i, e in enumerate(alone):
        e.init()
        Ea, ma = e.run_block(4, E0[i], step0=0, **blk)
        assert Eg[i] == Ea and np.array_equal(mg[i], ma)
        assert np.array_equal(grouped[i].walkers()[0], e.walkers()[0])
