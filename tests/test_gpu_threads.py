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
