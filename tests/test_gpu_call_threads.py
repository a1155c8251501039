"""fem25_misfit_dev and fem25_postsolve_dev from several host threads on one
context, each with a stream, receivers and sizes of its own: every output equals
the same call made alone, bit for bit."""
import threading

import numpy as np
import pytest

import oracle
from fem25_b200 import Context, synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SIZES = [(2, 9), (37, 40), (5, 700), (16, 3)]  # sources, receivers of each thread
CALLS = 60


def _field(rng, *shape):
    return (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)


@pytest.mark.parametrize("kind", ["misfit", "postsolve"])
def test_overlapping_calls(kind):
    mesh, _, _ = synth.make_config(4, nx=22, nz=11)
    g = oracle.graph_build(mesh)
    ctx = Context(mesh, g)
    nodes = np.unique(g.lm.reshape(-1, 3), axis=0)
    nodes = nodes[(nodes > 0).all(axis=1)]
    jobs = []
    for k, (nsrc, nrec) in enumerate(SIZES):
        rng = np.random.default_rng(k)
        mrdof = nodes[rng.choice(len(nodes), nrec, replace=False)].astype(np.int32)
        sol, ue = (torch.from_numpy(_field(rng, nsrc, g.ndof)).cuda() for _ in range(2))
        head = (nsrc, mrdof, rng.uniform(-9, 9, nrec), 0.7, 1e-4, 20.0, _field(rng, nrec, 3))
        data = (_field(rng, nsrc, nrec, 3), rng.uniform(0.5, 1.5, (nsrc, nrec, 3)).astype(np.float32))
        jobs.append((head, ue, sol, data, torch.cuda.Stream()))

    def call(job):
        head, ue, sol, data, st = job
        with torch.cuda.stream(st):
            s, rhs = sol.clone(), torch.zeros_like(sol)
            if kind == "misfit":
                est, mis = ctx.misfit(*head, s, *data, rhs, stream=st)
            else:
                est, mis = ctx.postsolve(*head, ue, s, *data, rhs, stream=st)
            return [a.view(np.uint32) for a in (est, mis, s.cpu().numpy(), rhs.cpu().numpy())]

    torch.cuda.synchronize()
    alone = [call(j) for j in jobs]
    bad = []

    def work(k):
        for n in range(CALLS):
            try:
                if not all(np.array_equal(a, b) for a, b in zip(call(jobs[k]), alone[k])):
                    bad.append((k, n))
            except Exception as e:  # noqa: BLE001
                bad.append((k, n, repr(e)))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad[:5]
    ctx.close()
