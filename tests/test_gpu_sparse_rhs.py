"""Right-hand-side groups of the sparse solve: one column, partly filled and
full groups of 8, 16 and 32 columns, more than one group, and NRHS x fronts on
either side of the rule that narrows the groups of levels with few fronts; all
three operators.  Residual ||op(A) x - b|| / ||b|| <= 1e-11, the bound of the
sparse solve's tests on the small configuration."""
import numpy as np
import pytest

import oracle
from fem25_b200 import Context, synth
from tests import helpers

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def factored():
    mesh, pairs, _ = synth.make_config(0)
    g = oracle.graph_build(mesh)
    ctx = Context(mesh, g)
    a = torch.zeros(g.nzero, dtype=torch.complex128, device="cuda:0")
    ctx.assemble("S", *pairs[9], a)
    ctx.sparse_factor(a)
    A = helpers.csr_matrix(g, a.cpu().numpy())
    yield ctx, g, (A, A.T.tocsr(), A.conj().T.tocsr())
    ctx.close()


@pytest.mark.parametrize("nrhs", [1, 3, 8, 9, 16, 17, 32, 41])
def test_sparse_solve_groups(factored, nrhs):
    ctx, g, mats = factored
    rng = np.random.default_rng(nrhs)
    b = rng.standard_normal((nrhs, g.ndof)) + 1j * rng.standard_normal((nrhs, g.ndof))
    for trans, mat in enumerate(mats):
        x = torch.from_numpy(b).cuda()
        ctx.sparse_solve(x, trans)
        got = x.cpu().numpy()
        for k in range(nrhs):
            assert np.linalg.norm(mat @ got[k] - b[k]) <= 1e-11 * np.linalg.norm(b[k]), (trans, k)
