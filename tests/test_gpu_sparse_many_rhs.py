"""Many right-hand sides through the larger fronts' kernels.  A level's CTAs take
16 or 32 right-hand sides once its fronts times the groups reach two for each SM:
with 32 fronts a level (that of this mesh with the most larger fronts) that is
160 right-hand sides for 16 and 320 for 32 on 148 SMs, the last group full or partly
filled.  Triangles in shared memory, and with FEM25_PANEL_WIDTH=1 in x; all three
operators.  Two random combinations of the columns must satisfy
||op(A) X w - B w|| <= 1e-10 ||B w||, the bound of the residual tests on this mesh: a
wrong column shows in both."""
import numpy as np
import pytest

import oracle
from fem25_b200 import Context, synth
from tests import helpers

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def factored():
    mesh, pairs, _ = synth.make_config(1, nx=49, nz=46)
    g = oracle.graph_build(mesh)
    ctx = Context(mesh, g)
    a = torch.zeros(g.nzero, dtype=torch.complex128, device="cuda:0")
    ctx.assemble("B", *pairs[70], a)
    ctx.sparse_factor(a)
    A = helpers.csr_matrix(g, a.cpu().numpy())
    yield ctx, g, (A, A.T.tocsr(), A.conj().T.tocsr())
    ctx.close()


@pytest.mark.parametrize("any_size", [False, True])
@pytest.mark.parametrize("nrhs", [160, 309, 320])
def test_sparse_solve_wide_groups(factored, nrhs, any_size, monkeypatch):
    if any_size:
        monkeypatch.setenv("FEM25_PANEL_WIDTH", "1")
    ctx, g, mats = factored
    gen = torch.Generator(device="cuda:0")
    gen.manual_seed(nrhs)

    def rand(*shape):
        return torch.randn(shape, generator=gen, dtype=torch.complex128, device="cuda:0")

    b, w = rand(nrhs, g.ndof), rand(2, nrhs)
    want = (w @ b).cpu().numpy()
    for trans, mat in enumerate(mats):
        x = b.clone()
        ctx.sparse_solve(x, trans)
        got = (w @ x).cpu().numpy()
        for k in range(2):
            assert np.linalg.norm(mat @ got[k] - want[k]) <= 1e-10 * np.linalg.norm(want[k]), (trans, k)
