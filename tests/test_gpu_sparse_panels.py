"""The factorisation of fronts beyond shared memory (more than 96 own DOFs) at
every sub-panel width it can take (8, 4 and 2 columns in registers, one column
at a time for any size), on a mesh whose largest separator (564 rows) needs two
rows a thread at width 8 and whose fronts end in ragged panels and tiles.
Residual ||op(A) x - b|| / ||b|| <= 1e-10, the bound of the sparse solve's other
residual tests on the layered mesh."""
import numpy as np
import pytest

import oracle
from fem25_b200 import Context, synth
from tests import helpers

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [8, 4, 2, 1])
def test_sparse_factor_panel_widths(width, monkeypatch):
    monkeypatch.setenv("FEM25_PANEL_WIDTH", str(width))
    mesh, pairs, _ = synth.make_config(1, nx=49, nz=46)
    g = oracle.graph_build(mesh)
    ctx = Context(mesh, g)
    f, py = pairs[70]
    a = torch.zeros(g.nzero, dtype=torch.complex128, device="cuda:0")
    ctx.assemble("B", f, py, a)
    ctx.sparse_factor(a)
    assert ctx.sparse_info()[4] > 512
    A = helpers.csr_matrix(g, a.cpu().numpy())
    rng = np.random.default_rng(3)
    b = rng.standard_normal((2, g.ndof)) + 1j * rng.standard_normal((2, g.ndof))
    for trans, mat in ((0, A), (1, A.T.tocsr())):
        x = torch.from_numpy(b).cuda()
        ctx.sparse_solve(x, trans)
        got = x.cpu().numpy()
        for k in range(2):
            assert np.linalg.norm(mat @ got[k] - b[k]) <= 1e-10 * np.linalg.norm(b[k]), (trans, k)
    ctx.close()
