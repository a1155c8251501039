"""Sparse solve of a mesh in three disconnected parts: its dissection has fronts
without a boundary below the root (beside fronts that have one, in the same
launches) and a root without DOFs of its own; once with separators that fit
shared memory and once with larger ones (more than 96 own DOFs).  All three
operators on a diagonally dominant matrix of the mesh's pattern; residual
||op(A) x - b|| / ||b|| <= 1e-11, the bound of the sparse solve's tests on the
small configuration."""
import dataclasses

import numpy as np
import pytest

import oracle
from fem25_b200 import Context, synth
from tests import helpers

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _parts(sizes):
    meshes, x0, a0 = [], 0.0, 0
    for i, (nx, nz) in enumerate(sizes):
        m = synth.structured_mesh(nx, nz, 500.0 * nx, 500.0 * nz, 2, seed=i)
        synth.halfspace_model(m, i)
        m.ieng, m.xlocs = m.ieng + np.int32(a0), m.xlocs + x0
        x0, a0 = x0 + 500.0 * nx + 5000.0, a0 + m.nnpg
        meshes.append(m)

    def cat(name, axis=0):
        return np.ascontiguousarray(np.concatenate([getattr(m, name) for m in meshes], axis=axis))

    names = ("ieng", "cdomain", "cnnpg", "xlocs", "zlocs", "xd", "zd", "dens")
    return dataclasses.replace(meshes[0], nelem=sum(m.nelem for m in meshes), nnpg=a0,
                               ecoeff=cat("ecoeff", 1), **{n: cat(n) for n in names})


@pytest.mark.parametrize("sizes, largest", [([(12, 8), (6, 8), (6, 8)], 96),
                                            ([(20, 12), (10, 12), (10, 12)], 144)])
def test_sparse_disconnected_parts(sizes, largest):
    mesh = _parts(sizes)
    g = oracle.graph_build(mesh)
    ctx = Context(mesh, g)
    rng = np.random.default_rng(largest)
    a = rng.standard_normal(g.nzero) + 1j * rng.standard_normal(g.nzero)
    row = np.repeat(np.arange(g.ndof), np.diff(g.irptr))
    a[row == g.jcptr - 1] += 2.0 * np.sqrt(np.diff(g.irptr))
    ctx.sparse_factor(torch.from_numpy(a).cuda())
    assert ctx.sparse_info()[4] == largest
    A = helpers.csr_matrix(g, a)
    b = rng.standard_normal((3, g.ndof)) + 1j * rng.standard_normal((3, g.ndof))
    for trans, mat in enumerate((A, A.T.tocsr(), A.conj().T.tocsr())):
        x = torch.from_numpy(b).cuda()
        ctx.sparse_solve(x, trans)
        got = x.cpu().numpy()
        for k in range(3):
            assert np.linalg.norm(mat @ got[k] - b[k]) <= 1e-11 * np.linalg.norm(b[k]), (trans, k)
    ctx.close()
