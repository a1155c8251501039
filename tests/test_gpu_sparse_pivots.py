"""Pivots of the sparse factorisation.

Choice: beside ones on the diagonal, every node's first two DOFs p < q hold
  [ 1      2^60 ]
  [ 1 + d  1    ]
whose partial pivoting must take row q.  Then x_p = (b_q - x_q) / (1 + d) loses
nothing; with row p as the pivot x_p is b_p - 2^60 x_q and wrong by about 2^7.  For
|x| < 2 the right order leaves a handful of roundings of numbers below 5, so 2e-14
bounds the error.  d from 2^-12 to 2^-40, in fronts of every kernel of the
factorisation (the small ones, and the larger ones at each sub-panel width).

Range: powers of two scale the matrix and the right-hand side until the squares of
the entries under- or overflow, where 1 / pivot is still a normal number.  Scaling by a
power of two is exact, so only the order of the solve's sums differs from the unscaled
solution: 1e-9 relative leaves two orders above the known-field errors of such meshes."""
import numpy as np
import pytest

import oracle
from fem25_b200 import Context, synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def case():
    mesh, pairs, _ = synth.make_config(1, nx=49, nz=46)
    g = oracle.graph_build(mesh)
    ctx = Context(mesh, g)
    yield ctx, g, pairs
    ctx.close()


@pytest.mark.parametrize("bits", [12, 40])
@pytest.mark.parametrize("width", [8, 4, 2, 1])
def test_pivot_choice(case, width, bits, monkeypatch):
    monkeypatch.setenv("FEM25_PANEL_WIDTH", str(width))
    ctx, g, _ = case
    row = np.repeat(np.arange(g.ndof), np.diff(g.irptr))
    col = g.jcptr - 1
    nodes = np.unique(np.asarray(g.lm).reshape(-1, 3), axis=0) - 1
    nodes = nodes[(nodes >= 0).all(axis=1)]
    p, q = nodes[:, 0], nodes[:, 1]
    assert (p < q).all()
    a = (row == col).astype(np.complex128)
    key = row.astype(np.int64) * g.ndof + col
    a[np.searchsorted(key, p.astype(np.int64) * g.ndof + q)] = 2.0 ** 60
    a[np.searchsorted(key, q.astype(np.int64) * g.ndof + p)] = 1.0 + 2.0 ** -bits
    rng = np.random.default_rng(bits)
    x = rng.uniform(0.5, 1.4, g.ndof) + 1j * rng.uniform(0.5, 1.4, g.ndof)
    b = x.copy()
    b[p] = x[p] + 2.0 ** 60 * x[q]
    b[q] = (1.0 + 2.0 ** -bits) * x[p] + x[q]
    ctx.sparse_factor(torch.from_numpy(a).cuda())
    d = torch.from_numpy(b[None]).cuda()
    ctx.sparse_solve(d, 0)
    assert np.abs(d.cpu().numpy()[0] - x).max() <= 2e-14


@pytest.mark.parametrize("exponent", [-560, -520, 520])
@pytest.mark.parametrize("width", [8, 1])
def test_pivot_range(case, width, exponent, monkeypatch):
    monkeypatch.setenv("FEM25_PANEL_WIDTH", str(width))
    ctx, g, pairs = case
    a = torch.zeros(g.nzero, dtype=torch.complex128, device="cuda:0")
    ctx.assemble("B", *pairs[70], a)
    rng = np.random.default_rng(5)
    b = torch.from_numpy(rng.standard_normal((1, g.ndof)) + 1j * rng.standard_normal((1, g.ndof))).cuda()
    scale = 2.0 ** (exponent - int(np.log2(float(a.abs().max()))))  # exponent: of the largest entry
    want, got = b.clone(), b * scale
    ctx.sparse_factor(a)
    ctx.sparse_solve(want, 0)
    ctx.sparse_factor(a * scale)
    ctx.sparse_solve(got, 0)
    assert float(torch.linalg.norm(got - want) / torch.linalg.norm(want)) <= 1e-9
