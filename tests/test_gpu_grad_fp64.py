"""The FP64 gradient's two-step interpolation (rows of 5 nodes along xi, then
even and odd parts along eta) at the edges of its field tiles: one field, a
full tile of two, ragged tiles within and across (omega, py) pairs, more than
one launch of 64 pairs, on skewed elements with topography.  Against the
oracle's point-by-point gradient, 2-norm relative per parameter: both evaluate
the same FP64 forms in another summation order, so 1e-11 leaves four orders
over the rounding of sums of a few thousand terms."""
import numpy as np
import pytest

import oracle
from fem25_b200 import FEM25_PREC_FP64, Context, synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npairs, nsrc", [(1, 1), (1, 2), (3, 1), (2, 5), (67, 1)])
def test_gradient_fp64_field_tiles(npairs, nsrc):
    mesh, pairs, _ = synth.make_config(4, nx=12, nz=9)
    g = oracle.graph_build(mesh)
    ctx = Context(mesh, g)
    rng = np.random.default_rng(5 + npairs)
    use = [pairs[(7 * k) % len(pairs)] for k in range(npairs)]
    shape = (npairs, nsrc, g.ndof)
    u = rng.standard_normal(shape) + 1j * rng.standard_normal(shape)
    lam = rng.standard_normal(shape) + 1j * rng.standard_normal(shape)
    ref = np.zeros((3, mesh.nnpg))
    for p, (f, py) in enumerate(use):
        oracle.grad_exact(mesh, g, f, py, u[p], lam[p], out=ref)
    got = torch.zeros((3, mesh.nnpg), dtype=torch.float64, device="cuda:0")
    ctx.gradient([p[0] for p in use], [p[1] for p in use], nsrc, torch.from_numpy(u).cuda(),
                 torch.from_numpy(lam).cuda(), got, FEM25_PREC_FP64)
    ctx.sync_status()
    got = got.cpu().numpy()
    for m in range(3):
        assert np.linalg.norm(got[m] - ref[m]) <= 1e-11 * np.linalg.norm(ref[m]), m
    ctx.close()
