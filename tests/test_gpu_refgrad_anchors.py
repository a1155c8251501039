"""The reference-compatible gradient on either side of one inversion anchor an SM
(148), where a CTA's threads take one node pair each or five: bit-identical to the
oracle's CFMAT_DIST + ADJFLAM_DIST, with and without accumulation over elements."""
import numpy as np
import pytest

import oracle
from fem25_b200 import Context, synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx, nz, few", [(12, 10, True), (18, 14, False)])
def test_reference_gradient_anchor_counts(nx, nz, few):
    mesh, pairs, _ = synth.make_config(0, nx=nx, nz=nz)
    g = oracle.graph_build(mesh)
    ctx, rg = Context(mesh, g), oracle.RefGrad(mesh, g)
    assert (rg.nnpinv <= 148) == few
    rng = np.random.default_rng(nx)
    wave, lam = ((rng.standard_normal(g.ndof) + 1j * rng.standard_normal(g.ndof)).astype(np.complex64)
                 for _ in range(2))
    f, py = pairs[7]
    for cinv, accumulate in (("PP", False), ("SS", True)):
        fm = rg.cfmat(f, py, wave, lisp=(cinv == "PP"), accumulate=accumulate)
        ref = rg.adjflam(fm, lam)
        out = torch.zeros(rg.nnpinv, dtype=torch.float32, device="cuda:0")
        ctx.cfmat_adjgrad(cinv, 1.7320508075688772, f, py, torch.from_numpy(wave).cuda(),
                          torch.from_numpy(lam).cuda(), out, accumulate=accumulate)
        assert np.array_equal(out.cpu().numpy().view(np.uint32), ref.view(np.uint32)), cinv
    ctx.close()
