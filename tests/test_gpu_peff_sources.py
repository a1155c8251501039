"""P_eff for source counts around the kernel's lane groups (32 sources a lane
slot, 64 a pass), bit-identical to the oracle's ASMB_PEFF: on a 4-element strip,
whose rows reach the DOF classes on both sides, with NDOF not a multiple of 32;
and the post-solve pass with the context's call buffer grown and reused between
calls of different sizes (compared with one call per source)."""
import numpy as np
import pytest

import oracle
from fem25_b200 import Context, synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def case():
    mesh, pairs, _ = synth.make_config(4, nx=22, nz=11)
    g = oracle.graph_build(mesh)
    ctx = Context(mesh, g)
    assert g.ndof % 32 != 0
    yield mesh, pairs, g, ctx
    ctx.close()


def _field(rng, *shape):
    return (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)


@pytest.mark.parametrize("nsrc", [1, 31, 33, 64, 65, 130])
def test_peff_source_groups(case, nsrc):
    mesh, pairs, g, ctx = case
    rng = np.random.default_rng(nsrc)
    ue = _field(rng, nsrc, g.ndof)
    a = torch.zeros(g.nzero, dtype=torch.complex64, device="cuda:0")
    ctx.assemble("B", *pairs[40], None, a)
    p = torch.full((nsrc, g.ndof), float("nan"), dtype=torch.complex64, device="cuda:0")
    ctx.asmb_peff(nsrc, a, torch.from_numpy(ue).cuda(), p)
    got, ah = p.cpu().numpy(), a.cpu().numpy()
    for s in range(nsrc):
        ref = oracle.peff(g, ah, ue[s])
        assert np.array_equal(got[s].view(np.uint32), ref.view(np.uint32)), s


@pytest.mark.parametrize("nsrc, reps", [(3, 1), (18, 14000), (5, 2)])
def test_postsolve_call_buffer(case, nsrc, reps):
    """reps receivers at MRDOF 0 (outside the mesh) beside nine inside it."""
    mesh, pairs, g, ctx = case
    rng = np.random.default_rng(reps)
    nodes = np.unique(g.lm.reshape(-1, 3), axis=0)
    nodes = nodes[(nodes > 0).all(axis=1)]
    mrdof = nodes[rng.choice(len(nodes), 9, replace=False)]
    mrdof = np.concatenate([mrdof, np.zeros((reps, 3), np.int32)]).astype(np.int32)
    nr = len(mrdof)
    sol, ue, obs = _field(rng, nsrc, g.ndof), _field(rng, nsrc, g.ndof), _field(rng, nsrc, nr, 3)
    w = rng.uniform(0.5, 1.5, (nsrc, nr, 3)).astype(np.float32)
    yrec, recv = rng.uniform(-9, 9, nr), _field(rng, nr, 3)
    d_ue = torch.from_numpy(ue).cuda()
    s2 = torch.from_numpy(sol).cuda()
    r2 = torch.zeros((nsrc, g.ndof), dtype=torch.complex64, device="cuda:0")
    e2, m2 = ctx.postsolve(nsrc, mrdof, yrec, 0.7, 1e-4, 20.0, recv, d_ue, s2, obs, w, r2)
    for s in (0, nsrc - 1):
        s1 = torch.from_numpy(sol[s:s + 1]).cuda()
        r1 = torch.zeros((1, g.ndof), dtype=torch.complex64, device="cuda:0")
        e1, m1 = ctx.postsolve(1, mrdof, yrec, 0.7, 1e-4, 20.0, recv, d_ue[s:s + 1].contiguous(), s1,
                               obs[s:s + 1], w[s:s + 1], r1)
        assert np.array_equal(e1[0].view(np.uint32), e2[s].view(np.uint32))
        assert np.array_equal(m1[:1].view(np.uint32), m2[s:s + 1].view(np.uint32))
        assert torch.equal(torch.view_as_real(s1[0]), torch.view_as_real(s2[s]))
        assert torch.equal(torch.view_as_real(r1[0]), torch.view_as_real(r2[s]))
