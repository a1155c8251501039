"""Workloads of the fem25 hot path, as an inversion program runs them.

One iteration of such a program assembles the (omega, py) systems of its mesh
(one at a time into device or host buffers, or a batch into a ring of device
slots), factors and solves them for its sources and for the adjoint sources,
forms the effective forces and the misfit around the solves, and reduces the
forward and adjoint fields into the model gradient.  Every case below is one
of these calls through ``fem25_b200.Context`` on a mesh of the sizes of the
package's configurations: the 40 x 20 half-space-sized mesh, the layered mesh
at 500 m elements, and the 300 x 150 jittered mesh.

    listed()            the cases
    draw(rng)           another case of the same ranges
    prepare(case, seed) the context, fields and buffers such a program holds
    run(state)          one call, and its outputs
    work(case)          bytes and operations the call cannot do without
    exact(case, seed)   the same outputs by dense torch arithmetic in 64 bits
"""
from __future__ import annotations

import dataclasses
import functools
import math

import numpy as np
import torch

from fem25_b200 import Context, synth
from fem25_b200.lib import (FEM25_PREC_FP64, FEM25_PREC_TF32X3, FEM25_PREC_TF32X3_POINTWISE,
                            graph_build, sparse_plan)

DEV = "cuda:0"
PREC = {"fp64": FEM25_PREC_FP64, "tf32x3": FEM25_PREC_TF32X3,
        "pointwise": FEM25_PREC_TF32X3_POINTWISE}
TWOPI = 6.2831853071795862


def _case(kind, nx, nz, jitter=0.0, strip=2, freq=0.8, cftype="B", **more):
    return dict(kind=kind, nx=nx, nz=nz, jitter=jitter, strip=strip, freq=freq, cftype=cftype,
                **more)


def listed():
    return [
        # one system of the small configuration into device buffers, FP64 and COMPLEX*8:
        # launch latency and a nearly empty GPU
        dict(_case("assemble", 40, 20, freq=0.5), name="assemble 40x20"),
        # the same call on an ordinary mesh: one system per (omega, py) before each solve
        dict(_case("assemble", 200, 60, cftype="S"), name="assemble 200x60"),
        # the 16 wavenumbers of the small configuration in one batched call
        dict(_case("batch", 40, 20, freq=0.5, nfreq=1, nky=16, nslots=16), name="batch 40x20"),
        # several frequencies and wavenumbers through a ring of slots that a solver drains
        dict(_case("batch", 200, 60, nfreq=4, nky=8, nslots=8), name="batch 200x60"),
        # the Fortran driver's call: model upload, then CDIST into pinned host memory
        dict(_case("driver", 100, 40), name="driver 100x40"),
        # exact gradient in FP64: 32 sources of two systems
        dict(_case("gradient", 200, 60, prec="fp64", npairs=2, nsrc=32), name="gradient fp64"),
        # the default split-precision gradient on a large unstructured mesh
        dict(_case("gradient", 300, 150, jitter=0.2, prec="tf32x3", npairs=2, nsrc=64),
             name="gradient tf32x3"),
        # the pointwise split-precision gradient, one source at every wavenumber of the
        # small configuration
        dict(_case("gradient", 40, 20, freq=0.5, prec="pointwise", npairs=16, nsrc=1),
             name="gradient pointwise"),
        # a new system factored and solved for its first source
        dict(_case("factor", 200, 60, trans=0), name="factor 200x60"),
        # the adjoint solves of a group of sources with kept factors
        dict(_case("solve", 200, 60, nrhs=32, trans=2), name="solve 200x60"),
        # effective forces before and misfit / adjoint sources after the solves
        dict(_case("sources", 200, 60, strip=4, nsrc=64, nrec=190), name="sources 200x60"),
        # the reference-compatible gradient of one source (CFMAT_DIST + ADJGRAD)
        dict(_case("refgrad", 200, 60, cinvtype="PP"), name="refgrad 200x60"),
    ]


def draw(rng):
    kind = rng.choice(["assemble", "assemble", "batch", "driver", "gradient", "gradient",
                       "gradient", "factor", "solve", "solve", "sources", "refgrad"])
    prec = rng.choice(["fp64", "tf32x3", "pointwise"])
    top = {"driver": 4000, "gradient": 45000 if prec == "tf32x3" else 12000}.get(kind, 12000)
    nelem = math.exp(rng.uniform(math.log(300), math.log(top)))
    aspect = rng.uniform(1.5, 3.4)
    strip = rng.choice([2, 2, 4])
    nx = max(12, int(math.sqrt(nelem * aspect)))
    nz = max(10, int(nelem / nx))
    case = _case(kind, nx, nz, jitter=rng.choice([0.0, 0.2]), strip=strip,
                 freq=round(rng.uniform(0.3, 1.6), 3), cftype=rng.choice("SB"))
    ne = nx * nz

    def count(most, budget):
        return int(math.exp(rng.uniform(0.0, math.log(max(1, min(most, budget // ne)) + 0.9))))

    if kind == "batch":
        case["nfreq"] = rng.choice([1, 2, 3, 4])
        case["nky"] = count(32 // case["nfreq"], 32 * 12000 // case["nfreq"])
        case["nslots"] = rng.choice([1, 3, 8, 16]) if ne < 6000 else rng.choice([1, 3, 8])
    elif kind == "gradient":
        case["prec"] = prec
        case["npairs"] = rng.choice([1, 2, 3, 4])
        fields = {"fp64": 64 * 12000, "tf32x3": 128 * 45000, "pointwise": 64 * 12000}[prec]
        case["nsrc"] = count(64, fields // case["npairs"])
    elif kind == "factor":
        case["trans"] = rng.choice([0, 1, 2])
    elif kind == "solve":
        case["nrhs"] = count(32, 32 * 12000)
        case["trans"] = rng.choice([0, 1, 2])
    elif kind == "sources":
        case["nsrc"] = count(64, 64 * 12000)
        case["nrec"] = rng.randint(3, nx - 2)
    elif kind == "refgrad":
        case["cinvtype"] = rng.choice(["PP", "SS"])
    return case


# ---------------------------------------------------------------------------
# what a program holds before the call
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=2)
def _grid(nx, nz, strip, jitter):
    """The mesh geometry, its graph and the DOF coordinates: read or built once
    by a program and kept over its whole run."""
    mesh = synth.structured_mesh(nx, nz, 500.0 * nx, 500.0 * nz, strip, seed=nx + nz, jitter=jitter,
                                 topo_amp=200.0 if jitter else 0.0)
    g = graph_build(mesh)
    x, z = synth.dof_coords(mesh, g)
    return mesh, g, x, z


def _with_model(mesh, seed):
    m = dataclasses.replace(mesh)
    synth.layered_model(m, seed)
    return m


def _mesh(case, seed):
    mesh, g, x, z = _grid(case["nx"], case["nz"], case["strip"], case["jitter"])
    return _with_model(mesh, seed), g, x, z


def _gen(seed):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    return gen


def _systems(case, mesh, nfreq, nky):
    """(freq, py) of nfreq frequencies up to the case's, nky wavenumbers each."""
    out = []
    for k in range(nfreq):
        f = case["freq"] * (k + 1) / nfreq
        out += [(f, float(py)) for py in synth.ky_list(f, nky + 1, synth.vs_min(mesh))[1:]]
    return out


def _fields(x, z, freqs, nsrc, gen, dtype=torch.complex128):
    """Waves of each frequency over the mesh, [len(freqs), nsrc, NDOF]: a plane
    wave with a smooth random phase and a lognormal amplitude, unit RMS."""
    xt, zt = torch.from_numpy(x).to(DEV), torch.from_numpy(z).to(DEV)
    out = torch.empty((len(freqs), nsrc, x.size), dtype=dtype, device=DEV)
    real = dict(generator=gen, dtype=torch.float64, device=DEV)
    for p, f in enumerate(freqs):
        k0 = TWOPI * f / 2500.0
        for s in range(nsrc):
            r = torch.randn(6, 2, **real) / 5000.0
            b = torch.rand(6, **real) * TWOPI
            phase = k0 * xt
            for m in range(6):
                phase = phase + torch.cos(r[m, 0] * xt + r[m, 1] * zt + b[m]) / math.sqrt(3.0)
            amp = torch.exp(0.1 * torch.randn(x.size, **real))
            amp /= torch.sqrt(torch.mean(amp * amp))
            out[p, s] = torch.polar(amp, phase)
    return out


def _receivers(mesh, g, nrec):
    """MRDOF [nrec, 3] of free-surface nodes, evenly spaced along the surface."""
    nl = mesh.nord + 1
    fs = (mesh.cnnpg == np.frombuffer(b"FS", np.uint8)).all(axis=1)
    el = np.nonzero(fs[mesh.ieng[:, 2] - 1] & fs[mesh.ieng[:, 3] - 1])[0]
    nodes = g.lm[el, nl * (nl - 1)]
    nodes = nodes[(nodes > 0).all(axis=1)]
    return np.ascontiguousarray(nodes[np.linspace(0, len(nodes) - 1, nrec).astype(int)], np.int32)


def _csr(ctx, case, py, out64=False):
    a = torch.empty(ctx.nzero, dtype=torch.complex64 if out64 else torch.complex128, device=DEV)
    ctx.assemble(case["cftype"], case["freq"], py, None if out64 else a, a if out64 else None)
    return a


def _apply(g, a, x, trans):
    """op(A) x for x [n, NDOF]; the pattern of A is symmetric."""
    crow = torch.from_numpy(g.irptr - 1).to(DEV)
    col = torch.from_numpy(g.jcptr - 1).to(DEV)
    if trans:
        row = torch.repeat_interleave(torch.arange(g.ndof, device=DEV), (crow[1:] - crow[:-1]).long())
        a = a[torch.argsort(col.long() * g.ndof + row)]
        a = a.conj().resolve_conj() if trans == 2 else a
    m = torch.sparse_csr_tensor(crow, col, a, size=(g.ndof, g.ndof))
    return (m @ x.t().contiguous()).t().contiguous()


def prepare(case, seed):
    kind = case["kind"]
    mesh, g, x, z = _mesh(case, seed)
    ctx = Context(mesh, g)
    gen = _gen(seed)
    st = dict(case=case, ctx=ctx, mesh=mesh)
    vmin = synth.vs_min(mesh)
    py = 0.4 / vmin
    if kind == "assemble":
        st.update(py=py, a128=torch.empty(g.nzero, dtype=torch.complex128, device=DEV),
                  a64=torch.empty(g.nzero, dtype=torch.complex64, device=DEV))
    elif kind == "batch":
        sys = _systems(case, mesh, case["nfreq"], case["nky"])
        stride = (2 * g.nzero + 15) // 16 * 16
        slots = min(case["nslots"], len(sys))
        st.update(freqs=[s[0] for s in sys], pys=[s[1] for s in sys], stride=stride, slots=slots,
                  ring=torch.zeros((slots, stride), dtype=torch.float64, device=DEV))
    elif kind == "driver":
        st.update(py=py, cdist=torch.empty(g.nzero, dtype=torch.complex64, pin_memory=True))
    elif kind == "gradient":
        sys = _systems(case, mesh, 1, case["npairs"])
        freqs = [s[0] for s in sys]
        st.update(freqs=freqs, pys=[s[1] for s in sys], u=_fields(x, z, freqs, case["nsrc"], gen),
                  lam=_fields(x, z, freqs, case["nsrc"], gen),
                  grad=torch.zeros((3, mesh.nnpg), dtype=torch.float64, device=DEV))
    elif kind in ("factor", "solve"):
        a = _csr(ctx, case, py)
        nrhs = case.get("nrhs", 1)
        b = _apply(g, a, _fields(x, z, [case["freq"]], nrhs, gen)[0], case["trans"])
        st.update(a=a, b=b, x=torch.empty_like(b))
        if kind == "solve":
            ctx.sparse_factor(a)
    elif kind == "sources":
        st.update(py=py, a=_csr(ctx, case, py, out64=True), **_source_data(case, seed, mesh, g, x, z, gen))
        st.update(peff=torch.empty_like(st["ue"]), sol=torch.empty_like(st["ue"]),
                  rhs=torch.empty_like(st["ue"]))
    else:
        w = _fields(x, z, [case["freq"]] * 2, 1, gen, torch.complex64)
        st.update(py=py, wave=w[0, 0].contiguous(), adj=w[1, 0].contiguous(),
                  gradl=torch.zeros(ctx.ref_gradient_info()[0], dtype=torch.float32, device=DEV))
    return st


def _source_data(case, seed, mesh, g, x, z, gen):
    """Background fields, solutions and the data of a group of sources."""
    nsrc = case["nsrc"]
    mrdof = _receivers(mesh, g, case["nrec"])
    nrec = len(mrdof)
    ue = _fields(x, z, [case["freq"]], nsrc, gen, torch.complex64)[0]
    sol0 = _fields(x, z, [case["freq"]], nsrc, gen, torch.complex64)[0]
    rng = np.random.default_rng(seed)

    def wave(shape):
        return (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)

    return dict(ue=ue, sol0=sol0, mrdof=mrdof, yrec=rng.uniform(-900.0, 900.0, nrec),
                recv=(1.0 + 0.1 * wave((nrec, 3))).astype(np.complex64), obs=wave((nsrc, nrec, 3)),
                wghts=rng.uniform(0.5, 1.5, (nsrc, nrec, 3)).astype(np.float32))


AZMOD = 30.0
VPVS = 1.73


def run(st):
    case, ctx = st["case"], st["ctx"]
    kind = case["kind"]
    if kind == "assemble":
        ctx.assemble(case["cftype"], case["freq"], st["py"], st["a128"], st["a64"])
        return {"csr128": st["a128"], "csr64": st["a64"]}
    if kind == "batch":
        ctx.assemble_batch(case["cftype"], st["freqs"], st["pys"], st["ring"], st["stride"], st["slots"])
        return st["ring"]
    if kind == "driver":
        ctx.update_model(st["mesh"].ecoeff, st["mesh"].dens)
        ctx.asmble_driver(case["cftype"], case["freq"], st["py"], out=st["cdist"])
        return st["cdist"]
    if kind == "gradient":
        st["grad"].zero_()
        ctx.gradient(st["freqs"], st["pys"], case["nsrc"], st["u"], st["lam"], st["grad"],
                     PREC[case["prec"]])
        return st["grad"]
    if kind in ("factor", "solve"):
        if kind == "factor":
            ctx.sparse_factor(st["a"])
        st["x"].copy_(st["b"])
        ctx.sparse_solve(st["x"], case["trans"])
        return st["x"]
    if kind == "sources":
        ctx.asmb_peff(case["nsrc"], st["a"], st["ue"], st["peff"])
        st["sol"].copy_(st["sol0"])
        est, misfit = ctx.postsolve(case["nsrc"], st["mrdof"], st["yrec"], case["freq"], st["py"],
                                    AZMOD, st["recv"], st["ue"], st["sol"], st["obs"], st["wghts"],
                                    st["rhs"])
        return {"peff": st["peff"], "sol": st["sol"], "est": est, "rhs": st["rhs"], "misfit": misfit}
    st["gradl"].zero_()
    ctx.cfmat_adjgrad(case["cinvtype"], VPVS, case["freq"], st["py"], st["wave"], st["adj"], st["gradl"])
    return st["gradl"]


def work(case):
    """Sizes before the Dirichlet rows are removed: (4 nx + 1)(4 nz + 1) nodes of
    three DOFs, 9 (24 nx + 1)(24 nz + 1) nonzeros."""
    nx, nz, kind = case["nx"], case["nz"], case["kind"]
    ne, ndof = nx * nz, 3 * (4 * nx + 1) * (4 * nz + 1)
    nnz = 9 * (24 * nx + 1) * (24 * nz + 1)
    # the twelve affine parts of one element matrix by sum factorisation over the 13 x 13 points
    # (element values to points: 2 stages, products of two shape functions back: 2 stages)
    quad = ne * 12 * 2 * (13 * 13 * 5 * 5 + 13 * 5 ** 4)
    if kind == "assemble":
        return {"bytes": 24 * nnz, "flops": quad + 8 * nnz}
    if kind == "batch":
        n = case["nfreq"] * case["nky"]
        return {"bytes": 16 * nnz * min(n, case["nslots"]) + 12 * nnz, "flops": 6 * nnz * n}
    if kind == "driver":
        return {"bytes": 8 * nnz, "flops": quad + 8 * nnz}
    if kind == "gradient":
        n = case["npairs"] * case["nsrc"]
        # both fields read once; 12 real nodal vectors to values and two derivatives at the points
        # by sum factorisation, and about 90 operations at a point
        return {"bytes": 32 * ndof * n, "flops": ne * n * (12 * 2 * (2 * 5 * 13 * 5 + 3 * 13 * 13 * 5) + 90 * 169)}
    if kind in ("factor", "solve"):
        mesh, _, _, _ = _grid(nx, nz, case["strip"], case["jitter"])
        plan = sparse_plan(_with_model(mesh, 0))
        nrhs = case.get("nrhs", 1)
        if kind == "factor":
            return {"bytes": 16 * nnz + 2 * plan[2], "flops": plan[6] + plan[2] / 2}
        return {"bytes": plan[2] + 32 * ndof * nrhs, "flops": plan[2] / 2 * nrhs}
    if kind == "sources":
        return {"bytes": 5 * 8 * ndof * case["nsrc"], "flops": 4 * ndof * case["nsrc"]}
    return {"bytes": 16 * ndof, "flops": quad}


# ---------------------------------------------------------------------------
# the outputs by plain arithmetic in 64 bits
# ---------------------------------------------------------------------------
def _rule(n):
    """Lobatto points and weights on [-1, 1]."""
    p = np.polynomial.legendre.Legendre.basis(n - 1)
    x = np.concatenate([[-1.0], np.sort(p.deriv().roots().real), [1.0]])
    for _ in range(3):
        x[1:-1] -= p.deriv()(x[1:-1]) / p.deriv(2)(x[1:-1])
    return x, 2.0 / (n * (n - 1) * p(x) ** 2)


def _tables():
    """Shape functions of the 25 nodes and the 4 anchors at the 13 x 13 points:
    (N, dN/dxi, dN/deta), (S, dS/dxi, dS/deta) as [169, 25] and [169, 4], and the weights."""
    xq, w = _rule(13)
    node = np.array([-1.0, -math.sqrt(3.0 / 7.0), 0.0, math.sqrt(3.0 / 7.0), 1.0])
    l, d = np.ones((13, 5)), np.zeros((13, 5))
    for i in range(5):
        p = np.poly1d(np.poly(np.delete(node, i)) / np.prod(node[i] - np.delete(node, i)))
        l[:, i], d[:, i] = p(xq), p.deriv()(xq)
    xi, eta = np.tile(xq, 13), np.repeat(xq, 13)  # point q = ix + 13 iz

    def pair(a, b):  # node ix + 5 iz
        return np.einsum("zj,xi->zxji", b, a).reshape(169, 25)

    sx, se = np.array([-1, 1, 1, -1.0]), np.array([-1, -1, 1, 1.0])
    s = 0.25 * (1 + xi[:, None] * sx) * (1 + eta[:, None] * se)
    s1 = 0.25 * sx * (1 + eta[:, None] * se)
    s2 = 0.25 * se * (1 + xi[:, None] * sx)
    t = [pair(l, l), pair(d, l), pair(l, d), s, s1, s2, np.outer(w, w).reshape(-1)]
    return [torch.from_numpy(np.ascontiguousarray(v)).to(DEV) for v in t]


def _points(mesh, el, tabs):
    """Geometry and model of elements ``el`` at the points: dN/dx, dN/dz [e, 169, 25], the
    weights times the Jacobian, and the interpolation of an anchor array."""
    n, n1, n2, s, s1, s2, w = tabs
    ia = torch.from_numpy(mesh.ieng[el].astype(np.int64) - 1).to(DEV)

    def anchor(a):
        return torch.from_numpy(np.ascontiguousarray(a)).to(DEV)[ia]

    x, z = anchor(mesh.xlocs), anchor(mesh.zlocs)
    xx, xe, zx, ze = x @ s1.T, x @ s2.T, z @ s1.T, z @ s2.T
    jac = xx * ze - xe * zx
    nx = (ze / jac)[..., None] * n1 - (zx / jac)[..., None] * n2
    nz = (xx / jac)[..., None] * n2 - (xe / jac)[..., None] * n1
    return nx, nz, w * jac, lambda a: anchor(a) @ s.T, anchor


def _stretch(mesh, depth, vel, width, omega, cftype):
    k = 0 if cftype == "S" else 1
    dmax = mesh.dmax[k] if mesh.dmax[k] > 0 else -1.5 * vel * math.log(mesh.rcoeff[k]) / width
    prof = torch.abs(dmax * (depth / width) ** 2)
    alpha = math.pi * mesh.fcent[k] * (1.0 - depth / width)
    e = 1.0 / (mesh.kappa[k] + prof / torch.complex(alpha, torch.full_like(alpha, omega)))
    return torch.where(depth > 2.22e-16, e, torch.ones_like(e))


def _exact_csr(case, seed, systems):
    """The CSR values of each (freq, py) system, complex128."""
    mesh, g, _, _ = _mesh(case, seed)
    tabs = _tables()
    n = tabs[0].to(torch.complex128)
    key = torch.from_numpy(np.repeat(np.arange(g.ndof, dtype=np.int64), np.diff(g.irptr)) * g.ndof).to(DEV)
    key += torch.from_numpy(g.jcptr).to(DEV) - 1
    out = [torch.zeros((g.nzero, 2), dtype=torch.float64, device=DEV) for _ in systems]
    for e0 in range(0, mesh.nelem, 2000):
        el = np.arange(e0, min(mesh.nelem, e0 + 2000))
        nx, nz, wj, at, anchor = _points(mesh, el, tabs)
        lam, mu, rho = (at(a) * wj for a in (mesh.ecoeff[0], mesh.ecoeff[1], mesh.dens))
        xd, zd = at(mesh.xd), at(mesh.zd)
        pml = torch.from_numpy(mesh.cdomain[el] == ord("A")).to(DEV)[:, None]
        vel = torch.sqrt((anchor(mesh.ecoeff[0]) + 2 * anchor(mesh.ecoeff[1])) / anchor(mesh.dens)) @ tabs[3].T
        lm = torch.from_numpy(g.lm[el].reshape(len(el), 75).astype(np.int64) - 1).to(DEV)
        ok = (lm[:, :, None] >= 0) & (lm[:, None, :] >= 0)
        where = torch.searchsorted(key, (lm[:, :, None] * g.ndof + lm[:, None, :])[ok])
        for o, (freq, py) in zip(out, systems):
            omega = TWOPI * freq
            one = torch.ones_like(xd, dtype=torch.complex128)
            ex = torch.where(pml, _stretch(mesh, xd, vel, mesh.xwidth, omega, case["cftype"]), one)
            ez = torch.where(pml, _stretch(mesh, zd, vel, mesh.zwidth, omega, case["cftype"]), one)
            bx, bz = nx * ex[..., None], nz * ez[..., None]

            def block(a, c, b):
                return (a * c[..., None]).transpose(1, 2) @ b

            nb = n.expand(len(el), 169, 25)
            wpy = omega * py
            m = torch.zeros((len(el), 25, 3, 25, 3), dtype=torch.complex128, device=DEV)
            xxm, zzm = block(bx, mu, bx), block(bz, mu, bz)
            xzl, xzm = block(bx, lam, bz), block(bx, mu, bz)
            mass = block(nb, wpy ** 2 * mu - omega ** 2 * rho, nb)
            c11 = lam + 2 * mu
            m[:, :, 0, :, 0] = block(bx, c11, bx) + zzm + mass
            m[:, :, 2, :, 2] = block(bz, c11, bz) + xxm + mass
            m[:, :, 1, :, 1] = xxm + zzm + block(nb, wpy ** 2 * c11 - omega ** 2 * rho, nb)
            m[:, :, 0, :, 2] = xzl + xzm.transpose(1, 2)
            m[:, :, 2, :, 0] = xzl.transpose(1, 2) + xzm
            for c, d in ((0, bx), (2, bz)):
                dl, dm = block(d, lam, nb), block(d, mu, nb)
                m[:, :, c, :, 1] = -1j * wpy * (dl - dm.transpose(1, 2))
                m[:, :, 1, :, c] = 1j * wpy * (dl.transpose(1, 2) - dm)
            o.index_add_(0, where, torch.view_as_real(m.reshape(len(el), 75, 75)[ok]))
    return [torch.view_as_complex(o) for o in out]


def _exact_gradient(case, seed):
    mesh, g, x, z = _mesh(case, seed)
    sys = _systems(case, mesh, 1, case["npairs"])
    gen = _gen(seed)
    u = _fields(x, z, [s[0] for s in sys], case["nsrc"], gen)
    v = _fields(x, z, [s[0] for s in sys], case["nsrc"], gen)
    tabs = _tables()
    n = tabs[0].to(torch.complex128)
    grad = torch.zeros((3, mesh.nnpg), dtype=torch.float64, device=DEV)
    elems = np.nonzero(mesh.cdomain != ord("A"))[0]
    step = max(16, 20000 // case["nsrc"])
    for e0 in range(0, len(elems), step):
        el = elems[e0:e0 + step]
        nx, nz, wj, _, _ = _points(mesh, el, tabs)
        nx, nz = nx.to(torch.complex128), nz.to(torch.complex128)
        lm = torch.from_numpy(g.lm[el].astype(np.int64) - 1).to(DEV)
        acc = torch.zeros((3, len(el), 169), dtype=torch.float64, device=DEV)
        for p, (freq, py) in enumerate(sys):
            omega, iw = TWOPI * freq, 1j * TWOPI * freq * py
            parts = []
            for f in (u, v):
                # [source, element, node] of each component, then the points
                c = [torch.where(lm[..., k] >= 0, f[p][:, lm[..., k].clamp(min=0)], 0.0).permute(1, 2, 0)
                     for k in range(3)]
                val, dx, dz = ([t @ a for a in c] for t in (n, nx, nz))
                parts.append((val, [dx[0] + dz[2] - iw * val[1]],
                              [math.sqrt(2.0) * dx[0], math.sqrt(2.0) * dz[2],
                               math.sqrt(2.0) * iw * val[1], dz[0] + dx[2], dx[1] - iw * val[0],
                               dz[1] - iw * val[2]]))
            for m, k in ((0, 1), (1, 2), (2, 0)):
                t = sum((b.conj() * a).real.sum(-1) for a, b in zip(parts[0][k], parts[1][k]))
                acc[m] += t if m < 2 else -omega ** 2 * t
        ia = torch.from_numpy(mesh.ieng[el].astype(np.int64) - 1).to(DEV)
        for m in range(3):
            grad[m].index_add_(0, ia.reshape(-1), ((acc[m] * wj) @ tabs[3]).reshape(-1))
    return grad


def _exact_sources(case, seed):
    mesh, g, x, z = _mesh(case, seed)
    py = 0.4 / synth.vs_min(mesh)
    d = _source_data(case, seed, mesh, g, x, z, _gen(seed))
    ctx = Context(mesh, g)
    a = _csr(ctx, case, py, out64=True)  # an input: the assembled operator
    cnp = torch.from_numpy(g.cnp).to(DEV)
    crow = torch.from_numpy(g.irptr - 1).to(DEV).long()
    row = torch.repeat_interleave(torch.arange(g.ndof, device=DEV), crow[1:] - crow[:-1])
    col = torch.from_numpy(g.jcptr).to(DEV).long() - 1
    sign = ((cnp[row] == ord("E")) & (cnp[col] == ord("B"))).double() \
        - ((cnp[row] == ord("B")) & (cnp[col] == ord("E"))).double()
    k = torch.nonzero(sign)[:, 0]
    ak, row, col = a[k].to(torch.complex128) * sign[k], row[k], col[k]
    ue = d["ue"].to(torch.complex128)
    peff = torch.zeros_like(ue)
    for s in range(case["nsrc"]):
        peff[s].index_add_(0, row, ak * ue[s][col])
    sol = d["sol0"].to(torch.complex128) + torch.where(cnp == ord("E"), 1.0, 0.0) * ue
    rec, obs, wgt = (torch.from_numpy(d[q]).to(DEV) for q in ("recv", "obs", "wghts"))
    mr = torch.from_numpy(d["mrdof"].astype(np.int64) - 1).to(DEV)
    ph = torch.from_numpy(TWOPI * case["freq"] * py * d["yrec"]).to(DEV)
    shift = torch.polar(torch.ones_like(ph), ph)[:, None]
    est = rec.to(torch.complex128) * sol[:, mr] * shift
    ct, sn = math.cos(math.radians(AZMOD)), math.sin(math.radians(AZMOD))
    er = torch.stack([ct * est[..., 0] - sn * est[..., 1], sn * est[..., 0] + ct * est[..., 1], est[..., 2]], -1)
    dif = obs.to(torch.complex128) - er
    w2 = wgt.double() ** 2
    res = w2 * dif * shift.conj()
    back = torch.stack([ct * res[..., 0] + sn * res[..., 1], -sn * res[..., 0] + ct * res[..., 1], res[..., 2]], -1)
    rhs = torch.zeros_like(ue)
    rhs[:, mr.reshape(-1)] = back.conj().reshape(case["nsrc"], -1)
    return {"peff": peff, "sol": sol, "est": est, "rhs": rhs,
            "misfit": (w2 * dif.abs() ** 2).sum((1, 2))}


def exact(case, seed):
    kind = case["kind"]
    mesh, g, x, z = _mesh(case, seed)
    py = 0.4 / synth.vs_min(mesh)
    if kind == "assemble":
        a = _exact_csr(case, seed, [(case["freq"], py)])[0]
        return {"csr128": a, "csr64": a}
    if kind == "driver":
        return _exact_csr(case, seed, [(case["freq"], py)])[0]
    if kind == "batch":
        sys = _systems(case, mesh, case["nfreq"], case["nky"])
        stride = (2 * g.nzero + 15) // 16 * 16
        slots = min(case["nslots"], len(sys))
        ring = torch.zeros((slots, stride), dtype=torch.float64, device=DEV)
        last = [max(k for k in range(len(sys)) if k % slots == s) for s in range(slots)]
        for s, k in enumerate(last):  # a slot holds the last system written to it
            a = _exact_csr(case, seed, [sys[k]])[0]
            ring[s, :2 * g.nzero] = torch.view_as_real(a).reshape(-1)
        return ring
    if kind == "gradient":
        return _exact_gradient(case, seed)
    if kind in ("factor", "solve"):  # the right-hand side is op(A) of this
        return _fields(x, z, [case["freq"]], case.get("nrhs", 1), _gen(seed))[0]
    if kind == "sources":
        return _exact_sources(case, seed)
    return None  # the reference's masked sums of single-precision products have no such value
