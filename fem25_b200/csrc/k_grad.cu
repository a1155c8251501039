// Exact adjoint gradient with respect to the anchor-node lambda, mu, rho:
//   g_{m,p} = sum_{pairs,s} Re( lam_s^H dA/dm_p u_s )
// evaluated without forming derivative matrices.  For the KM25ISOQ operator
// (estiff25.f:64-154) the bilinear form lam^H A u at a quadrature point with
// weight W = w_xi w_eta |J| splits into
//   lambda:  conj(div L) div U,   div V = V1,x + V3,z - i wpy V2
//   mu:      2 conj(L1,x) U1,x + 2 conj(L3,z) U3,z + 2 wpy^2 conj(L2) U2
//            + conj(L1,z + L3,x)(U1,z + U3,x)
//            + conj(L2,x - i wpy L1)(U2,x - i wpy U1)
//            + conj(L2,z - i wpy L3)(U2,z - i wpy U3)
//   rho:     -omega^2 sum_i conj(L_i) U_i
// and the derivative with respect to the anchor value m_p weights each point
// by the bilinear anchor function SF_p (cjac.f:98-108).  Fields are
// interpolated to the 13x13 points with the one-dimensional factors of the SHL
// table (dshl.f:1-243) and the inverse Jacobian (cjac.f:128-134).
//
// Bound: FP64 operations.  Interpolating with the full table costs 25 x 36
// multiply-adds at every point (900 of about 1 000); the shape functions are
// products l_ix(xi) l_ie(eta), so the kernel takes them in two steps:
//   along xi:  V[ie][qx] = sum_ix l(qx, ix) f[ie][ix], D = the same with l'
//   along eta: value = sum_ie l(qz, ie) V, d/dxi = sum_ie l(qz, ie) D,
//              d/deta = sum_ie l'(qz, ie) V
// which is 15 multiply-adds per real nodal vector at a point instead of 75,
// and the point rule is symmetric (l_i(-z) = l_{4-i}(z)), so rows ie and 4 - ie
// are stored as sum and difference and one thread serves the points qz and
// 12 - qz from one even and one odd part: 10.5.  Per element and source about
// 21 k multiply-adds of interpolation and 16 k of the forms are left.
// A CTA takes one element with 96 threads (13 x 7 point pairs), four CTAs an
// SM; the next tile's fields arrive by cp.async while this one is computed.
// 12 000 elements, 64 (pair, source) fields: 3.6 ms against 13.2 ms with the full
// table (1 224 bytes of field per element and source would take 0.2 ms); the
// shared-memory pipe is then 75 % busy and the FP64 pipe 53 %.  The forms of both
// points at once fill the 168 registers that four CTAs leave (64 bytes of stack).
#include <cstdlib>

#include "ctx.cuh"
#include "kcommon.cuh"

namespace fem25 {

constexpr int kGThreads = 96;          // >= 13 x 7 pairs of points
constexpr int kHalf = kNint / 2 + 1;   // 7 rows qz, each with its mirror 12 - qz
// staged rows of one complex nodal vector: [V, D][even 0, even 1, centre, odd
// 0, odd 1][re, im][13] doubles.  Real and imaginary parts are separate rows
// because a warp's lanes read one row at their 13 values of qx: as 8-byte words
// those are free of bank conflicts, as 16-byte words they took 5.9 wavefronts a
// load.  The strides (28 = 12 x 285 mod 16) let the lanes of an xi task, one
// vector each and then the next row, store without conflicts at TILE 2.
constexpr int kRow = 28;
constexpr int kVec = 285;
static_assert(kRow >= 2 * kNint && kVec >= 2 * kNl * kRow, "staged rows overlap");

struct GradArgs {
  int npairs, nsrc, ndof, nnpg;
  long long field_stride;  // complex entries per (pair, source) = ndof
};

__device__ __forceinline__ double re_cj(double2 a, double2 b) {
  return a.x * b.x + a.y * b.y;  // Re(conj(a) b)
}

// Values at a point of one field: div V, V1,x, V3,z, V1,z + V3,x,
// V2,x - i wpy V1, V2,z - i wpy V3 and the three components
struct GradPoint {
  double2 div, exx, ezz, exz, e12, e32, v0, v1, v2;
};

// inverse Jacobian rows: d/dx = ax d/dxi + bx d/deta, d/dz = az d/dxi + bz d/deta
struct GradJac {
  double ax, bx, az, bz;
};

// Even and odd halves of l(x, .) and l'(x, .) at the points x and 12 - x:
// sum_i l_i(x) f_i = le . (f0 + f4, f1 + f3, f2) + lo . (f0 - f4, f1 - f3), the
// odd part changes sign at 12 - x; for l' the even part does.
struct ShapeHalf {
  double le[3], lo[2], de[3], do_[2];
};
struct ShapeHalves {
  ShapeHalf h[kHalf];
};

// value, d/dxi, d/deta of one real vector at qz (a) and 12 - qz (b)
struct GradPair {
  double na, nb, xa, xb, ya, yb;
};

__device__ __forceinline__ GradPair eta_step(const ShapeHalf &t, const double (&v)[kNl],
                                             const double (&d)[kNl]) {
  GradPair o;
  const double ev = t.le[0] * v[0] + t.le[1] * v[1] + t.le[2] * v[2];
  const double ov = t.lo[0] * v[3] + t.lo[1] * v[4];
  o.na = ev + ov;
  o.nb = ev - ov;
  const double ex = t.le[0] * d[0] + t.le[1] * d[1] + t.le[2] * d[2];
  const double ox = t.lo[0] * d[3] + t.lo[1] * d[4];
  o.xa = ex + ox;
  o.xb = ex - ox;
  const double ey = t.de[0] * v[0] + t.de[1] * v[1] + t.de[2] * v[2];
  const double oy = t.do_[0] * v[3] + t.do_[1] * v[4];
  o.ya = oy + ey;
  o.yb = oy - ey;
  return o;
}

// Both points of a thread for the field whose staged components start at st
// (component stride kVec)
__device__ __forceinline__ void grad_points(const double *st, const ShapeHalf &t, const GradJac &ja,
                                            const GradJac &jb, double wpy, GradPoint &pa,
                                            GradPoint &pb) {
  double2 ax[3], az[3], bx[3], bz[3], na[3], nb[3];
#pragma unroll
  for (int k = 0; k < 3; k++) {
    double vr[kNl], vi[kNl], dr[kNl], di[kNl];
#pragma unroll
    for (int r = 0; r < kNl; r++) {
      const double *v = st + k * kVec + r * kRow, *d = v + kNl * kRow;
      vr[r] = v[0];
      vi[r] = v[kNint];
      dr[r] = d[0];
      di[r] = d[kNint];
    }
    const GradPair re = eta_step(t, vr, dr), im = eta_step(t, vi, di);
    na[k] = make_double2(re.na, im.na);
    nb[k] = make_double2(re.nb, im.nb);
    ax[k] = make_double2(ja.ax * re.xa + ja.bx * re.ya, ja.ax * im.xa + ja.bx * im.ya);
    az[k] = make_double2(ja.az * re.xa + ja.bz * re.ya, ja.az * im.xa + ja.bz * im.ya);
    bx[k] = make_double2(jb.ax * re.xb + jb.bx * re.yb, jb.ax * im.xb + jb.bx * im.yb);
    bz[k] = make_double2(jb.az * re.xb + jb.bz * re.yb, jb.az * im.xb + jb.bz * im.yb);
  }
  auto forms = [&](const double2 (&x)[3], const double2 (&z)[3], const double2 (&n)[3],
                   GradPoint &p) {
    p.div = make_double2(x[0].x + z[2].x + wpy * n[1].y, x[0].y + z[2].y - wpy * n[1].x);
    p.exx = x[0];
    p.ezz = z[2];
    p.exz = make_double2(z[0].x + x[2].x, z[0].y + x[2].y);
    p.e12 = make_double2(x[1].x + wpy * n[0].y, x[1].y - wpy * n[0].x);
    p.e32 = make_double2(z[1].x + wpy * n[2].y, z[1].y - wpy * n[2].x);
    p.v0 = n[0];
    p.v1 = n[1];
    p.v2 = n[2];
  };
  forms(ax, az, na, pa);
  forms(bx, bz, nb, pb);
}

// lambda, mu and rho forms of one point added to acc
__device__ __forceinline__ void grad_forms(const GradPoint &u, const GradPoint &l, double wpy,
                                           double w2, double (&acc)[3]) {
  acc[0] += re_cj(l.div, u.div);
  const double v1 = re_cj(l.v1, u.v1);
  const double diag = re_cj(l.exx, u.exx) + re_cj(l.ezz, u.ezz) + wpy * wpy * v1;
  acc[1] += 2.0 * diag + re_cj(l.exz, u.exz) + re_cj(l.e12, u.e12) + re_cj(l.e32, u.e32);
  acc[2] += -w2 * (re_cj(l.v0, u.v0) + v1 + re_cj(l.v2, u.v2));
}

// TILE (pair, source) fields of u and lambda pass through shared memory per
// step, in pair-then-source order over the launch's pairs; the result does not
// depend on TILE (each point sums them in that order).
template <int TILE>
__global__ void __launch_bounds__(kGThreads, 4)
    k_grad_plain(MeshView mv, DevTables dt, GradArgs ga, const int *__restrict__ elems,
                 const int *__restrict__ lm, PairTable pt, ShapeHalves tb,
                 const double2 *__restrict__ u, const double2 *__restrict__ lam,
                 double *__restrict__ grad, int *__restrict__ err) {
  extern __shared__ double2 sm2[];
  double2 *fld = sm2;                        // [TILE][u, lambda][75]
  double *st = reinterpret_cast<double *>(fld + TILE * 2 * kNee);  // [TILE][u, lambda][3][kVec]
  __shared__ int dof[kNee];
  __shared__ double red[12][kGThreads / 32];
  const int t = threadIdx.x;
  const int e = elems[blockIdx.x];
  const int4 ie = mv.ieng[e];
  for (int k = t; k < kNee; k += kGThreads) dof[k] = lm[(size_t)e * kNee + k];
  __syncthreads();
  const int ncomb = ga.npairs * ga.nsrc;
  // fields of tile i; fixed DOFs (0) are zero-filled
  auto fetch = [&](int i) {
    const int c0 = i * TILE, nc = min(TILE, ncomb - c0);
    for (int j = t; j < nc * 2 * kNee; j += kGThreads) {
      const int s = j / (2 * kNee), r = j - s * 2 * kNee;
      const bool isl = r >= kNee;
      const int d = dof[isl ? r - kNee : r];
      const double2 *src = (isl ? lam : u) + (d > 0 ? (size_t)(c0 + s) * ga.field_stride + d - 1 : 0);
      const int bytes = d > 0 ? 16 : 0;
      asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(
                       (unsigned)__cvta_generic_to_shared(fld + j)),
                   "l"(src), "r"(bytes)
                   : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  if (ncomb > 0) fetch(0);
  const bool act = t < kNint * kHalf;
  const int qx = act ? t % kNint : 0, qz = act ? t / kNint : 0;
  const int q2[2] = {qx + kNint * qz, qx + kNint * (kNint - 1 - qz)};
  // the centre row is its own mirror: its second point carries no weight
  const bool own[2] = {act, act && qz != kNint - 1 - qz};
  GradJac jac[2];
  double wq[2];
#pragma unroll
  for (int h = 0; h < 2; h++) {
    QGeo g;
    const bool ok = quad_geo(mv, dt, ie, q2[h], false, g);
    if (!ok && act) atomicCAS(err, 0, e + 1);
    jac[h].ax = g.dzdeta / g.rjac;
    jac[h].bx = -g.dzdxi / g.rjac;
    jac[h].az = -g.dxdeta / g.rjac;
    jac[h].bz = g.dxdxi / g.rjac;
    wq[h] = dt.wts[qx] * dt.wts[q2[h] / kNint] * g.rjac;
  }
  const ShapeHalf et = tb.h[qz];
  double acc[2][3] = {{0.0, 0.0, 0.0}, {0.0, 0.0, 0.0}};
  const int ntile = (ncomb + TILE - 1) / TILE;
  for (int i = 0; i < ntile; i++) {
    const int c0 = i * TILE, nc = min(TILE, ncomb - c0);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();  // tile i's fields visible; tile i - 1's staged rows read
    // ---- xi step: task (row r, nodal vector): r = 0, 1 the sums of rows r and
    // 4 - r, r = 2 the centre row, r = 3, 4 the differences (the halves sit in
    // the eta coefficients); points x and 12 - x from one even and one odd part
    for (int task = t; task < 6 * kNl * nc; task += kGThreads) {
      const int r = task / (6 * nc), vec = task - r * 6 * nc;  // vec = 3 (2 s + field) + comp
      const double2 *f = fld + (vec / 3) * kNee + vec % 3;
      const int r0 = r < 3 ? r : r - 3;
      const double sg = r < 2 ? 1.0 : r == 2 ? 0.0 : -1.0;
      double2 a[kNl];
#pragma unroll
      for (int ix = 0; ix < kNl; ix++) {
        const double2 lo = f[3 * (kNl * r0 + ix)], hi = f[3 * (kNl * (kNl - 1 - r0) + ix)];
        a[ix] = make_double2(lo.x + sg * hi.x, lo.y + sg * hi.y);
      }
      const double2 e0 = make_double2(a[0].x + a[4].x, a[0].y + a[4].y);
      const double2 e1 = make_double2(a[1].x + a[3].x, a[1].y + a[3].y);
      const double2 o0 = make_double2(a[0].x - a[4].x, a[0].y - a[4].y);
      const double2 o1 = make_double2(a[1].x - a[3].x, a[1].y - a[3].y);
      double *ov = st + vec * kVec + r * kRow, *od = ov + kNl * kRow;
#pragma unroll
      for (int x = 0; x < kHalf; x++) {
        const ShapeHalf &h = tb.h[x];
        const double2 ev = make_double2(h.le[0] * e0.x + h.le[1] * e1.x + h.le[2] * a[2].x,
                                        h.le[0] * e0.y + h.le[1] * e1.y + h.le[2] * a[2].y);
        const double2 od2 = make_double2(h.lo[0] * o0.x + h.lo[1] * o1.x,
                                         h.lo[0] * o0.y + h.lo[1] * o1.y);
        const double2 ed = make_double2(h.de[0] * e0.x + h.de[1] * e1.x + h.de[2] * a[2].x,
                                        h.de[0] * e0.y + h.de[1] * e1.y + h.de[2] * a[2].y);
        const double2 dd = make_double2(h.do_[0] * o0.x + h.do_[1] * o1.x,
                                        h.do_[0] * o0.y + h.do_[1] * o1.y);
        ov[x] = ev.x + od2.x;
        ov[kNint + x] = ev.y + od2.y;
        od[x] = dd.x + ed.x;
        od[kNint + x] = dd.y + ed.y;
        if (x < kHalf - 1) {
          ov[kNint - 1 - x] = ev.x - od2.x;
          ov[2 * kNint - 1 - x] = ev.y - od2.y;
          od[kNint - 1 - x] = dd.x - ed.x;
          od[2 * kNint - 1 - x] = dd.y - ed.y;
        }
      }
    }
    __syncthreads();
    if (i + 1 < ntile) fetch(i + 1);  // the tile's fields are consumed
    // ---- eta step and forms at the thread's two points
    if (act) {
      for (int s = 0; s < nc; s++) {
        const double2 pr = pt.p[(c0 + s) / ga.nsrc];
        GradPoint ua, ub, la, lb;
        grad_points(st + (2 * s) * 3 * kVec + qx, et, jac[0], jac[1], pr.y, ua, ub);
        grad_points(st + (2 * s + 1) * 3 * kVec + qx, et, jac[0], jac[1], pr.y, la, lb);
        grad_forms(ua, la, pr.y, pr.x * pr.x, acc[0]);
        grad_forms(ub, lb, pr.y, pr.x * pr.x, acc[1]);
      }
    }
  }
  // g_{m, anchor a} = sum_q SF_a(q) W_q acc_m(q)
  double v[12];
#pragma unroll
  for (int a = 0; a < 4; a++) {
    const double fa = own[0] ? dt.sf[4 * q2[0] + a] * wq[0] : 0.0;
    const double fb = own[1] ? dt.sf[4 * q2[1] + a] * wq[1] : 0.0;
#pragma unroll
    for (int m = 0; m < 3; m++) v[3 * a + m] = fa * acc[0][m] + fb * acc[1][m];
  }
#pragma unroll
  for (int k = 0; k < 12; k++) {
    double x = v[k];
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    v[k] = x;
  }
  const int warp = t / 32, lane = t % 32, nw = kGThreads / 32;
  if (lane == 0)
    for (int k = 0; k < 12; k++) red[k][warp] = v[k];
  __syncthreads();
  if (t < 12) {
    double x = 0.0;
    for (int w = 0; w < nw; w++) x += red[t][w];
    const int a = t / 3, m = t % 3;
    const int anchor = (a == 0 ? ie.x : a == 1 ? ie.y : a == 2 ? ie.z : ie.w) - 1;
    atomicAdd(&grad[(size_t)m * ga.nnpg + anchor], x);
  }
}

ShapeTabs shape_tables(const Tables &t) {
  // Lagrange basis on the 5 GLL points (the factors of SHL, dshl.f:100-243)
  ShapeTabs tb;
  for (int q = 0; q < kNint; q++) {
    const double x = t.xigll[q];
    for (int i = 0; i < kNl; i++) {
      double v = 1.0, dsum = 0.0;
      for (int k = 0; k < kNl; k++)
        if (k != i) v *= (x - t.xipts[k]) / (t.xipts[i] - t.xipts[k]);
      for (int m = 0; m < kNl; m++) {
        if (m == i) continue;
        double p = 1.0 / (t.xipts[i] - t.xipts[m]);
        for (int k = 0; k < kNl; k++)
          if (k != i && k != m) p *= (x - t.xipts[k]) / (t.xipts[i] - t.xipts[k]);
        dsum += p;
      }
      tb.l[q][i] = v;
      tb.d[q][i] = dsum;
    }
  }
  return tb;
}

static ShapeHalves shape_halves(const Tables &tab) {
  const ShapeTabs t = shape_tables(tab);
  ShapeHalves o;
  for (int q = 0; q < kHalf; q++) {
    ShapeHalf &h = o.h[q];
    for (int i = 0; i < 2; i++) {
      h.le[i] = 0.5 * (t.l[q][i] + t.l[q][kNl - 1 - i]);
      h.lo[i] = 0.5 * (t.l[q][i] - t.l[q][kNl - 1 - i]);
      h.de[i] = 0.5 * (t.d[q][i] + t.d[q][kNl - 1 - i]);
      h.do_[i] = 0.5 * (t.d[q][i] - t.d[q][kNl - 1 - i]);
    }
    h.le[2] = t.l[q][2];
    h.de[2] = t.d[q][2];
  }
  return o;
}

static size_t grad_smem(int tile) {
  return (size_t)tile * (sizeof(double2) * 2 * kNee + sizeof(double) * 6 * kVec);
}

template <int TILE>
static cudaError_t grad_tile_launch(Ctx *c, const GradArgs &ga, const PairTable &pt,
                                    const double *u, const double *lam, double *grad,
                                    cudaStream_t st) {
  cudaError_t e;
  if ((e = cudaFuncSetAttribute(k_grad_plain<TILE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)grad_smem(TILE))))
    return e;
  k_grad_plain<TILE><<<c->n_nonpml, kGThreads, grad_smem(TILE), st>>>(
      c->mv, c->dt, ga, c->d_nonpml, c->d_lm, pt, shape_halves(c->tab), (const double2 *)u,
      (const double2 *)lam, grad, c->d_err);
  return cudaGetLastError();
}

// The tile width (fields of both kinds staged per shared-memory pass) trades
// shared memory per CTA against barriers per field: 2 keeps four CTAs on an SM
// (32 KB each) and is the default, 4 keeps three, 8 one (12 000 elements, 64
// fields: 3.6, 4.7 and 7.4 ms).  FEM25_GRAD_TILE forces 2, 4 or 8.
cudaError_t launch_grad_plain(Ctx *c, const PairTable &pt, int npairs, int nsrc, const double *u,
                              const double *lam, double *grad, cudaStream_t st) {
  GradArgs ga;
  ga.npairs = npairs;
  ga.nsrc = nsrc;
  ga.ndof = c->ndof;
  ga.nnpg = c->nnpg;
  ga.field_stride = c->ndof;
  if (c->n_nonpml == 0) return cudaSuccess;
  int tile = 2;
  if (const char *env = std::getenv("FEM25_GRAD_TILE")) {
    const int w = std::atoi(env);
    tile = (w == 2 || w == 8) ? w : 4;
  }
  c->grad_tile = tile;
  switch (tile) {
    case 4: return grad_tile_launch<4>(c, ga, pt, u, lam, grad, st);
    case 8: return grad_tile_launch<8>(c, ga, pt, u, lam, grad, st);
    default: return grad_tile_launch<2>(c, ga, pt, u, lam, grad, st);
  }
}

}  // namespace fem25
