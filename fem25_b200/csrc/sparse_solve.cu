// Sparse direct solve of one assembled system on the GPU: multifrontal LU
// with a nested-dissection ordering of the element mesh.  It stands in for
// the host MUMPS factor / solve hop of the reference (forward solve
// bielak25.f90:443-446, 545-551; transpose adjoint solve adjgrad.f90:327-341)
// on meshes far beyond the dense solve's reach, so the assemble -> solve ->
// misfit -> adjoint -> gradient loop stays on the device at the sizes of the
// benchmark meshes.
//
// Ordering (host, once per context).  The elements are bisected recursively
// along the longer side of their centroids' bounding box; the DOFs shared by
// the two halves that no coarser separator has taken form the separator of
// the tree node, and a leaf (at most kLeafElems elements) keeps every DOF of
// its elements that no separator took.  Because two DOFs are coupled only
// through an element they share, a separator splits the matrix graph.  The
// tree is the elimination tree: front t holds its own DOFs (the "fully
// summed" rows and columns, eliminated there) and its boundary: the DOFs of
// its subtree's elements owned by an ancestor, ordered by elimination.
//
// Factorisation (device, sparse_factor.cu), level by level from the leaves: every
// front of a level is assembled in a work buffer -- the update (Schur complement)
// blocks of its two children, plus the CSR entries whose first eliminated DOF it
// owns -- and partially factored: F11 = P L11 U11 with partial pivoting
// restricted to the fully summed rows, L21 = F21 U11^-1, U12 = L11^-1 P F12,
// update = F22 - L21 U12.  The factors (L11\U11 over L21, and U12) go to a store
// kept by the context; the update blocks live until the parent level has consumed
// them (two work buffers, alternating).
//
// Solve (device), one launch per level: forward elimination from the leaves,
// back substitution from the root, for op(A) = A, A^T (MUMPS ICNTL(9) != 1)
// or A^H; a CTA per (front, group of right-hand sides), the triangles in
// blocks of 32 rows whose diagonal blocks the store holds inverted.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <numeric>

#include "sparse.cuh"

namespace fem25 {

// ---------------------------------------------------------------------------
// symbolic analysis (host)
// ---------------------------------------------------------------------------
namespace {

struct Builder {
  const int *lm_all;  // LM(3,25,NELEM), 1-based DOFs
  std::vector<double> cx, cz;
  std::vector<int> owner;    // DOF -> front (0-based DOF)
  std::vector<int> mark;     // scratch stamps per DOF
  int stamp = 0;
  std::vector<SpFront> fr;
  std::vector<std::vector<int>> own_list;   // per front, its own DOFs (ascending)
  std::vector<std::vector<int>> elems;      // per front, its subtree's elements

  int rec(std::vector<int> &E, int depth) {
    const int *lm = lm_all;
    if ((int)E.size() <= sp::kLeafElems) {
      std::vector<int> own;
      for (int e : E)
        for (int q = 0; q < kNee; q++) {
          const int d = lm[(size_t)e * kNee + q] - 1;
          if (d >= 0 && owner[d] == -1) {
            owner[d] = -3;  // claimed by this leaf (id given below)
            own.push_back(d);
          }
        }
      std::sort(own.begin(), own.end());
      const int id = (int)fr.size();
      for (int d : own) owner[d] = id;
      SpFront f{};
      f.k = (int)own.size();
      f.parent = -1;
      f.child[0] = f.child[1] = -1;
      f.level = depth;
      fr.push_back(f);
      own_list.push_back(std::move(own));
      elems.push_back(E);
      return id;
    }
    // bisect along the longer side of the centroids' bounding box
    double x0 = 1e300, x1 = -1e300, z0 = 1e300, z1 = -1e300;
    for (int e : E) {
      x0 = std::min(x0, cx[e]);
      x1 = std::max(x1, cx[e]);
      z0 = std::min(z0, cz[e]);
      z1 = std::max(z1, cz[e]);
    }
    const bool alongx = (x1 - x0) >= (z1 - z0);
    const size_t h = E.size() / 2;
    std::nth_element(E.begin(), E.begin() + h, E.end(), [&](int a, int b) {
      const double va = alongx ? cx[a] : cz[a], vb = alongx ? cx[b] : cz[b];
      return va < vb || (va == vb && a < b);
    });
    std::vector<int> E1(E.begin(), E.begin() + h), E2(E.begin() + h, E.end());
    // separator: free DOFs of both halves
    ++stamp;
    for (int e : E1)
      for (int q = 0; q < kNee; q++) {
        const int d = lm[(size_t)e * kNee + q] - 1;
        if (d >= 0) mark[d] = stamp;
      }
    std::vector<int> sep;
    for (int e : E2)
      for (int q = 0; q < kNee; q++) {
        const int d = lm[(size_t)e * kNee + q] - 1;
        if (d >= 0 && mark[d] == stamp && owner[d] == -1) {
          owner[d] = -2;  // taken by this separator (id given below)
          sep.push_back(d);
        }
      }
    const int c1 = rec(E1, depth + 1);
    const int c2 = rec(E2, depth + 1);
    std::sort(sep.begin(), sep.end());
    const int id = (int)fr.size();
    for (int d : sep) owner[d] = id;
    SpFront f{};
    f.k = (int)sep.size();
    f.parent = -1;
    f.child[0] = c1;
    f.child[1] = c2;
    f.level = depth;
    fr[c1].parent = id;
    fr[c2].parent = id;
    fr.push_back(f);
    own_list.push_back(std::move(sep));
    elems.push_back(E);
    return id;
  }
};

}  // namespace

// The dissection of a mesh (host only): the fronts with their own and
// boundary DOFs, elimination positions, levels and the offsets of every
// front's work and factor blocks.
struct FrontPlan {
  std::vector<SpFront> fr;
  std::vector<std::vector<int>> own, bnd;
  std::vector<long long> pos;
  std::vector<int> owner;
  std::vector<std::vector<int>> lev;
  std::vector<long long> lev_work;
  long long fac_elems = 0, bnd_tot = 0, map_tot = 0;
  int nlev = 0;
};

static int plan_fronts(int nelem, int n, const int *lm, const int *ieng, const double *xa,
                       const double *za, FrontPlan *pl, std::string *msg) {
  Builder b;
  b.lm_all = lm;
  b.cx.resize(nelem);
  b.cz.resize(nelem);
  for (int e = 0; e < nelem; e++) {
    double x = 0, z = 0;
    for (int a = 0; a < 4; a++) {
      const int p = ieng[4 * e + a] - 1;
      x += xa[p];
      z += za[p];
    }
    b.cx[e] = 0.25 * x;
    b.cz[e] = 0.25 * z;
  }
  b.owner.assign(n, -1);
  b.mark.assign(n, 0);
  std::vector<int> E(nelem);
  std::iota(E.begin(), E.end(), 0);
  b.rec(E, 0);
  for (int d = 0; d < n; d++)
    if (b.owner[d] < 0) {
      *msg = "sparse solve: a DOF belongs to no element";
      return FEM25_ERR_PATTERN;
    }
  const int nf = (int)b.fr.size();
  // elimination positions (postorder = front id order)
  std::vector<long long> &pos = pl->pos;
  pos.assign(n, 0);
  long long p = 0;
  for (int t = 0; t < nf; t++) {
    b.fr[t].own0 = p;
    for (int d : b.own_list[t]) pos[d] = p++;
  }
  // boundaries: DOFs of the subtree's elements owned by an ancestor (id > t)
  std::vector<std::vector<int>> &bnd = pl->bnd;
  bnd.assign(nf, {});
  {
    std::vector<int> seen(n, -1);
    for (int t = 0; t < nf; t++) {
      std::vector<int> &B = bnd[t];
      for (int e : b.elems[t])
        for (int q = 0; q < kNee; q++) {
          const int d = lm[(size_t)e * kNee + q] - 1;
          if (d >= 0 && b.owner[d] > t && seen[d] != t) {
            seen[d] = t;
            B.push_back(d);
          }
        }
      std::sort(B.begin(), B.end(), [&](int x, int y) { return pos[x] < pos[y]; });
      b.fr[t].m = (int)B.size();
      b.elems[t].clear();
      b.elems[t].shrink_to_fit();
    }
  }
  // levels, offsets
  int nlev = 0;
  for (auto &f : b.fr) nlev = std::max(nlev, f.level + 1);
  pl->lev.assign(nlev, {});
  pl->lev_work.assign(nlev, 0);
  long long bnd_tot = 0, fac = 0;
  for (int t = 0; t < nf; t++) {
    SpFront &f = b.fr[t];
    const long long nn = (long long)f.k + f.m;
    f.bnd0 = bnd_tot;
    bnd_tot += f.m;
    f.map0 = pl->map_tot;
    pl->map_tot += 2 * nn;
    f.fac0 = fac;
    fac += nn * f.k + (long long)f.k * f.m;
    f.work0 = pl->lev_work[f.level];
    pl->lev_work[f.level] += nn * nn;
    pl->lev[f.level].push_back(t);
  }
  pl->fac_elems = fac;
  pl->bnd_tot = bnd_tot;
  pl->nlev = nlev;
  pl->fr = std::move(b.fr);
  pl->own = std::move(b.own_list);
  pl->owner = std::move(b.owner);
  return 0;
}

// fronts, levels, factor bytes, largest level work bytes, largest own count,
// largest front order, real flops of one factorisation (8 per complex
// multiply-add)
static void plan_stats(const std::vector<SpFront> &fr, long long fac_elems,
                       const std::vector<long long> &lev_work, long long *out) {
  int kmax = 0, nmax = 0, nlev = 0;
  double flops = 0.0;
  for (const SpFront &f : fr) {
    kmax = std::max(kmax, f.k);
    nmax = std::max(nmax, f.k + f.m);
    nlev = std::max(nlev, f.level + 1);
    const double k = f.k, m = f.m;
    flops += 8.0 / 3.0 * k * k * k + 8.0 * k * k * m + 8.0 * k * m * m;
  }
  long long wmax = 0;
  for (long long w : lev_work) wmax = std::max(wmax, w);
  out[0] = (long long)fr.size();
  out[1] = nlev;
  out[2] = fac_elems * 16;
  out[3] = wmax * 16;
  out[4] = kmax;
  out[5] = nmax;
  out[6] = (long long)flops;
}

int sparse_plan_info(int nelem, int ndof, const int *lm, const int *ieng, const double *x,
                     const double *z, long long *out, std::string *msg) {
  FrontPlan pl;
  const int r = plan_fronts(nelem, ndof, lm, ieng, x, z, &pl, msg);
  if (r) return r;
  plan_stats(pl.fr, pl.fac_elems, pl.lev_work, out);
  return 0;
}

// Builds the ordering, the fronts, the extend-add maps and the CSR-entry map;
// uploads them.  0, or a FEM25 status with *msg.
static int sparse_analyse(Ctx *c, SparseLU *s, cudaStream_t st, std::string *msg) {
  const int n = c->ndof;
  FrontPlan pl;
  {
    const int r = plan_fronts(c->nelem, n, c->h_lm.data(), c->h_ieng.data(), c->h_x.data(),
                              c->h_z.data(), &pl, msg);
    if (r) return r;
  }
  const int nf = (int)pl.fr.size();
  const int nlev = pl.nlev;
  const std::vector<long long> &pos = pl.pos;
  const std::vector<std::vector<int>> &bnd = pl.bnd;
  struct {
    std::vector<SpFront> &fr;
    std::vector<std::vector<int>> &own_list;
    std::vector<int> &owner;
  } b{pl.fr, pl.own, pl.owner};
  // index of DOF d in front t (own: by position; boundary: by search)
  auto local = [&](int t, int d) -> int {
    const SpFront &f = b.fr[t];
    if (b.owner[d] == t) return (int)(pos[d] - f.own0);
    const std::vector<int> &B = bnd[t];
    auto it = std::lower_bound(B.begin(), B.end(), d,
                               [&](int x, int y) { return pos[x] < pos[y]; });
    if (it == B.end() || *it != d) return -1;
    return f.k + (int)(it - B.begin());
  };
  s->lev = pl.lev;
  s->lev_work = pl.lev_work;
  s->fac_elems = pl.fac_elems;
  s->max_work = 0;
  for (long long w : s->lev_work) s->max_work = std::max(s->max_work, w);
  const long long bnd_tot = pl.bnd_tot;
  // pull maps: index in a front -> index in the boundary of child 0 / 1, or -1
  std::vector<int> pull(pl.map_tot, -1), own_all(n), bnd_all(bnd_tot);
  for (int t = 0; t < nf; t++) {
    const SpFront &f = b.fr[t];
    std::copy(b.own_list[t].begin(), b.own_list[t].end(), own_all.begin() + f.own0);
    std::copy(bnd[t].begin(), bnd[t].end(), bnd_all.begin() + f.bnd0);
    if (f.m > 0 && f.parent < 0) {
      *msg = "sparse solve: a boundary DOF has no parent front";
      return FEM25_ERR_PATTERN;
    }
    if (f.m == 0) continue;
    const SpFront &pf = b.fr[f.parent];
    int *map = pull.data() + pf.map0 + (pf.child[0] == t ? 0 : (long long)pf.k + pf.m);
    for (int i = 0; i < f.m; i++) {
      const int li = local(f.parent, bnd[t][i]);
      if (li < 0) {
        *msg = "sparse solve: a boundary DOF is missing from the parent front";
        return FEM25_ERR_PATTERN;
      }
      map[li] = i;
    }
  }
  // CSR entries -> (front, local offset), grouped by level
  std::vector<int> jc(c->nzero);
  cudaError_t e;
  if ((e = cudaMemcpy(jc.data(), c->d_jcptr, sizeof(int) * c->nzero, cudaMemcpyDeviceToHost))) {
    *msg = std::string("sparse solve: ") + cudaGetErrorString(e);
    return FEM25_ERR_CUDA;
  }
  // two passes over the rows in chunks: count the entries of each level per
  // chunk, then place each entry at its level's and chunk's next slot
  const int nchunk = 256;
  const int rows_per = (n + nchunk - 1) / nchunk;
  std::vector<long long> cnt((size_t)nchunk * nlev, 0);
  int bad = 0;
  auto entry_front = [&](int i, int j) { return pos[i] <= pos[j] ? b.owner[i] : b.owner[j]; };
#pragma omp parallel for schedule(dynamic, 1)
  for (int ch = 0; ch < nchunk; ch++) {
    long long *cc = cnt.data() + (size_t)ch * nlev;
    const int i1 = std::min(n, (ch + 1) * rows_per);
    for (int i = ch * rows_per; i < i1; i++)
      for (int q = c->h_irptr[i] - 1; q < c->h_irptr[i + 1] - 1; q++)
        cc[b.fr[entry_front(i, jc[q] - 1)].level]++;
  }
  s->lev_ent0.assign(nlev + 1, 0);
  std::vector<long long> cur((size_t)nchunk * nlev);
  {
    long long acc = 0;
    for (int l = 0; l < nlev; l++) {
      s->lev_ent0[l] = acc;
      for (int ch = 0; ch < nchunk; ch++) {
        cur[(size_t)ch * nlev + l] = acc;
        acc += cnt[(size_t)ch * nlev + l];
      }
    }
    s->lev_ent0[nlev] = acc;
  }
  std::vector<int> sidx(c->nzero);
  std::vector<long long> sloc(c->nzero);
#pragma omp parallel for schedule(dynamic, 1) reduction(+ : bad)
  for (int ch = 0; ch < nchunk; ch++) {
    long long *cc = cur.data() + (size_t)ch * nlev;
    const int i1 = std::min(n, (ch + 1) * rows_per);
    for (int i = ch * rows_per; i < i1; i++)
      for (int q = c->h_irptr[i] - 1; q < c->h_irptr[i + 1] - 1; q++) {
        const int j = jc[q] - 1;
        const int t = entry_front(i, j);
        const int li = local(t, i), lj = local(t, j);
        if (li < 0 || lj < 0) {
          bad++;
          continue;
        }
        const long long nn = (long long)b.fr[t].k + b.fr[t].m;
        const long long o = cc[b.fr[t].level]++;
        sidx[o] = q;
        sloc[o] = b.fr[t].work0 + li + (long long)lj * nn;
      }
  }
  if (bad) {
    *msg = "sparse solve: a matrix entry couples DOFs of no common front";
    return FEM25_ERR_PATTERN;
  }
  std::vector<int>().swap(jc);
  // fronts with k <= kSmallK first in each level's list
  s->lev_nsmall.assign(nlev, 0);
  s->lev_ksmall.assign(nlev, 0);
  s->lev_msmall.assign(nlev, 0);
  s->lev_kmax.assign(nlev, 0);
  s->lev_mmax.assign(nlev, 0);
  s->lev_nmax.assign(nlev, 0);
  auto small = [&](int t) { return b.fr[t].k <= sp::kSmallK; };
  for (int l = 0; l < nlev; l++) {
    std::stable_partition(s->lev[l].begin(), s->lev[l].end(), small);
    for (int t : s->lev[l]) {
      const SpFront &f = b.fr[t];
      s->lev_kmax[l] = std::max(s->lev_kmax[l], f.k);
      s->lev_mmax[l] = std::max(s->lev_mmax[l], f.m);
      s->lev_nmax[l] = std::max(s->lev_nmax[l], f.k + f.m);
      if (small(t)) {
        s->lev_nsmall[l]++;
        s->lev_ksmall[l] = std::max(s->lev_ksmall[l], f.k);
        s->lev_msmall[l] = std::max(s->lev_msmall[l], f.m);
      }
    }
  }
  // level front lists, concatenated
  std::vector<int> lf;
  s->lev_off.assign(nlev + 1, 0);
  for (int l = 0; l < nlev; l++) {
    s->lev_off[l] = (long long)lf.size();
    lf.insert(lf.end(), s->lev[l].begin(), s->lev[l].end());
  }
  s->lev_off[nlev] = (long long)lf.size();
  // upload
  auto up = [&](void **d, const void *h, size_t bytes) -> cudaError_t {
    cudaError_t r = cudaMalloc(d, bytes ? bytes : 16);
    if (r == cudaSuccess && bytes) r = cudaMemcpy(*d, h, bytes, cudaMemcpyHostToDevice);
    return r;
  };
  if ((e = up((void **)&s->d_fr, b.fr.data(), sizeof(SpFront) * nf)) ||
      (e = up((void **)&s->d_own, own_all.data(), sizeof(int) * n)) ||
      (e = up((void **)&s->d_bnd, bnd_all.data(), sizeof(int) * bnd_tot)) ||
      (e = up((void **)&s->d_pull, pull.data(), sizeof(int) * pull.size())) ||
      (e = up((void **)&s->d_lev_fronts, lf.data(), sizeof(int) * lf.size())) ||
      (e = up((void **)&s->d_ent_idx, sidx.data(), sizeof(int) * sidx.size())) ||
      (e = up((void **)&s->d_ent_loc, sloc.data(), sizeof(long long) * sloc.size()))) {
    *msg = std::string("sparse solve: ") + cudaGetErrorString(e) + " (symbolic tables)";
    return FEM25_ERR_ALLOC;
  }
  s->fr = std::move(b.fr);
  s->nfront = nf;
  s->nlevel = nlev;
  s->analysed = true;
  (void)st;
  return 0;
}

// ---------------------------------------------------------------------------
// solve (device): x is [nrhs][NDOF]
// ---------------------------------------------------------------------------
// Per front, with y its own rows of x and x_b its boundary rows:
//   op(A) = A    forward: y = L11^-1 P y, x_b -= L21 y
//                backward: y -= U12 x_b, y = U11^-1 y
//   A^T / A^H    forward: y = U11^-op y, x_b -= U12^op y
//                backward: y -= L21^op x_b, y = P^T L11^-op y
// Bound: reading the factors (once a pass for a group of right-hand sides); the
// operations are 8 flops a factor entry and right-hand side.  Every factor entry
// is read by one lane of one warp straight into a tensor-core operand (8 rows x
// 4 columns a warp, 128-byte column pieces, or 64-byte ones of op(A) = A^T) and
// meets 8 NT right-hand sides from shared memory, so the factors need no staging
// and one right-hand side is the same kernel with 7 idle columns (its padded
// operations stay under the time of the reads).  The triangles are products with
// the inverted 32 x 32 diagonal blocks, two barriers a block.
// A front's boundary rows belong to ancestors and fronts of one level share
// them, so the forward updates add with atomics.
struct SolveArgs {
  const int *fronts;
  const SpFront *fr;
  const int *own, *bnd;
  const double2 *fac;
  const int *perm;
  double2 *x;
  int ndof, nrhs, trans;  // trans 0: A, 1: A^T, 2: A^H
};

// entries (r, c) of a block of op(A): p[r rs + c cs], conjugated by sg = -1
struct SpView {
  const double2 *p;
  long long rs, cs;
  double sg;
  __device__ __forceinline__ double2 at(int r, int c) const {
    const double2 v = __ldg(p + r * rs + c * cs);
    return make_double2(v.x, sg * v.y);
  }
};

// One front's step of the forward (fwd) or backward pass
struct SpStep {
  int k, m;
  bool unit;        // the triangle's diagonal is 1
  SpView tri, rect; // triangle (own x own), rectangle (fwd: boundary x own, bwd: own x boundary)
  __device__ __forceinline__ SpStep(const SolveArgs &a, const SpFront &f, bool fwd) {
    k = f.k;
    m = f.m;
    const long long n = (long long)f.k + f.m;
    const double2 *L = a.fac + f.fac0, *U12 = L + n * f.k;
    const bool t = a.trans != 0;
    const double sg = a.trans == 2 ? -1.0 : 1.0;
    unit = fwd != t;
    tri = t ? SpView{L, n, 1, sg} : SpView{L, 1, n, sg};
    if (fwd)
      rect = t ? SpView{U12, f.k, 1, sg} : SpView{L + f.k, 1, n, sg};
    else
      rect = t ? SpView{L + f.k, n, 1, sg} : SpView{U12, 1, f.k, sg};
  }
  // entry of the inverted diagonal block's triangle
  __device__ __forceinline__ double2 diag(int r, int c, bool lower) const {
    if (r >= k || c >= k || (lower ? c > r : c < r)) return make_double2(0.0, 0.0);
    if (r == c && unit) return make_double2(1.0, 0.0);
    return tri.at(r, c);
  }
};

// z[NT] (8 rows from r0 x 8 NT columns) += V(r0.., c0..c0 + nc) Y, Y in shared
// memory with row stride 8 NT + 2 (free of conflicts for the operand's lanes) and
// zero rows from nc to the next multiple of 4.  Rows of V end at nr: the lanes
// past them (and past the last column) read the last one, and their rows of z
// are not to be kept.
template <int NT>
__device__ __forceinline__ void sp_product(const SpView &V, int r0, int nr, int c0, int nc,
                                           const double2 *Y, ZTile (&z)[NT]) {
  constexpr int ld = 8 * NT + 2;
  const int lane = threadIdx.x & 31, lr = lane >> 2, lk = lane & 3;
  const double2 *row = V.p + (long long)min(r0 + lr, nr - 1) * V.rs + c0 * V.cs;
  const long long cs4 = 4 * V.cs;
  Y += lk * ld + lr;
  for (int q0 = 0; q0 < nc; q0 += 32) {
    double2 a[8];
    if (q0 + 32 <= nc) {
      const double2 *p = row + (q0 + lk) * V.cs;
#pragma unroll
      for (int q = 0; q < 8; q++) a[q] = __ldg(p + q * cs4);
    } else {
#pragma unroll
      for (int q = 0; q < 8; q++) a[q] = __ldg(row + min(q0 + 4 * q + lk, nc - 1) * V.cs);
    }
#pragma unroll
    for (int q = 0; q < 8; q++)
      if (q0 + 4 * q < nc) {
        const double2 v = make_double2(a[q].x, V.sg * a[q].y);
#pragma unroll
        for (int t = 0; t < NT; t++) z[t].mma(v, Y[(q0 + 4 * q) * ld + 8 * t]);
      }
  }
}

// Y[r][s] = x(s0 + s, idx[pm ? pm[r] : r]), zero past n rows (up to npad) and ns
// columns.  With 32 columns a lane keeps its rows and a warp walks columns (the
// index is read once); with few, a warp takes 32 rows of a column at a time, so
// that one right-hand side still spreads over the warps.
template <int NT, int NW>
__device__ __forceinline__ void sp_gather(const SolveArgs &a, const int *idx, const int *pm, int n,
                                          int npad, int s0, int ns, double2 *Y) {
  constexpr int ld = 8 * NT + 2;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const double2 zero = make_double2(0.0, 0.0);
  if constexpr (NT == 4) {
    for (int r = lane; r < npad; r += 32) {
      const int d = r < n ? idx[pm ? pm[r] : r] : -1;
#pragma unroll 4
      for (int s = warp; s < 8 * NT; s += NW)
        Y[r * ld + s] = d >= 0 && s < ns ? a.x[(long long)(s0 + s) * a.ndof + d] : zero;
    }
  } else {
    const int nch = (npad + 31) / 32;
#pragma unroll 4
    for (int it = warp; it < nch * ns; it += NW) {
      const int ch = it / ns, s = it - ch * ns, r = 32 * ch + lane;
      double2 v = zero;
      if (r < n) v = a.x[(long long)(s0 + s) * a.ndof + idx[pm ? pm[r] : r]];
      if (r < npad) Y[r * ld + s] = v;
    }
    if (ns < 8 * NT)
      for (int e = threadIdx.x; e < npad * 8 * NT; e += 32 * NW)
        if (e % (8 * NT) >= ns) Y[e / (8 * NT) * ld + e % (8 * NT)] = zero;
  }
}
template <int NT, int NW>
__device__ __forceinline__ void sp_scatter(const SolveArgs &a, const int *idx, const int *pm, int n,
                                           int s0, int ns, const double2 *Y) {
  constexpr int ld = 8 * NT + 2;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if constexpr (NT == 4) {
    for (int r = lane; r < n; r += 32) {
      const int d = idx[pm ? pm[r] : r];
#pragma unroll 4
      for (int s = warp; s < ns; s += NW) a.x[(long long)(s0 + s) * a.ndof + d] = Y[r * ld + s];
    }
  } else {
    const int nch = (n + 31) / 32;
#pragma unroll 4
    for (int it = warp; it < nch * ns; it += NW) {
      const int ch = it / ns, s = it - ch * ns, r = 32 * ch + lane;
      if (r < n) a.x[(long long)(s0 + s) * a.ndof + idx[pm ? pm[r] : r]] = Y[r * ld + s];
    }
  }
}

// rows r0 + lane / 4 of x(rows idx) -= z, by atomics or plainly
template <int NT, bool ATOMIC>
__device__ __forceinline__ void sp_subtract(const SolveArgs &a, const int *idx, int r0, int nr,
                                            int s0, const ZTile (&z)[NT]) {
  const int lane = threadIdx.x & 31, r = r0 + (lane >> 2);
  if (r >= nr) return;
  double2 *row = a.x + idx[r];
#pragma unroll
  for (int t = 0; t < NT; t++)
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int s = s0 + 8 * t + 2 * (lane & 3) + h;
      if (s >= a.nrhs) continue;
      double2 *o = row + (long long)s * a.ndof;
      if (ATOMIC) {
        atomicAdd(&o->x, -z[t].r[h]);
        atomicAdd(&o->y, -z[t].i[h]);
      } else {
        *o = make_double2(o->x - z[t].r[h], o->y - z[t].i[h]);
      }
    }
}

// Triangle of a front held in Y ([kp][8 NT + 2], rows past k zero): blocks of 32
// rows, from the top (lower) or the bottom; NW warps.
template <int NT, int NW>
__device__ __forceinline__ void sp_triangle(const SpStep &st, double2 *Y, bool lower) {
  constexpr int ld = 8 * NT + 2;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, lr = lane >> 2, lk = lane & 3;
  const int kt = (st.k + 7) / 8, nblk = (st.k + 31) / 32;
  for (int b = 0; b < nblk; b++) {
    const int jb = 32 * (lower ? b : nblk - 1 - b), nd = min(4, kt - jb / 8);
    // inverted diagonal block: warp = row tile
    ZTile z[NT];
    if (warp < nd) {
#pragma unroll
      for (int q = 0; q < 8; q++) {
        const bool in = lower ? q <= 2 * warp + 1 : q >= 2 * warp && q < 2 * nd;
        if (in) {
          const double2 v = st.diag(jb + 8 * warp + lr, jb + 4 * q + lk, lower);
#pragma unroll
          for (int t = 0; t < NT; t++) z[t].mma(v, Y[(jb + 4 * q + lk) * ld + 8 * t + lr]);
        }
      }
    }
    __syncthreads();
    if (warp < nd)
#pragma unroll
      for (int t = 0; t < NT; t++)
#pragma unroll
        for (int h = 0; h < 2; h++)
          Y[(jb + 8 * warp + lr) * ld + 8 * t + 2 * lk + h] = make_double2(z[t].r[h], z[t].i[h]);
    __syncthreads();
    // rows still to come
    const int t0 = lower ? jb / 8 + 4 : 0, t1 = lower ? kt : jb / 8;
    for (int ti = t0 + warp; ti < t1; ti += NW) {
      ZTile y[NT];
      sp_product<NT>(st.tri, 8 * ti, st.k, jb, min(32, st.k - jb), Y + jb * ld, y);
#pragma unroll
      for (int t = 0; t < NT; t++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
          double2 *o = Y + (8 * ti + lr) * ld + 8 * t + 2 * lk + h;
          if (8 * ti + lr < st.k) *o = make_double2(o->x - y[t].r[h], o->y - y[t].i[h]);
        }
    }
    __syncthreads();
  }
}

constexpr int kFwdThreads = 128;  // small fronts: CTA per (front, 8 NT right-hand sides)
// more threads where the right-hand sides fill them
template <int NT>
constexpr int kBwdThreads = NT == 4 ? 256 : 128;
constexpr int kChunk = 64;          // boundary rows staged at a time in the backward pass

// Fronts with k <= kSmallK, forward: own rows in shared memory.
template <int NT>
__global__ void __launch_bounds__(kFwdThreads) k_sp_fwd(SolveArgs a) {
  constexpr int NW = kFwdThreads / 32;
  extern __shared__ double2 Y[];
  const SpFront f = a.fr[a.fronts[blockIdx.x]];
  if (f.k == 0) return;
  const SpStep st(a, f, true);
  const int s0 = blockIdx.y * 8 * NT, ns = min(8 * NT, a.nrhs - s0), kp = (f.k + 7) & ~7;
  const int *ow = a.own + f.own0, *bd = a.bnd + f.bnd0;
  sp_gather<NT, NW>(a, ow, a.trans ? nullptr : a.perm + f.own0, f.k, kp, s0, ns, Y);
  __syncthreads();
  sp_triangle<NT, NW>(st, Y, true);
  sp_scatter<NT, NW>(a, ow, nullptr, f.k, s0, ns, Y);
  for (int r0 = 8 * (threadIdx.x >> 5); r0 < f.m; r0 += 8 * NW) {
    ZTile z[NT];
    sp_product<NT>(st.rect, r0, f.m, 0, f.k, Y, z);
    sp_subtract<NT, true>(a, bd, r0, f.m, s0, z);
  }
}

// The same, backward: boundary rows staged in chunks, then the triangle.
template <int NT>
__global__ void __launch_bounds__(kBwdThreads<NT>, 512 / kBwdThreads<NT>) k_sp_bwd(SolveArgs a) {
  constexpr int ld = 8 * NT + 2, NW = kBwdThreads<NT> / 32;
  constexpr int kMine = (sp::kSmallK / 8 + NW - 1) / NW;  // row tiles of a warp
  extern __shared__ double2 Y[];
  const SpFront f = a.fr[a.fronts[blockIdx.x]];
  if (f.k == 0) return;
  const SpStep st(a, f, false);
  const int s0 = blockIdx.y * 8 * NT, ns = min(8 * NT, a.nrhs - s0), kp = (f.k + 7) & ~7;
  double2 *xb = Y + kp * ld;  // [kChunk][ld]
  const int *ow = a.own + f.own0, *bd = a.bnd + f.bnd0;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, lr = lane >> 2, lk = lane & 3;
  sp_gather<NT, NW>(a, ow, nullptr, f.k, kp, s0, ns, Y);
  ZTile z[kMine][NT];
  for (int c0 = 0; c0 < f.m; c0 += kChunk) {
    const int nc = min(kChunk, f.m - c0);
    __syncthreads();
    sp_gather<NT, NW>(a, bd + c0, nullptr, nc, (nc + 3) & ~3, s0, ns, xb);
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kMine; q++)
      if (8 * (warp + NW * q) < f.k)
        sp_product<NT>(st.rect, 8 * (warp + NW * q), f.k, c0, nc, xb, z[q]);
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < kMine; q++) {
    const int r = 8 * (warp + NW * q) + lr;
    if (r < f.k)
#pragma unroll
      for (int t = 0; t < NT; t++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
          double2 *o = Y + r * ld + 8 * t + 2 * lk + h;
          *o = make_double2(o->x - z[q][t].r[h], o->y - z[q][t].i[h]);
        }
  }
  __syncthreads();
  sp_triangle<NT, NW>(st, Y, false);
  sp_scatter<NT, NW>(a, ow, a.trans ? a.perm + f.own0 : nullptr, f.k, s0, ns, Y);
}

constexpr int kTriThreads = 512;
constexpr size_t kTriSmemMax = 200 * 1024;

// Larger fronts: their triangle, a CTA per (front, gc <= 8 right-hand sides) with
// all own rows in shared memory ([kp][ldx]), gc the most that fit.  Block by
// block of 32 rows, left-looking: the rows' products with everything solved so
// far are split over four groups of warps by columns (the factor's entries loaded
// a chunk ahead, across the barriers too), summed through shared memory, then the
// inverted diagonal block.  Right-looking in place in x each block waited
// for a round of x loads and stores: 370 us for 720 rows, 24 blocks; this takes
// 170 us.
__global__ void __launch_bounds__(kTriThreads) k_sp_tri(SolveArgs a, int fwd, int gc, int ldx) {
  extern __shared__ double2 X[];
  __shared__ double2 part[4][32][9];
  const SpFront f = a.fr[a.fronts[blockIdx.x]];
  if (f.k == 0) return;
  const SpStep st(a, f, fwd);
  const bool lower = fwd;
  const int s0 = blockIdx.y * gc, ns = min(gc, a.nrhs - s0), k = f.k;
  const int *ow = a.own + f.own0, *pm = a.perm + f.own0;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, lr = lane >> 2, lk = lane & 3;
  const int rt = warp & 3, ks = warp >> 2;  // row tile, group of columns
  const int kp = (k + 31) & ~31, nblk = kp / 32;
  const bool perm_in = fwd && a.trans == 0, perm_out = !fwd && a.trans != 0;
  const double2 zero = make_double2(0.0, 0.0);
  for (int e = tid; e < kp * gc; e += kTriThreads) {
    const int r = e % kp, s = e / kp;
    X[r * ldx + s] = r < k && s < ns
                         ? a.x[(long long)(s0 + s) * a.ndof + ow[perm_in ? pm[r] : r]]
                         : zero;
  }
  // Rows and columns past k read the last ones instead: such rows are not kept,
  // such columns meet the zero rows of X.
  const long long cs = st.tri.cs, cs4 = 4 * cs;
  auto load = [&](double2 (&v)[8], int jb, int c) {  // 32 columns from c of the row tile
    const double2 *row = st.tri.p + (long long)min(jb + 8 * rt + lr, k - 1) * st.tri.rs;
    if (c + 32 <= k) {
      const double2 *p = row + (c + lk) * cs;
#pragma unroll
      for (int q = 0; q < 8; q++) v[q] = __ldg(p + q * cs4);
    } else {
#pragma unroll
      for (int q = 0; q < 8; q++) v[q] = __ldg(row + min(c + 4 * q + lk, k - 1) * cs);
    }
  };
  const double2 *Xl = X + lk * ldx + (lr < gc ? lr : 0);
  auto product = [&](ZTile (&z)[2], const double2 (&v)[8], int c) {
    const double2 *xc = Xl + c * ldx;
#pragma unroll
    for (int q = 0; q < 8; q++) {
      double2 b = xc[4 * q * ldx];
      if (lr >= gc) b = zero;
      z[q & 1].mma(make_double2(v[q].x, st.tri.sg * v[q].y), b);
    }
  };
  auto first = [&](int b) { return 32 * (lower ? b : nblk - 1 - b); };
  double2 va[8], vb[8], dv[8];
  if (ks == 0) load(dv, first(0), first(0));
  __syncthreads();
  for (int b = 0; b < nblk; b++) {
    const int jb = first(b), r0 = jb + 8 * rt;
    const int c1 = lower ? jb : kp;  // columns solved so far: [0, jb) or [jb + 32, kp)
    int c = (lower ? 0 : jb + 32) + 32 * ks;
    ZTile z[2];
    while (c < c1) {  // va holds the columns from c
      if (c + 128 < c1) load(vb, jb, c + 128);
      product(z, va, c);
      c += 128;
      if (c >= c1) break;
      if (c + 128 < c1) load(va, jb, c + 128);
      product(z, vb, c);
      c += 128;
    }
#pragma unroll
    for (int h = 0; h < 2; h++)
      part[ks][8 * rt + lr][2 * lk + h] =
          make_double2(z[0].r[h] + z[1].r[h], z[0].i[h] + z[1].i[h]);
    // the next block's first columns are on their way during what follows
    const int jn = first(b + 1), cn = (lower ? 0 : jn + 32) + 32 * ks;
    if (b + 1 < nblk && cn < (lower ? jn : kp)) load(va, jn, cn);
    __syncthreads();
    if (tid < 256) {
      const int r = tid >> 3, s = tid & 7;
      if (s < gc && jb + r < k) {
        double2 *o = X + (jb + r) * ldx + s;
        double2 v = *o;
#pragma unroll
        for (int q = 0; q < 4; q++) {
          v.x -= part[q][r][s].x;
          v.y -= part[q][r][s].y;
        }
        *o = v;
      }
    }
    __syncthreads();
    if (ks == 0) {
      ZTile y[2];
#pragma unroll
      for (int q = 0; q < 8; q++) {
        const int r = 8 * rt + lr, cc = 4 * q + lk;
        if (lower ? cc > r : cc < r) dv[q] = zero;
        if (cc == r && st.unit) dv[q] = make_double2(1.0, 0.0);
      }
      product(y, dv, jb);
      if (b + 1 < nblk) load(dv, jn, jn);
      // the first four warps have all read the block before they overwrite it
      asm volatile("bar.sync 1, 128;" ::: "memory");
      if (r0 + lr < k)
#pragma unroll
        for (int h = 0; h < 2; h++)
          if (2 * lk + h < gc)
            X[(r0 + lr) * ldx + 2 * lk + h] =
                make_double2(y[0].r[h] + y[1].r[h], y[0].i[h] + y[1].i[h]);
    }
    __syncthreads();
  }
  for (int e = tid; e < k * ns; e += kTriThreads) {
    const int r = e % k, s = e / k;
    a.x[(long long)(s0 + s) * a.ndof + ow[perm_out ? pm[r] : r]] = X[r * ldx + s];
  }
}

// Fronts whose rows do not fit shared memory keep them in x: the permutation of P
// (inv = 0) or P^T, a CTA per (front, right-hand side) with the old values in
// shared memory; beyond what fits, one thread replays the interchanges.
constexpr int kPermMax = 14000;
__global__ void k_sp_permute(SolveArgs a, const int *__restrict__ swap, int inv) {
  extern __shared__ double2 Y[];
  const SpFront f = a.fr[a.fronts[blockIdx.x]];
  const int *ow = a.own + f.own0, *pm = a.perm + f.own0, *sw = swap + f.own0;
  for (int s = blockIdx.y; s < a.nrhs; s += gridDim.y) {
    double2 *x = a.x + (long long)s * a.ndof;
    if (f.k > kPermMax) {
      if (threadIdx.x == 0)
        for (int q = 0; q < f.k; q++) {
          const int j = inv ? f.k - 1 - q : q;
          const double2 v = x[ow[j]];
          x[ow[j]] = x[ow[sw[j]]];
          x[ow[sw[j]]] = v;
        }
      continue;
    }
    for (int r = threadIdx.x; r < f.k; r += blockDim.x) Y[r] = x[ow[r]];
    __syncthreads();
    for (int r = threadIdx.x; r < f.k; r += blockDim.x)
      if (inv)
        x[ow[pm[r]]] = Y[r];
      else
        x[ow[r]] = Y[pm[r]];
    __syncthreads();
  }
}

// Their triangle, a CTA per (front, 8 NT right-hand sides): the block being
// solved in shared memory, the rows still to come updated in x.
template <int NT>
__global__ void __launch_bounds__(kTriThreads) k_sp_tri_any(SolveArgs a, int fwd) {
  constexpr int ld = 8 * NT + 2, NW = kTriThreads / 32;
  __shared__ double2 Y[32 * ld];
  const SpFront f = a.fr[a.fronts[blockIdx.x]];
  const SpStep st(a, f, fwd);
  const bool lower = fwd;
  const int s0 = blockIdx.y * 8 * NT, ns = min(8 * NT, a.nrhs - s0), k = f.k;
  const int *ow = a.own + f.own0;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, lr = lane >> 2, lk = lane & 3;
  const int kt = (k + 7) / 8, nblk = (k + 31) / 32;
  for (int b = 0; b < nblk; b++) {
    const int jb = 32 * (lower ? b : nblk - 1 - b), nd = min(4, kt - jb / 8);
    for (int e = tid; e < 32 * 8 * NT; e += kTriThreads) {
      const int r = e % 32, s = e / 32;
      double2 v = make_double2(0.0, 0.0);
      if (jb + r < k && s < ns) v = a.x[(long long)(s0 + s) * a.ndof + ow[jb + r]];
      Y[r * ld + s] = v;
    }
    __syncthreads();
    ZTile z[NT];
    if (warp < nd) {
#pragma unroll
      for (int q = 0; q < 8; q++) {
        const bool in = lower ? q <= 2 * warp + 1 : q >= 2 * warp && q < 2 * nd;
        if (in) {
          const double2 v = st.diag(jb + 8 * warp + lr, jb + 4 * q + lk, lower);
#pragma unroll
          for (int t = 0; t < NT; t++) z[t].mma(v, Y[(4 * q + lk) * ld + 8 * t + lr]);
        }
      }
    }
    __syncthreads();
    if (warp < nd) {
      const int r = jb + 8 * warp + lr;
#pragma unroll
      for (int t = 0; t < NT; t++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int s = 8 * t + 2 * lk + h;
          const double2 v = make_double2(z[t].r[h], z[t].i[h]);
          Y[(8 * warp + lr) * ld + s] = v;
          if (r < k && s < ns) a.x[(long long)(s0 + s) * a.ndof + ow[r]] = v;
        }
    }
    __syncthreads();
    const int t0 = lower ? jb / 8 + 4 : 0, t1 = lower ? kt : jb / 8;
    for (int ti = t0 + warp; ti < t1; ti += NW) {
      ZTile y[NT];
      sp_product<NT>(st.tri, 8 * ti, k, jb, min(32, k - jb), Y, y);
      sp_subtract<NT, false>(a, ow, 8 * ti, k, s0, y);
    }
    __syncthreads();
  }
}

// Their rectangle, 64 rows a CTA over blockIdx.y (a warp per 8), the right-hand
// side of the summed index staged in chunks: forward x_b -= rect y (atomics),
// backward y -= rect x_b.
template <int NT>
__global__ void __launch_bounds__(256) k_sp_rect(SolveArgs a, int fwd) {
  // longer chunks where the columns are few: 40 KB of shared memory for any NT
  constexpr int ld = 8 * NT + 2, kChunk = 256 / NT;
  __shared__ double2 Y[kChunk * ld];
  const SpFront f = a.fr[a.fronts[blockIdx.x]];
  const SpStep st(a, f, fwd);
  const int rows = fwd ? f.m : f.k, cols = fwd ? f.k : f.m;
  if (64 * (int)blockIdx.y >= rows || cols == 0) return;
  const int *ri = fwd ? a.bnd + f.bnd0 : a.own + f.own0;
  const int *ci = fwd ? a.own + f.own0 : a.bnd + f.bnd0;
  const int s0 = blockIdx.z * 8 * NT, ns = min(8 * NT, a.nrhs - s0);
  const int tid = threadIdx.x, r0 = 64 * blockIdx.y + 8 * (tid >> 5);
  ZTile z[NT];
  for (int c0 = 0; c0 < cols; c0 += kChunk) {
    const int nc = min(kChunk, cols - c0);
    __syncthreads();
    sp_gather<NT, 8>(a, ci + c0, nullptr, nc, (nc + 3) & ~3, s0, ns, Y);
    __syncthreads();
    if (r0 < rows) sp_product<NT>(st.rect, r0, rows, c0, nc, Y, z);
  }
  if (r0 >= rows) return;
  if (fwd)
    sp_subtract<NT, true>(a, ri, r0, rows, s0, z);
  else
    sp_subtract<NT, false>(a, ri, r0, rows, s0, z);
}

// ---------------------------------------------------------------------------
// host drivers
// ---------------------------------------------------------------------------
void free_sparse(Ctx *c) {
  SparseLU *s = c->sparse;
  if (!s) return;
  void *ptrs[] = {s->d_fr,   s->d_own,  s->d_bnd,  s->d_pull,    s->d_lev_fronts, s->d_ent_idx,
                  s->d_ent_loc, s->d_fac, s->d_perm, s->d_swap, s->d_work[0], s->d_work[1],
                  s->d_info};
  for (void *p : ptrs)
    if (p) cudaFree(p);
  for (int g = 0; g < sp::kStreams; g++) {
    for (cudaStream_t q : {s->st[g], s->side[g]})
      if (q) cudaStreamDestroy(q);
    for (cudaEvent_t q : {s->done[g], s->applied[g], s->updated[g]})
      if (q) cudaEventDestroy(q);
  }
  if (s->ready) cudaEventDestroy(s->ready);
  delete s;
  c->sparse = nullptr;
}

void sparse_info(const Ctx *c, long long *out) {
  const SparseLU *s = c->sparse;
  if (!s) {
    for (int i = 0; i < 7; i++) out[i] = 0;
    return;
  }
  plan_stats(s->fr, s->fac_elems, s->lev_work, out);
}

#define SPCK(expr, what)                                                   \
  do {                                                                     \
    cudaError_t e_ = (expr);                                               \
    if (e_ != cudaSuccess) {                                               \
      *msg = std::string("sparse solve: ") + (what) + ": " + cudaGetErrorString(e_); \
      return e_ == cudaErrorMemoryAllocation ? FEM25_ERR_ALLOC : FEM25_ERR_CUDA;     \
    }                                                                      \
  } while (0)

template <int NT>
static cudaError_t sparse_solve_attributes() {
  constexpr size_t row = sizeof(double2) * (8 * NT + 2);
  const cudaError_t e = cudaFuncSetAttribute(
      k_sp_fwd<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(row * sp::kSmallK));
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(k_sp_bwd<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)(row * (sp::kSmallK + kChunk)));
}

static int sparse_factor_run(Ctx *c, const double *csr128, cudaStream_t st, std::string *msg) {
  if (!c->sparse) c->sparse = new SparseLU();
  SparseLU *s = c->sparse;
  s->factored = false;
  if (!s->analysed) {
    const int r = sparse_analyse(c, s, st, msg);
    if (r) return r;
  }
  SPCK(sparse_factor_attributes(), "kernel attributes");
  SPCK(cudaFuncSetAttribute(k_sp_permute, cudaFuncAttributeMaxDynamicSharedMemorySize,
                            (int)(sizeof(double2) * kPermMax)),
       "kernel attributes");
  SPCK(cudaFuncSetAttribute(k_sp_tri, cudaFuncAttributeMaxDynamicSharedMemorySize,
                            (int)kTriSmemMax),
       "kernel attributes");
  SPCK(sparse_solve_attributes<1>(), "kernel attributes");
  SPCK(sparse_solve_attributes<2>(), "kernel attributes");
  SPCK(sparse_solve_attributes<4>(), "kernel attributes");
  // streams, events and buffers each by itself: a call after one that failed makes what
  // is missing
  if (!s->ready) {
    // the groups' own streams go before their side streams: a panel must not queue
    // behind the update beside it
    int least = 0, greatest = 0;
    SPCK(cudaDeviceGetStreamPriorityRange(&least, &greatest), "streams");
    auto stream = [](cudaStream_t *q, int priority) {
      return *q ? cudaSuccess : cudaStreamCreateWithPriority(q, cudaStreamNonBlocking, priority);
    };
    auto event = [](cudaEvent_t *q) {
      return *q ? cudaSuccess : cudaEventCreateWithFlags(q, cudaEventDisableTiming);
    };
    for (int g = 0; g < sp::kStreams; g++) {
      SPCK(stream(&s->st[g], greatest), "streams");
      SPCK(stream(&s->side[g], least), "streams");
      for (cudaEvent_t *q : {&s->done[g], &s->applied[g], &s->updated[g]}) SPCK(event(q), "events");
    }
    SPCK(event(&s->ready), "events");
  }
  auto keep = [](auto **p, size_t n) {
    return *p ? cudaSuccess : cudaMalloc(p, sizeof(**p) * std::max(n, (size_t)1));
  };
  SPCK(keep(&s->d_fac, (size_t)s->fac_elems), "factor store");
  SPCK(keep(&s->d_perm, (size_t)c->ndof), "pivots");
  SPCK(keep(&s->d_swap, (size_t)c->ndof), "pivots");
  SPCK(keep(&s->d_work[0], (size_t)s->max_work), "work");
  SPCK(keep(&s->d_work[1], (size_t)s->max_work), "work");
  SPCK(keep(&s->d_info, 1), "status");
  SPCK(cudaMemsetAsync(s->d_info, 0, sizeof(int), st), "status");
  const double2 *csr = reinterpret_cast<const double2 *>(csr128);
  int nsm = 0;
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, c->device);
  for (int l = s->nlevel - 1; l >= 0; l--)  // from the leaves
    SPCK(sparse_factor_level(s, l, csr, s->d_work[l & 1], s->d_work[(l + 1) & 1], nsm, st),
         "factorisation");
  // zero pivots of any front
  int info = 0;
  SPCK(cudaMemcpyAsync(&info, s->d_info, sizeof(int), cudaMemcpyDeviceToHost, st), "status");
  SPCK(cudaStreamSynchronize(st), "factorisation");
  if (info != 0) {
    *msg = "sparse solve: zero pivot in front " + std::to_string(info - 1) +
           " (matrix singular to working precision)";
    return FEM25_ERR_ARG;
  }
  s->factored = true;
  return 0;
}

int sparse_factor(Ctx *c, const double *csr128, cudaStream_t st, std::string *msg) {
  const int r = sparse_factor_run(c, csr128, st, msg);
  if (r) {  // nothing of this call outlives it: a level may have stopped between its streams
    for (int g = 0; g < sp::kStreams; g++)
      for (cudaStream_t q : {c->sparse->st[g], c->sparse->side[g]})
        if (q) cudaStreamSynchronize(q);
    cudaStreamSynchronize(st);
  }
  return r;
}

// One level's launches of a pass, 8 NT right-hand sides a CTA
template <int NT>
static cudaError_t sparse_solve_level(const SparseLU *s, SolveArgs a, int l, bool fwd,
                                      cudaStream_t st) {
  const unsigned groups = (unsigned)((a.nrhs + 8 * NT - 1) / (8 * NT));
  const int nsmall = s->lev_nsmall[l], nbig = (int)s->lev[l].size() - nsmall;
  constexpr size_t row = sizeof(double2) * (8 * NT + 2);
  a.fronts = s->d_lev_fronts + s->lev_off[l];
  if (nsmall > 0 && s->lev_ksmall[l] > 0) {
    const size_t kp = (size_t)(s->lev_ksmall[l] + 7) & ~7;
    if (fwd)
      k_sp_fwd<NT><<<dim3(nsmall, groups), kFwdThreads, row * kp, st>>>(a);
    else
      k_sp_bwd<NT><<<dim3(nsmall, groups), kBwdThreads<NT>, row * (kp + kChunk), st>>>(a);
  }
  if (nbig > 0) {
    a.fronts += nsmall;
    const int kmax = s->lev_kmax[l], mmax = s->lev_mmax[l];
    const dim3 rect(nbig, ((fwd ? mmax : kmax) + 63) / 64, groups);
    // right-hand sides of a triangle's CTA: 8, or fewer so that the largest
    // front's rows fit (strides without bank conflicts); FEM25_PANEL_WIDTH=1
    // selects the any-size kernels, as in the factorisation
    const size_t kp = (size_t)(kmax + 31) & ~31;
    int gc = 8;
    auto ldx = [](int g) { return g > 2 ? g + 2 : g; };
    while (gc > 1 && (a.nrhs <= gc / 2 || sizeof(double2) * kp * ldx(gc) > kTriSmemMax)) gc /= 2;
    const char *env = std::getenv("FEM25_PANEL_WIDTH");
    const bool any = sizeof(double2) * kp * ldx(gc) > kTriSmemMax || (env && std::atoi(env) == 1);
    const dim3 perm(nbig, std::min(a.nrhs, 65535));
    const size_t psm = sizeof(double2) * (size_t)std::min(kmax, kPermMax);
    if (!fwd && mmax > 0) k_sp_rect<NT><<<rect, 256, 0, st>>>(a, 0);
    if (any) {
      if (fwd && a.trans == 0) k_sp_permute<<<perm, 256, psm, st>>>(a, s->d_swap, 0);
      k_sp_tri_any<NT><<<dim3(nbig, groups), kTriThreads, 0, st>>>(a, fwd);
      if (!fwd && a.trans != 0) k_sp_permute<<<perm, 256, psm, st>>>(a, s->d_swap, 1);
    } else {
      k_sp_tri<<<dim3(nbig, (a.nrhs + gc - 1) / gc), kTriThreads, sizeof(double2) * kp * ldx(gc),
                 st>>>(a, fwd, gc, ldx(gc));
    }
    if (fwd && mmax > 0) k_sp_rect<NT><<<rect, 256, 0, st>>>(a, 1);
  }
  return cudaGetLastError();
}

int sparse_solve(Ctx *c, int nrhs, int trans, double *rhs, cudaStream_t st, std::string *msg) {
  SparseLU *s = c->sparse;
  if (!s || !s->factored) {
    *msg = "sparse solve: no factorisation (call fem25_sparse_factor_dev first)";
    return FEM25_ERR_ARG;
  }
  SolveArgs a{nullptr, s->d_fr, s->d_own, s->d_bnd, s->d_fac, s->d_perm,
              reinterpret_cast<double2 *>(rhs), c->ndof, nrhs, trans};
  int nsm = 0;
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, c->device);
  // Right-hand sides a CTA: as many as there are, up to 32, so that the factors
  // are read once; fewer where a level has too few fronts to fill the GPU.
  const int most = nrhs <= 8 ? 1 : nrhs <= 16 ? 2 : 4;
  for (int pass = 0; pass < 2; pass++)
    for (int q = 0; q < s->nlevel; q++) {
      const bool fwd = pass == 0;
      const int l = fwd ? s->nlevel - 1 - q : q;  // forward from the leaves, back from the root
      const long long nf = (long long)s->lev[l].size();
      int nt = most;
      while (nt > 1 && nf * ((nrhs + 8 * nt - 1) / (8 * nt)) < 2 * nsm) nt /= 2;
      SPCK(nt == 1   ? sparse_solve_level<1>(s, a, l, fwd, st)
           : nt == 2 ? sparse_solve_level<2>(s, a, l, fwd, st)
                     : sparse_solve_level<4>(s, a, l, fwd, st),
           "solve");
    }
  SPCK(cudaGetLastError(), "solve");
  return 0;
}

}  // namespace fem25
