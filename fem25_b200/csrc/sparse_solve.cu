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
#include <numeric>

#include "sparse.cuh"

namespace fem25 {

namespace {
constexpr int kThreads = 256;
constexpr int kRhsPerCta = 8;  // right-hand sides per solve CTA
}  // namespace

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
// The triangular solves of one front, blocked by 32 rows: warp 0 solves the
// 32 x 32 diagonal triangle of a block with the block's right-hand-side
// values in registers (lane = row; values passed on by shuffles), the CTA
// then updates the rows still to come with the solved block (kept in shared
// memory): two CTA barriers per 32 rows.  Row r of the own block is the DOF
// own[r]; the right-hand sides [r0, r0 + nr) of x (one CTA per group of
// kRhsPerCta).
//   op(A) = A    forward: interchanges, L11 (unit lower), x_b -= L21 x_own
//                backward: x_own -= U12 x_b, U11 (upper)
//   A^T / A^H    forward: U11^op (lower), x_b -= U12^op x_own
//                backward: x_own -= L21^op x_b, L11^op (unit upper), inverse
//                interchanges
// The boundary rows x_b of a front belong to ancestors; fronts of one level
// may share them, so the forward updates add with atomics.
struct SolveArgs {
  const int *fronts;
  const SpFront *fr;
  const int *own, *bnd;
  const double2 *fac;
  const int *swap;
  double2 *x;
  int ndof, nrhs, trans;  // trans 0: A, 1: A^T, 2: A^H
};

__device__ __forceinline__ double2 sp_op(double2 v, int trans) {
  return trans == 2 ? cconj(v) : v;
}

// element (i, j) of op(T) for the front's F11 (ld n) or L21 rows: op(T)(i, j)
// = T(i, j) for A, T(j, i) (conjugated for A^H) for A^T / A^H
__device__ __forceinline__ double2 sp_el(const double2 *T, long long n, int i, int j, int trans) {
  return trans == 0 ? T[i + (long long)j * n] : sp_op(T[j + (long long)i * n], trans);
}

template <int R>
__global__ void __launch_bounds__(kThreads) k_sp_solve_fwd(SolveArgs a) {
  __shared__ double2 xs[32][R];
  __shared__ double2 tb[32][33];  // the block's diagonal triangle, op applied
  const SpFront f = a.fr[a.fronts[blockIdx.x]];
  const int r0 = blockIdx.y * R, nr = min(R, a.nrhs - r0);
  if (nr <= 0 || f.k == 0) return;
  const long long n = (long long)f.k + f.m;
  const int k = f.k, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int *ow = a.own + f.own0;
  const double2 *F = a.fac + f.fac0;          // F11 and L21, ld n
  double2 *x = a.x + (long long)r0 * a.ndof;
  const int tr = a.trans;
  if (tr == 0 && tid < nr) {  // row interchanges of P
    double2 *xr = x + (long long)tid * a.ndof;
    for (int j = 0; j < k; j++) {
      const int p = a.swap[f.own0 + j];
      if (p != j) {
        const double2 t = xr[ow[j]];
        xr[ow[j]] = xr[ow[p]];
        xr[ow[p]] = t;
      }
    }
  }
  __syncthreads();
  // lower triangle T: L11 (unit) for A, U11^op (non-unit) for A^T / A^H
  for (int jb = 0; jb < k; jb += 32) {
    const int nb = min(32, k - jb);
    for (int q = tid; q < nb * nb; q += blockDim.x) {
      const int i = q % nb, j = q / nb;
      if (i > j) tb[i][j] = sp_el(F, n, jb + i, jb + j, tr);
      if (i == j) tb[i][i] = tr != 0 ? sp_el(F, n, jb + i, jb + i, tr) : make_double2(1.0, 0.0);
    }
    __syncthreads();
    if (warp == 0) {
      double2 v[R];
#pragma unroll
      for (int s = 0; s < R; s++)
        v[s] = (lane < nb && s < nr) ? x[(long long)s * a.ndof + ow[jb + lane]] : make_double2(0.0, 0.0);
      double2 y[R];
#pragma unroll
      for (int s = 0; s < R; s++) y[s] = make_double2(0.0, 0.0);
      for (int i = 0; i < nb; i++) {  // times the inverted triangle
        const double2 tli = lane >= i && lane < nb ? tb[lane][i] : make_double2(0.0, 0.0);
#pragma unroll
        for (int s = 0; s < R; s++) {
          const double2 xi = make_double2(-__shfl_sync(0xffffffffu, v[s].x, i),
                                          -__shfl_sync(0xffffffffu, v[s].y, i));
          y[s] = cfms(y[s], tli, xi);
        }
      }
#pragma unroll
      for (int s = 0; s < R; s++) v[s] = y[s];
      if (lane < nb)
#pragma unroll
        for (int s = 0; s < R; s++)
          if (s < nr) {
            x[(long long)s * a.ndof + ow[jb + lane]] = v[s];
            xs[lane][s] = v[s];
          }
    }
    __syncthreads();
    for (int r = jb + nb + tid; r < k; r += blockDim.x) {
      double2 acc[R];
#pragma unroll
      for (int s = 0; s < R; s++)
        acc[s] = s < nr ? x[(long long)s * a.ndof + ow[r]] : make_double2(0.0, 0.0);
      for (int i = 0; i < nb; i++) {
        const double2 t = sp_el(F, n, r, jb + i, tr);
#pragma unroll
        for (int s = 0; s < R; s++) acc[s] = cfms(acc[s], t, xs[i][s]);
      }
#pragma unroll
      for (int s = 0; s < R; s++)
        if (s < nr) x[(long long)s * a.ndof + ow[r]] = acc[s];
    }
    __syncthreads();
  }
}

// The rectangular part of a front's solve step, spread over CTAs of
// kThreads rows each (blockIdx.y: row tile, blockIdx.z: group of
// right-hand sides):
//   fwd: boundary rows   x_b -= L21 x_own (A), U12^op x_own (A^T / A^H),
//        added with atomics (fronts of a level share boundary rows)
//   bwd: own rows        x_own -= U12 x_b (A), L21^op x_b (A^T / A^H)
// The right-hand-side values of the summed index pass through shared memory
// in chunks of kThreads, so each thread's dot product streams its matrix row.
template <int R>
__global__ void __launch_bounds__(kThreads) k_sp_solve_rect(SolveArgs a, int fwd) {
  __shared__ double2 xc[kThreads][R];
  const SpFront f = a.fr[a.fronts[blockIdx.x]];
  const int r0 = blockIdx.z * R, nr = min(R, a.nrhs - r0);
  const int rows = fwd ? f.m : f.k, cols = fwd ? f.k : f.m;
  const int row0 = blockIdx.y * blockDim.x;
  if (nr <= 0 || row0 >= rows || cols == 0) return;
  const long long n = (long long)f.k + f.m;
  const int k = f.k, tid = threadIdx.x, tr = a.trans;
  const double2 *F = a.fac + f.fac0, *U12 = F + n * k;
  const int *rowidx = (fwd ? a.bnd + f.bnd0 : a.own + f.own0);
  const int *colidx = (fwd ? a.own + f.own0 : a.bnd + f.bnd0);
  double2 *x = a.x + (long long)r0 * a.ndof;
  const int r = row0 + tid;
  double2 acc[R];
#pragma unroll
  for (int s = 0; s < R; s++) acc[s] = make_double2(0.0, 0.0);
  for (int c0 = 0; c0 < cols; c0 += blockDim.x) {
    const int nc = min((int)blockDim.x, cols - c0);
    __syncthreads();
    if (tid < nc) {
      const int d = colidx[c0 + tid];
#pragma unroll
      for (int s = 0; s < R; s++)
        xc[tid][s] = s < nr ? x[(long long)s * a.ndof + d] : make_double2(0.0, 0.0);
    }
    __syncthreads();
    if (r < rows) {
#pragma unroll 4
      for (int j = 0; j < nc; j++) {
        const int c = c0 + j;
        // element (r, c) of the rectangular block
        double2 t;
        if (fwd)
          t = tr == 0 ? F[k + r + (long long)c * n] : sp_op(U12[c + (long long)r * k], tr);
        else
          t = tr == 0 ? U12[r + (long long)c * k] : sp_op(F[k + c + (long long)r * n], tr);
#pragma unroll
        for (int s = 0; s < R; s++) acc[s] = cfms(acc[s], t, xc[j][s]);
      }
    }
  }
  if (r >= rows) return;
  const int d = rowidx[r];
#pragma unroll
  for (int s = 0; s < R; s++)
    if (s < nr) {
      double2 *o = x + (long long)s * a.ndof + d;
      if (fwd) {  // acc = -(product)
        atomicAdd(reinterpret_cast<double *>(o), acc[s].x);
        atomicAdd(reinterpret_cast<double *>(o) + 1, acc[s].y);
      } else {
        *o = make_double2(o->x + acc[s].x, o->y + acc[s].y);
      }
    }
}

template <int R>
__global__ void __launch_bounds__(kThreads) k_sp_solve_bwd(SolveArgs a) {
  __shared__ double2 xs[32][R];
  __shared__ double2 tb[32][33];  // the block's diagonal triangle, op applied
  const SpFront f = a.fr[a.fronts[blockIdx.x]];
  const int r0 = blockIdx.y * R, nr = min(R, a.nrhs - r0);
  if (nr <= 0 || f.k == 0) return;
  const long long n = (long long)f.k + f.m;
  const int k = f.k, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int *ow = a.own + f.own0;
  const double2 *F = a.fac + f.fac0;
  double2 *x = a.x + (long long)r0 * a.ndof;
  const int tr = a.trans;
  // upper triangle T: U11 (non-unit) for A, L11^op (unit) for A^T / A^H;
  // blocks of 32 rows from the bottom
  for (int jb = ((k - 1) / 32) * 32; jb >= 0; jb -= 32) {
    const int nb = min(32, k - jb);
    for (int q = tid; q < nb * nb; q += blockDim.x) {
      const int i = q % nb, j = q / nb;
      if (i < j) tb[i][j] = sp_el(F, n, jb + i, jb + j, tr);
      if (i == j) tb[i][i] = tr == 0 ? sp_el(F, n, jb + i, jb + i, tr) : make_double2(1.0, 0.0);
    }
    __syncthreads();
    if (warp == 0) {
      double2 v[R];
#pragma unroll
      for (int s = 0; s < R; s++)
        v[s] = (lane < nb && s < nr) ? x[(long long)s * a.ndof + ow[jb + lane]] : make_double2(0.0, 0.0);
      double2 y[R];
#pragma unroll
      for (int s = 0; s < R; s++) y[s] = make_double2(0.0, 0.0);
      for (int i = 0; i < nb; i++) {  // times the inverted triangle
        const double2 tli = lane <= i ? tb[lane][i] : make_double2(0.0, 0.0);
#pragma unroll
        for (int s = 0; s < R; s++) {
          const double2 xi = make_double2(-__shfl_sync(0xffffffffu, v[s].x, i),
                                          -__shfl_sync(0xffffffffu, v[s].y, i));
          y[s] = cfms(y[s], tli, xi);
        }
      }
#pragma unroll
      for (int s = 0; s < R; s++) v[s] = y[s];
      if (lane < nb)
#pragma unroll
        for (int s = 0; s < R; s++)
          if (s < nr) {
            x[(long long)s * a.ndof + ow[jb + lane]] = v[s];
            xs[lane][s] = v[s];
          }
    }
    __syncthreads();
    for (int r = tid; r < jb; r += blockDim.x) {
      double2 acc[R];
#pragma unroll
      for (int s = 0; s < R; s++)
        acc[s] = s < nr ? x[(long long)s * a.ndof + ow[r]] : make_double2(0.0, 0.0);
      for (int i = 0; i < nb; i++) {
        const double2 t = sp_el(F, n, r, jb + i, tr);
#pragma unroll
        for (int s = 0; s < R; s++) acc[s] = cfms(acc[s], t, xs[i][s]);
      }
#pragma unroll
      for (int s = 0; s < R; s++)
        if (s < nr) x[(long long)s * a.ndof + ow[r]] = acc[s];
    }
    __syncthreads();
  }
  if (tr != 0 && tid < nr) {  // inverse row interchanges
    double2 *xr = x + (long long)tid * a.ndof;
    for (int j = k - 1; j >= 0; j--) {
      const int p = a.swap[f.own0 + j];
      if (p != j) {
        const double2 t = xr[ow[j]];
        xr[ow[j]] = xr[ow[p]];
        xr[ow[p]] = t;
      }
    }
  }
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

int sparse_factor(Ctx *c, const double *csr128, cudaStream_t st, std::string *msg) {
  if (!c->sparse) c->sparse = new SparseLU();
  SparseLU *s = c->sparse;
  s->factored = false;
  if (!s->analysed) {
    const int r = sparse_analyse(c, s, st, msg);
    if (r) return r;
  }
  SPCK(sparse_factor_attributes(), "kernel attributes");
  if (!s->d_fac) {
    SPCK(cudaMalloc(&s->d_fac, sizeof(double2) * std::max(s->fac_elems, 1LL)), "factor store");
    SPCK(cudaMalloc(&s->d_perm, sizeof(int) * std::max(c->ndof, 1)), "pivots");
    SPCK(cudaMalloc(&s->d_swap, sizeof(int) * std::max(c->ndof, 1)), "pivots");
    SPCK(cudaMalloc(&s->d_work[0], sizeof(double2) * std::max(s->max_work, 1LL)), "work");
    SPCK(cudaMalloc(&s->d_work[1], sizeof(double2) * std::max(s->max_work, 1LL)), "work");
    SPCK(cudaMalloc(&s->d_info, sizeof(int)), "status");
  }
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

// the level-by-level launches of one solve, R right-hand sides per CTA
template <int R>
static void sparse_solve_levels(const SparseLU *s, SolveArgs a, cudaStream_t st) {
  const unsigned nchunk = (unsigned)((a.nrhs + R - 1) / R);
  auto tiles = [](int rows) { return (unsigned)std::max(1, (rows + kThreads - 1) / kThreads); };
  for (int l = s->nlevel - 1; l >= 0; l--) {  // forward, from the leaves
    a.fronts = s->d_lev_fronts + s->lev_off[l];
    const unsigned nfl = (unsigned)s->lev[l].size();
    k_sp_solve_fwd<R><<<dim3(nfl, nchunk), kThreads, 0, st>>>(a);
    if (s->lev_mmax[l] > 0)
      k_sp_solve_rect<R><<<dim3(nfl, tiles(s->lev_mmax[l]), nchunk), kThreads, 0, st>>>(a, 1);
  }
  for (int l = 0; l < s->nlevel; l++) {  // backward, from the root
    a.fronts = s->d_lev_fronts + s->lev_off[l];
    const unsigned nfl = (unsigned)s->lev[l].size();
    if (s->lev_mmax[l] > 0)
      k_sp_solve_rect<R><<<dim3(nfl, tiles(s->lev_kmax[l]), nchunk), kThreads, 0, st>>>(a, 0);
    k_sp_solve_bwd<R><<<dim3(nfl, nchunk), kThreads, 0, st>>>(a);
  }
}

int sparse_solve(Ctx *c, int nrhs, int trans, double *rhs, cudaStream_t st, std::string *msg) {
  SparseLU *s = c->sparse;
  if (!s || !s->factored) {
    *msg = "sparse solve: no factorisation (call fem25_sparse_factor_dev first)";
    return FEM25_ERR_ARG;
  }
  SolveArgs a{nullptr, s->d_fr, s->d_own, s->d_bnd, s->d_fac, s->d_swap,
              reinterpret_cast<double2 *>(rhs), c->ndof, nrhs, trans};
  if (nrhs == 1)
    sparse_solve_levels<1>(s, a, st);
  else
    sparse_solve_levels<kRhsPerCta>(s, a, st);
  SPCK(cudaGetLastError(), "solve");
  return 0;
}

}  // namespace fem25
