// Numeric factorisation of the sparse direct solve's fronts, one level of the
// dissection tree at a time (the tree, the fronts and their storage are
// described in sparse_solve.cu).  Per level:
//   k_sp_pull       F11, F12, F21 = the update blocks of its two children
//   k_sp_entries    + the CSR entries whose first eliminated DOF it owns
//   F11 = P L11 U11, partial pivoting among the fully summed rows:
//     k <= 96       k_sp_lu (F11 in shared memory), then k_sp_trsm for
//                   U12 = L11^-1 P F12 and L21 = F21 U11^-1
//     larger        panels of 32 columns: k_sp_panel, k_sp_panel_apply (row
//                   interchanges, the panel's rows of U, its part of L21),
//                   k_sp_gemm (trailing update of everything but F22)
//   k_sp_gemm       F22 = the children's update blocks - L21 U12, once, over all k
// What bounds it: FP64 operations, 8/3 k^3 + 8 k^2 m + 8 k m^2 a front, most of
// them in products.  The products run on the FP64 tensor cores (mma m8n8k4;
// measured 36.9 TFLOP/s against 36.6 for DFMA, but an operand read from shared
// memory feeds 8 columns), with every 32 x 32 diagonal triangle inverted once so
// that the triangular solves are products too.  Pivot searches are the serial
// part: about 0.4 us a column, which is why a panel lives in registers.
#include <climits>
#include <cstdlib>

#include "sparse.cuh"
#include "sparse_tiles.h"

namespace fem25 {

namespace {

constexpr int kPanelThreads = 512;
constexpr int kSmThreads = 256, kSmRows = 390, kSmLd = kSmRows + 1;  // panel in shared memory
constexpr int kLuThreads = 256;
constexpr int kLuRows = 128;     // threads of k_sp_lu that hold a row of a sub-panel
constexpr int kTrsmThreads = 128, kStrip = 32;
using sp::kGt;
constexpr int kGemmThreads = 128, kTile = 64, kKc = 8;
constexpr int kGemmLda = kGt + 2, kGemmLdb = kKc + 4;  // conflict-free fragment reads
constexpr int kGemmStage = kKc * kGemmLda + kGt * kGemmLdb;  // double2 per stage

// ---------------------------------------------------------------------------
// assembly of a level's fronts
// ---------------------------------------------------------------------------
// Front entry (i, j) = its two children's update entries at (map[i], map[j]),
// where map is the position in the child's boundary or -1: the child's update
// block starts at row and column k of its front.  Every entry is written once,
// so nothing is cleared first and no child is added by read-modify-write.  F22,
// most of a front, is left to k_sp_gemm, which takes the children's entries in as it
// writes it (written here and read back there it cost 36.0 ms instead of 34.0 over a
// factorisation of 331 GFLOP and a solve).
struct Children {
  const int *map[2];
  const double2 *base[2] = {nullptr, nullptr};
  long long ld[2] = {0, 0};
  __device__ __forceinline__ Children(const SpFront &f, const SpFront *__restrict__ fr,
                                      const int *__restrict__ pull,
                                      const double2 *__restrict__ wchild) {
    map[0] = pull + f.map0;
    map[1] = map[0] + f.k + f.m;
    for (int s = 0; s < 2; s++)
      if (f.child[s] >= 0) {
        const SpFront g = fr[f.child[s]];
        ld[s] = (long long)g.k + g.m;
        base[s] = wchild + g.work0 + g.k * (ld[s] + 1);
      }
  }
};

__global__ void k_sp_pull(const int *__restrict__ fronts, const SpFront *__restrict__ fr,
                          const int *__restrict__ pull, const double2 *__restrict__ wchild,
                          double2 *__restrict__ work) {
  const SpFront f = fr[fronts[blockIdx.x]];
  const int n = f.k + f.m;
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const Children ch(f, fr, pull, wchild);
  for (int j = blockIdx.y * nw + (threadIdx.x >> 5); j < n; j += gridDim.y * nw) {
    const int j0 = ch.base[0] ? ch.map[0][j] : -1, j1 = ch.base[1] ? ch.map[1][j] : -1;
    double2 *dst = work + f.work0 + (long long)j * n;
    const double2 *c0 = ch.base[0] + j0 * ch.ld[0], *c1 = ch.base[1] + j1 * ch.ld[1];
    const int rows = j < f.k ? n : f.k;
#pragma unroll 2
    for (int i = lane; i < rows; i += 32) {
      double2 v = make_double2(0.0, 0.0);
      const int i0 = j0 >= 0 ? ch.map[0][i] : -1, i1 = j1 >= 0 ? ch.map[1][i] : -1;
      if (i0 >= 0) v = c0[i0];
      if (i1 >= 0) {
        const double2 w = c1[i1];
        v.x += w.x;
        v.y += w.y;
      }
      dst[i] = v;
    }
  }
}

// the level's CSR entries (each has a place of its own)
__global__ void k_sp_entries(long long n, const int *__restrict__ idx,
                             const long long *__restrict__ loc, const double2 *__restrict__ csr,
                             double2 *__restrict__ work) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    double2 *o = work + loc[i];
    const double2 v = csr[idx[i]];
    o->x += v.x;
    o->y += v.y;
  }
}

// ---------------------------------------------------------------------------
// sub-panel LU in registers
// ---------------------------------------------------------------------------
// Candidate of a pivot search: |re| + |im| as the bits of a non-negative double, which
// order like it (NaN counts as 0), and its row; INT_MAX: none.
struct Pivot {
  unsigned hi, lo;
  int row;
  // takes v of row r where it is larger; rows come in ascending order
  __device__ __forceinline__ void offer(double2 v, int r) {
    const double a = fabs(v.x) + fabs(v.y);
    const unsigned h = a >= 0.0 ? (unsigned)__double2hiint(a) : 0u;
    const unsigned l = a >= 0.0 ? (unsigned)__double2loint(a) : 0u;
    if (row == INT_MAX || h > hi || (h == hi && l > lo)) {
      hi = h;
      lo = l;
      row = r;
    }
  }
  // lane of the warp's largest candidate, the lowest row among equals.  The upper
  // words mostly decide; the lower words and rows are compared where they do not.
  __device__ __forceinline__ int winner() const {
    constexpr unsigned kAll = 0xffffffffu;
    const unsigned h = __reduce_max_sync(kAll, hi);
    unsigned m = __ballot_sync(kAll, hi == h);
    if (m & (m - 1)) {  // the same for every lane
      const unsigned l = __reduce_max_sync(kAll, hi == h ? lo : 0u);
      const bool in = hi == h && lo == l;
      const int r = __reduce_min_sync(kAll, in ? row : INT_MAX);
      m = __ballot_sync(kAll, in && row == r);
    }
    return __ffs(m) - 1;
  }
};

template <int W, int NW>
struct PanelShared {
  Pivot cand[2][NW];
  double2 prow[2][W], jrow[2][W];
  int swap[W];
};

// neither zero nor NaN
__device__ __forceinline__ bool pivot_ok(double2 v) { return fabs(v.x) + fabs(v.y) > 0.0; }

// barrier over the first T threads of the CTA (T a multiple of 32)
template <int T>
__device__ __forceinline__ void bar_rows() {
  asm volatile("bar.sync 1, %0;" ::"n"(T) : "memory");
}

// 1 / v, zero when v is no pivot; scaled by a power of two around |v|, so that |v|^2
// neither under- nor overflows
__device__ __forceinline__ double2 crecip(double2 v) {
  if (!pivot_ok(v)) return make_double2(0.0, 0.0);
  const int e = (__double2hiint(fmax(fabs(v.x), fabs(v.y))) >> 20) - 1023;
  const double f = __hiloint2double((1023 - max(-1021, min(1021, e))) << 20, 0);
  const double x = f * v.x, y = f * v.y, d = 1.0 / (x * x + y * y);
  return make_double2(x * d * f, -y * d * f);
}

// LU with partial pivoting of the w <= W columns a[q][0..w) of rows
// r = t + q T < nrow; thread t keeps position r, interchanges move the contents.
// s.swap[j] = row interchanged with j.  Returns true when a pivot was zero (or NaN).
// Two barriers a column.
template <int W, int RPT, int T>
__device__ __forceinline__ bool lu_columns(double2 (&a)[RPT][W], int w, int nrow, int t,
                                           PanelShared<W, T / 32> &s) {
  const int lane = t & 31, warp = t >> 5;
  bool zero = false;
#pragma unroll
  for (int j = 0; j < W; j++) {
    if (j < w) {
      Pivot best{0u, 0u, INT_MAX};
#pragma unroll
      for (int q = 0; q < RPT; q++) {
        const int r = t + q * T;
        if (r >= j && r < nrow) best.offer(a[q][j], r);
      }
      if (lane == best.winner()) s.cand[j & 1][warp] = best;
      bar_rows<T>();
      Pivot all{0u, 0u, INT_MAX};
      if (lane < T / 32) all = s.cand[j & 1][lane];
      const int p = __shfl_sync(0xffffffffu, all.row, all.winner());
      if (t == 0) s.swap[j] = p;
#pragma unroll
      for (int q = 0; q < RPT; q++) {
        const int r = t + q * T;
        if (r == p)
#pragma unroll
          for (int c = 0; c < W; c++) s.prow[j & 1][c] = a[q][c];
        if (r == j && p != j)
#pragma unroll
          for (int c = 0; c < W; c++) s.jrow[j & 1][c] = a[q][c];
      }
      bar_rows<T>();
      double2 u[W];
#pragma unroll
      for (int c = j; c < W; c++) u[c] = s.prow[j & 1][c];
      const bool z = !pivot_ok(u[j]);
      zero |= z;
      const double2 inv = crecip(u[j]);
#pragma unroll
      for (int q = 0; q < RPT; q++) {
        const int r = t + q * T;
        if (r == p && p != j)
#pragma unroll
          for (int c = 0; c < W; c++) a[q][c] = s.jrow[j & 1][c];
        if (r == j)
#pragma unroll
          for (int c = 0; c < W; c++) a[q][c] = s.prow[j & 1][c];
        if (r > j && r < nrow) {
          const double2 l = cmul(a[q][j], inv);
          a[q][j] = l;
#pragma unroll
          for (int c = j + 1; c < W; c++) a[q][c] = cfms(a[q][c], l, u[c]);
        }
      }
    }
  }
  return zero;
}

// source row of row x after the w interchanges swap[0..w): j <-> swap[j] in order
__device__ __forceinline__ int swap_source(int x, const int *swap, int w) {
  for (int j = w - 1; j >= 0; j--) x = x == j ? swap[j] : x == swap[j] ? j : x;
  return x;
}

// ---------------------------------------------------------------------------
// inverses of a diagonal block's triangles, in place
// ---------------------------------------------------------------------------
// D (ld) holds an nb x nb unit lower \ upper LU.  Thread group `job` (of `gt`
// threads, index `g` in it) inverts the lower (up = 0) or upper (up = 1)
// triangle by elimination: step j subtracts column j's multipliers times row j
// of the inverse so far, all (i, c) of a step at once, one CTA barrier a step.
// Every thread of the CTA calls it (nb may differ between groups; steps = the
// largest).  buf: this group's [2][32] column copies, dinv: [32] reciprocals.
__device__ __forceinline__ void invert_triangle(double2 *D, int ld, int nb, int steps, bool up,
                                                bool on, int g, int gt, double2 (*buf)[sp::kNb],
                                                double2 *dinv) {
  if (on) {
    for (int i = g; i < nb; i += gt) {
      if (up) {
        const double2 d = D[i + i * ld];
        dinv[i] = crecip(d);
      } else {
        buf[0][i] = D[i];
      }
    }
  }
  __syncthreads();
  if (on && up)
    for (int i = g; i < nb - 1; i += gt) buf[0][i] = cmul(D[i + (nb - 1) * ld], dinv[nb - 1]);
  for (int s = 0; s < steps; s++) {
    __syncthreads();
    if (!on || s >= nb) continue;
    const double2 *cur = buf[s & 1];
    double2 *nxt = buf[(s + 1) & 1];
    if (!up) {
      const int j = s;
      for (int e = g; e < (nb - 1 - j) * sp::kNb; e += gt) {
        const int i = j + 1 + e / sp::kNb, c = e % sp::kNb;
        if (c < j) D[i + c * ld] = cfms(D[i + c * ld], cur[i], D[j + c * ld]);
        if (c == j) D[i + j * ld] = make_double2(-cur[i].x, -cur[i].y);
      }
      if (j + 1 < nb)
        for (int i = j + 2 + g; i < nb; i += gt) nxt[i] = D[i + (j + 1) * ld];
    } else {
      const int j = nb - 1 - s;
      for (int e = g; e < j * sp::kNb; e += gt) {
        const int i = e / sp::kNb, c = e % sp::kNb;
        if (c > j && c < nb) D[i + c * ld] = cfms(D[i + c * ld], cur[i], D[j + c * ld]);
        if (c == j) D[i + j * ld] = make_double2(-cur[i].x, -cur[i].y);
      }
      if (j > 0)
        for (int i = g; i < j - 1; i += gt) nxt[i] = cmul(D[i + (j - 1) * ld], dinv[j - 1]);
    }
  }
  __syncthreads();
  if (on && up)
    for (int e = g; e < nb * sp::kNb; e += gt) {
      const int i = e / sp::kNb, c = e % sp::kNb;
      if (c > i && c < nb) D[i + c * ld] = cmul(D[i + c * ld], dinv[i]);
      if (c == i) D[i + i * ld] = dinv[i];
    }
  __syncthreads();
}

// ---------------------------------------------------------------------------
// fronts with k <= kSmallK: F11 in shared memory, one CTA a front
// ---------------------------------------------------------------------------
// Blocked right-looking LU, sub-panels of 8 columns in the registers of the
// first 128 threads (one row each), the interchanges and the rows of U by warps
// and threads on shared memory, the trailing block by 8 x 8 tensor-core tiles.
// Writes L11 \ U11 with inverted diagonal blocks to the store, and perm.
__global__ void __launch_bounds__(kLuThreads)
    k_sp_lu(const int *__restrict__ fronts, const SpFront *__restrict__ fr,
            const double2 *__restrict__ work, double2 *__restrict__ fac, int *__restrict__ perm,
            int *__restrict__ swap, int *__restrict__ info) {
  constexpr int W = 8, kJobs = 2 * (sp::kSmallK / sp::kNb);
  extern __shared__ double2 A[];  // k x k, ld
  __shared__ PanelShared<W, kLuRows / 32> ps;
  __shared__ int pos[kLuRows];    // original row of each position
  __shared__ int sdst[2 * W], ssrc[2 * W];
  __shared__ double2 buf[kJobs][2][sp::kNb], dinv[kJobs][sp::kNb];
  const int t = fronts[blockIdx.x];
  const SpFront f = fr[t];
  const int k = f.k, n = f.k + f.m, ld = k | 1;
  if (k == 0) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int nw = kLuThreads / 32;
  const double2 *F = work + f.work0;
  for (int c = warp; c < k; c += nw)
    for (int r = lane; r < k; r += 32) cp16(A + r + c * ld, F + r + (long long)c * n, true);
  cp_commit();
  for (int r = tid; r < k; r += kLuThreads) pos[r] = r;
  cp_wait<0>();
  __syncthreads();
  bool zero = false;
  for (int cb = 0; cb < k; cb += W) {
    const int w = min(W, k - cb), nrow = k - cb;
    if (tid < kLuRows) {
      double2 a[1][W];
#pragma unroll
      for (int c = 0; c < W; c++)
        a[0][c] = (tid < nrow && c < w) ? A[cb + tid + (cb + c) * ld] : make_double2(0.0, 0.0);
      zero |= lu_columns<W, 1, kLuRows>(a, w, nrow, tid, ps);
      if (tid < nrow)
#pragma unroll
        for (int c = 0; c < W; c++)
          if (c < w) A[cb + tid + (cb + c) * ld] = a[0][c];
      bar_rows<kLuRows>();
      if (tid < w) swap[f.own0 + cb + tid] = cb + ps.swap[tid];
      if (tid < 2 * W) {
        const int d = tid < W ? tid : ps.swap[min(tid - W, w - 1)];
        const bool ok = tid < w || (tid >= W && tid - W < w);
        sdst[tid] = ok ? d : -1;
        ssrc[tid] = ok ? swap_source(d, ps.swap, w) : -1;
      }
    }
    __syncthreads();
    // interchanges on the other columns (half a warp a column) and on pos
    {
      const int h = lane >> 4, d = sdst[lane & 15], sr = ssrc[lane & 15];
      for (int c0 = 2 * warp; c0 < k - w + 1; c0 += 2 * nw) {
        const int cc = c0 + h;  // column k - w stands for pos
        const int col = cc < cb ? cc : cc + w;
        double2 v = make_double2(0.0, 0.0);
        int pv = 0;
        if (d >= 0 && cc < k - w) v = A[cb + sr + col * ld];
        if (d >= 0 && cc == k - w) pv = pos[cb + sr];
        __syncwarp();
        if (d >= 0 && cc < k - w) A[cb + d + col * ld] = v;
        if (d >= 0 && cc == k - w) pos[cb + d] = pv;
      }
    }
    __syncthreads();
    const int r0 = cb + w;  // trailing block
    if (r0 >= k) break;
    // the sub-panel's rows of U (w = 8 here)
    for (int c = r0 + tid; c < k; c += kLuThreads) {
      double2 u[W];
#pragma unroll
      for (int j = 0; j < W; j++) u[j] = A[cb + j + c * ld];
#pragma unroll
      for (int i = 1; i < W; i++)
#pragma unroll
        for (int j = 0; j < i; j++) u[i] = cfms(u[i], A[cb + i + (cb + j) * ld], u[j]);
#pragma unroll
      for (int j = 1; j < W; j++) A[cb + j + c * ld] = u[j];
    }
    __syncthreads();
    // trailing block: a warp takes column tiles, two row tiles at a time
    const int nt = (k - r0 + 7) / 8;
    for (int q = warp; q < nt * ((nt + 1) / 2); q += nw) {
      const int tj = q / ((nt + 1) / 2), ti = 2 * (q - tj * ((nt + 1) / 2));
      ZTile z[2];
#pragma unroll
      for (int kk = 0; kk < W; kk += 4) {
        const int cB = r0 + 8 * tj + (lane >> 2);
        const double2 b = cB < k ? A[cb + kk + (lane & 3) + cB * ld] : make_double2(0.0, 0.0);
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int rA = r0 + 8 * (ti + h) + (lane >> 2);
          const double2 l = rA < k ? A[rA + (cb + kk + (lane & 3)) * ld] : make_double2(0.0, 0.0);
          z[h].mma(l, b);
        }
      }
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int r = r0 + 8 * (ti + h) + (lane >> 2);
#pragma unroll
        for (int x = 0; x < 2; x++) {
          const int c = r0 + 8 * tj + 2 * (lane & 3) + x;
          if (r < k && c < k) {
            double2 *o = A + r + c * ld;
            *o = make_double2(o->x - z[h].r[x], o->y - z[h].i[x]);
          }
        }
      }
    }
    __syncthreads();
  }
  if (zero && tid == 0) atomicCAS(info, 0, t + 1);
  __syncthreads();
  // inverses of the diagonal blocks, a group of threads per triangle
  {
    const int nblk = (k + sp::kNb - 1) / sp::kNb, njob = 2 * nblk;
    const int gt = (kLuThreads / njob) & ~31;  // threads per job, whole warps
    const int job = tid / gt;
    const bool on = job < njob;
    const int b = on ? job >> 1 : 0;
    const int nb = min(sp::kNb, k - b * sp::kNb);
    invert_triangle(A + b * sp::kNb * (ld + 1), ld, nb, min(sp::kNb, k), job & 1, on, tid - job * gt,
                    gt, buf[on ? job : 0], dinv[on ? job : 0]);
  }
  double2 *L = fac + f.fac0;
  for (int c = warp; c < k; c += nw)
    for (int r = lane; r < k; r += 32) L[r + (long long)c * n] = A[r + c * ld];
  for (int r = tid; r < k; r += kLuThreads) perm[f.own0 + r] = pos[r];
}

// The triangular solves of a small front, strips of 32: blockIdx.y below the
// front's count of column strips: U12 = L11^-1 P F12 of 32 boundary columns;
// then row strips of L21 = F21 U11^-1.  A warp owns 8 columns (rows) of its strip,
// so that warps never wait for one another: per block of 32 the product with the
// inverted diagonal block, then the update of the rows (columns) still to come, as
// 8 x 8 tensor-core tiles whose factor operand is loaded straight from the store
// (16 loads in flight a lane).  Staging it in shared memory cost two CTA barriers a
// block and left two CTAs an SM: 4.8 ms over all levels against 4.4.
// Rows and columns past k read the last ones instead; they meet zeros, or their
// results are not kept.
__global__ void __launch_bounds__(kTrsmThreads)
    k_sp_trsm(const int *__restrict__ fronts, const SpFront *__restrict__ fr,
              const double2 *__restrict__ work, double2 *__restrict__ fac,
              const int *__restrict__ perm) {
  extern __shared__ double2 X[];
  const SpFront f = fr[fronts[blockIdx.x]];
  const int k = f.k, m = f.m, n = k + m;
  const int nstrip = (m + kStrip - 1) / kStrip;
  if (k == 0 || (int)blockIdx.y >= 2 * nstrip) return;
  const bool rows = (int)blockIdx.y >= nstrip;  // L21
  const int s0 = ((int)blockIdx.y - (rows ? nstrip : 0)) * kStrip, ns = min(kStrip, m - s0);
  const int kp = (k + 7) & ~7;
  const int ldx = rows ? kStrip + 2 : kp + 5;  // X[strip row][k] or X[k][strip column]
  const double2 *F = work + f.work0;
  double2 *L = fac + f.fac0;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int lr = lane >> 2, lk = lane & 3;
  constexpr int nw = kTrsmThreads / 32;
  const double2 zero = make_double2(0.0, 0.0), one = make_double2(1.0, 0.0);
  if (!rows) {
    for (int c = 8 * warp; c < 8 * warp + 8; c++)
      for (int r = lane; r < kp; r += 32)
        X[r + c * ldx] = (c < ns && r < k)
                             ? F[perm[f.own0 + r] + (long long)(k + s0 + c) * n] : zero;
    __syncwarp();
  } else {
    for (int c = warp; c < kp; c += nw)
      X[lane + c * ldx] = (lane < ns && c < k) ? F[k + s0 + lane + (long long)c * n] : zero;
    __syncthreads();
  }
  auto at = [&](int r, int c) {
    return L[min(r, k - 1) + (long long)min(c, k - 1) * n];
  };
  for (int jb = 0; jb < k; jb += sp::kNb) {
    const int rest = kp - jb;  // from the block on, padded
    const int nt = rest / 8, nd = min(4, nt);
    if (!rows) {
      double2 *Xw = X + jb + 8 * warp * ldx;  // this warp's 8 columns, from row jb
      double2 b[8];
#pragma unroll
      for (int q = 0; q < 8; q++) b[q] = 4 * q < rest ? Xw[4 * q + lk + lr * ldx] : zero;
      ZTile z[4];
#pragma unroll
      for (int ti = 0; ti < 4; ti++)
        if (ti < nd) {
          double2 a[8];
#pragma unroll
          for (int q = 0; q <= 2 * ti + 1; q++) a[q] = at(jb + 8 * ti + lr, jb + 4 * q + lk);
#pragma unroll
          for (int q = 0; q <= 2 * ti + 1; q++) {
            const int r = 8 * ti + lr, c = 4 * q + lk;  // strictly lower, unit diagonal
            z[ti].mma(c < r ? a[q] : c == r ? one : zero, b[q]);
          }
        }
      __syncwarp();
#pragma unroll
      for (int ti = 0; ti < 4; ti++)
        if (ti < nd)
#pragma unroll
          for (int x = 0; x < 2; x++)
            if (jb + 8 * ti + lr < k)
              Xw[8 * ti + lr + (2 * lk + x) * ldx] = make_double2(z[ti].r[x], z[ti].i[x]);
      __syncwarp();
#pragma unroll
      for (int q = 0; q < 8; q++) b[q] = 4 * q < rest ? Xw[4 * q + lk + lr * ldx] : zero;
      for (int ti = 4; ti < nt; ti += 2) {
        ZTile y[2];
        double2 a[2][8];
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
          for (int q = 0; q < 8; q++) a[h][q] = at(jb + 8 * (ti + h) + lr, jb + 4 * q + lk);
#pragma unroll
        for (int q = 0; q < 8; q++) {
          y[0].mma(a[0][q], b[q]);
          y[1].mma(a[1][q], b[q]);
        }
#pragma unroll
        for (int h = 0; h < 2; h++)
          if (jb + 8 * (ti + h) + lr < k)
#pragma unroll
            for (int x = 0; x < 2; x++) {
              double2 *o = Xw + 8 * (ti + h) + lr + (2 * lk + x) * ldx;
              *o = make_double2(o->x - y[h].r[x], o->y - y[h].i[x]);
            }
      }
      __syncwarp();
    } else {
      double2 *Xw = X + 8 * warp + jb * ldx;  // this warp's 8 rows, from column jb
      double2 a[8];
#pragma unroll
      for (int q = 0; q < 8; q++) a[q] = 4 * q < rest ? Xw[lr + (4 * q + lk) * ldx] : zero;
      ZTile z[4];
#pragma unroll
      for (int tj = 0; tj < 4; tj++)
        if (tj < nd) {
          double2 b[8];
#pragma unroll
          for (int q = 0; q <= 2 * tj + 1; q++) b[q] = at(jb + 4 * q + lk, jb + 8 * tj + lr);
#pragma unroll
          for (int q = 0; q <= 2 * tj + 1; q++)  // upper with the diagonal
            z[tj].mma(a[q], 4 * q + lk <= 8 * tj + lr ? b[q] : zero);
        }
      __syncwarp();
#pragma unroll
      for (int tj = 0; tj < 4; tj++)
        if (tj < nd)
#pragma unroll
          for (int x = 0; x < 2; x++)
            if (jb + 8 * tj + 2 * lk + x < k)
              Xw[lr + (8 * tj + 2 * lk + x) * ldx] = make_double2(z[tj].r[x], z[tj].i[x]);
      __syncwarp();
#pragma unroll
      for (int q = 0; q < 8; q++) a[q] = 4 * q < rest ? Xw[lr + (4 * q + lk) * ldx] : zero;
      for (int tj = 4; tj < nt; tj += 2) {
        ZTile y[2];
        double2 b[2][8];
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
          for (int q = 0; q < 8; q++) b[h][q] = at(jb + 4 * q + lk, jb + 8 * (tj + h) + lr);
#pragma unroll
        for (int q = 0; q < 8; q++) {
          y[0].mma(a[q], b[0][q]);
          y[1].mma(a[q], b[1][q]);
        }
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
          for (int x = 0; x < 2; x++)
            if (jb + 8 * (tj + h) + 2 * lk + x < k) {
              double2 *o = Xw + lr + (8 * (tj + h) + 2 * lk + x) * ldx;
              *o = make_double2(o->x - y[h].r[x], o->y - y[h].i[x]);
            }
      }
      __syncwarp();
    }
  }
  if (!rows) {
    double2 *U12 = L + (long long)n * k;
    for (int c = 8 * warp; c < min(8 * warp + 8, ns); c++)
      for (int r = lane; r < k; r += 32) U12[r + (long long)(s0 + c) * k] = X[r + c * ldx];
  } else {
    __syncthreads();
    for (int c = warp; c < k; c += nw)
      if (lane < ns) L[k + s0 + lane + (long long)c * n] = X[lane + c * ldx];
  }
}

// ---------------------------------------------------------------------------
// fronts with k > kSmallK: panels of 32 columns
// ---------------------------------------------------------------------------
// Columns [jb, jb + 32) of F11, rows from jb, one CTA a front: sub-panels of W
// columns in registers (RPT rows a thread, chosen so that W RPT stays at 16),
// each applied to the panel's columns to its right; then the diagonal block's
// triangles are inverted in place.
// SM: the panel stays in shared memory between its sub-panels (up to kSmRows rows).
template <int W, int RPT, int T, bool SM>
__global__ void __launch_bounds__(T)
    k_sp_panel(const int *__restrict__ fronts, const SpFront *__restrict__ fr,
               double2 *__restrict__ work, int jb, int *__restrict__ swap, int *__restrict__ info) {
  constexpr int kRight = sp::kNb - W;
  extern __shared__ double2 panel[];  // SM: [32][kSmLd]
  __shared__ PanelShared<W, T / 32> ps;
  __shared__ double2 Ls[W][W], Us[W][kRight > 0 ? kRight : 1];
  __shared__ int sdst[2 * W], ssrc[2 * W];
  __shared__ double2 D[sp::kNb][sp::kNb + 1];
  __shared__ double2 buf[2][2][sp::kNb], dinv[2][sp::kNb];
  const int t = fronts[blockIdx.x];
  const SpFront f = fr[t];
  const int k = f.k;
  if (jb >= k) return;
  const long long nf = (long long)f.k + f.m;
  const int nb = min(sp::kNb, k - jb), tid = threadIdx.x;
  double2 *const G = work + f.work0 + jb * (nf + 1);  // the panel: rows and columns from jb
  double2 *const F = SM ? panel : G;
  const long long n = SM ? kSmLd : nf;
  if (SM) {
    for (int c = tid >> 5; c < nb; c += T / 32)
      for (int r = tid & 31; r < k - jb; r += 32) cp16(F + r + c * n, G + r + c * nf, true);
    cp_commit();
    cp_wait<0>();
    __syncthreads();
  }
  bool zero = false;
  for (int s0 = 0; s0 < nb; s0 += W) {
    const int w = min(W, nb - s0), cb = s0, nrow = k - jb - cb;  // cb: within the panel
    double2 a[RPT][W];
#pragma unroll
    for (int q = 0; q < RPT; q++) {
      const int r = tid + q * T;
#pragma unroll
      for (int c = 0; c < W; c++)
        a[q][c] = (r < nrow && c < w) ? F[cb + r + (cb + c) * n] : make_double2(0.0, 0.0);
    }
    zero |= lu_columns<W, RPT, T>(a, w, nrow, tid, ps);
#pragma unroll
    for (int q = 0; q < RPT; q++) {
      const int r = tid + q * T;
      if (r < nrow)
#pragma unroll
        for (int c = 0; c < W; c++)
          if (c < w) F[cb + r + (cb + c) * n] = a[q][c];
    }
    if (tid < W)
#pragma unroll
      for (int c = 0; c < W; c++) Ls[tid][c] = a[0][c];
    __syncthreads();  // ps.swap complete
    if (tid < w) swap[f.own0 + jb + cb + tid] = jb + cb + ps.swap[tid];
    if (tid < 2 * w) {
      const int d = tid < w ? tid : ps.swap[tid - w];
      sdst[tid] = d;
      ssrc[tid] = swap_source(d, ps.swap, w);
    }
    __syncthreads();
    // the interchanges on the panel's other columns
    {
      // 2 w rows of at most 32 - w columns: up to kPass rounds of T entries
      constexpr int kPass = (2 * W * (sp::kNb - W) + T - 1) / T;
      const int i = tid % (2 * w), per = T / (2 * w);
      double2 v[kPass];
#pragma unroll
      for (int u = 0; u < kPass; u++) {
        const int cc = tid / (2 * w) + u * per;
        v[u] = cc < nb - w && tid < per * 2 * w ? F[(cc < s0 ? cc : cc + w) * n + cb + ssrc[i]]
                                                : make_double2(0.0, 0.0);
      }
      __syncthreads();
#pragma unroll
      for (int u = 0; u < kPass; u++) {
        const int cc = tid / (2 * w) + u * per;
        if (cc < nb - w && tid < per * 2 * w) F[(cc < s0 ? cc : cc + w) * n + cb + sdst[i]] = v[u];
      }
    }
    const int ncr = nb - s0 - w;
    if (ncr <= 0) break;
    __syncthreads();
    // rows of U of the panel's remaining columns
    if (tid < ncr) {
      double2 u[W];
      double2 *col = F + cb + (cb + w + tid) * n;
#pragma unroll
      for (int j = 0; j < W; j++) u[j] = col[j];
#pragma unroll
      for (int i = 1; i < W; i++)
#pragma unroll
        for (int j = 0; j < i; j++) u[i] = cfms(u[i], Ls[i][j], u[j]);
#pragma unroll
      for (int j = 0; j < W; j++) {
        if (j > 0) col[j] = u[j];
        Us[j][tid] = u[j];
      }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < RPT; q++) {
      const int r = tid + q * T;
      if (r >= w && r < nrow) {
        double2 *row = F + cb + r + (cb + w) * n;
#pragma unroll 4
        for (int c = 0; c < ncr; c++) {
          double2 x = row[c * n];
#pragma unroll
          for (int j = 0; j < W; j++) x = cfms(x, a[q][j], Us[j][c]);
          row[c * n] = x;
        }
      }
    }
    __syncthreads();
  }
  if (zero && tid == 0) atomicCAS(info, 0, t + 1);
  __syncthreads();
  for (int e = tid; e < sp::kNb * sp::kNb; e += T) {
    const int r = e % sp::kNb, c = e / sp::kNb;
    if (r < nb && c < nb) D[c][r] = F[r + c * n];
  }
  __syncthreads();
  const int job = tid / (T / 2);
  invert_triangle(&D[0][0], sp::kNb + 1, nb, nb, job, true, tid % (T / 2), T / 2, buf[job],
                  dinv[job]);
  for (int e = tid; e < sp::kNb * sp::kNb; e += T) {
    const int r = e % sp::kNb, c = e / sp::kNb;
    if (r < nb && c < nb) F[r + c * n] = D[c][r];
  }
  if (SM) {
    __syncthreads();
    for (int c = tid >> 5; c < nb; c += T / 32)
      for (int r = tid & 31; r < k - jb; r += 32) G[r + c * nf] = F[r + c * n];
  }
}

// The same panel for any number of rows, a column at a time in global memory
// (more than 4 096 rows, where a sub-panel no longer fits the registers).
__global__ void __launch_bounds__(kPanelThreads)
    k_sp_panel_any(const int *__restrict__ fronts, const SpFront *__restrict__ fr,
                   double2 *__restrict__ work, int jb, int *__restrict__ swap,
                   int *__restrict__ info) {
  constexpr int T = kPanelThreads;
  __shared__ Pivot cand[T / 32];
  __shared__ double2 u[sp::kNb];
  __shared__ double2 D[sp::kNb][sp::kNb + 1];
  __shared__ double2 buf[2][2][sp::kNb], dinv[2][sp::kNb];
  const int t = fronts[blockIdx.x];
  const SpFront f = fr[t];
  const int k = f.k;
  if (jb >= k) return;
  const long long n = (long long)f.k + f.m;
  const int nb = min(sp::kNb, k - jb), tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double2 *F = work + f.work0;
  bool zero = false;
  for (int j = 0; j < nb; j++) {
    double2 *col = F + (jb + j) * n;
    Pivot best{0u, 0u, INT_MAX};
    for (int r = jb + j + tid; r < k; r += T) best.offer(col[r], r);
    if (lane == best.winner()) cand[warp] = best;
    __syncthreads();
    Pivot all{0u, 0u, INT_MAX};
    if (lane < T / 32) all = cand[lane];
    const int p = __shfl_sync(0xffffffffu, all.row, all.winner());
    if (tid == 0) swap[f.own0 + jb + j] = p;
    if (tid < nb) {
      double2 *c = F + (jb + tid) * n;
      const double2 x = c[jb + j], y = c[p];
      c[jb + j] = y;
      c[p] = x;
      u[tid] = y;
    }
    __syncthreads();
    const double2 d = u[j];
    const bool z = !pivot_ok(d);
    zero |= z;
    const double2 inv = crecip(d);
    for (int r = jb + j + 1 + tid; r < k; r += T) {
      const double2 l = cmul(col[r], inv);
      col[r] = l;
      for (int c = j + 1; c < nb; c++) {
        double2 *o = F + r + (jb + c) * n;
        *o = cfms(*o, l, u[c]);
      }
    }
    __syncthreads();
  }
  if (zero && tid == 0) atomicCAS(info, 0, t + 1);
  for (int e = tid; e < sp::kNb * sp::kNb; e += T) {
    const int r = e % sp::kNb, c = e / sp::kNb;
    if (r < nb && c < nb) D[c][r] = F[jb + r + (jb + c) * n];
  }
  __syncthreads();
  const int job = tid / (T / 2);
  invert_triangle(&D[0][0], sp::kNb + 1, nb, nb, job, true, tid % (T / 2), T / 2, buf[job],
                  dinv[job]);
  for (int e = tid; e < sp::kNb * sp::kNb; e += T) {
    const int r = e % sp::kNb, c = e / sp::kNb;
    if (r < nb && c < nb) F[jb + r + (jb + c) * n] = D[c][r];
  }
}

// What follows a panel of a larger front, strips of 64 over blockIdx.y: columns
// right of the panel (interchanges, then the panel's rows of U: inv(L) times
// them), columns of L left of it (interchanges only), and rows of F21 (times
// inv(U): the panel's part of L21).
__global__ void __launch_bounds__(kGemmThreads)
    k_sp_panel_apply(const int *__restrict__ fronts, const SpFront *__restrict__ fr,
                     double2 *__restrict__ work, int jb, const int *__restrict__ swap) {
  constexpr int NB = sp::kNb, ldT = NB + 4, ldD = NB + 2, ldR = kTile + 2;
  extern __shared__ double2 sh[];
  double2 *X = sh;               // [64 columns][32 rows], or [32 columns][64 rows]
  double2 *D = sh + kTile * ldT;
  __shared__ int sw[NB], src[NB], dst[NB], dsrc[NB];
  const SpFront f = fr[fronts[blockIdx.x]];
  const int k = f.k, m = f.m;
  if (jb >= k) return;
  const int n = k + m, nb = min(NB, k - jb), c1 = jb + nb;
  const int nright = (n - c1 + kTile - 1) / kTile, nleft = (jb + kTile - 1) / kTile;
  const int nrow = (m + kTile - 1) / kTile;
  int y = blockIdx.y;
  if (y >= nright + nleft + nrow) return;
  double2 *F = work + f.work0;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, lr = lane >> 2, lk = lane & 3;
  const double2 zero = make_double2(0.0, 0.0), one = make_double2(1.0, 0.0);
  if (y >= nright + nleft) {
    // L21: X(64 x 32) inv(U)
    const int r0 = k + (y - nright - nleft) * kTile;
    for (int e = tid; e < NB * kTile; e += kGemmThreads) {
      const int r = e % kTile, c = e / kTile;
      X[r + c * ldR] = (c < nb && r0 + r < n) ? F[r0 + r + (long long)(jb + c) * n] : zero;
    }
    for (int e = tid; e < NB * NB; e += kGemmThreads) {
      const int r = e % NB, c = e / NB;
      D[r + c * ldT] = (r <= c && c < nb) ? F[jb + r + (long long)(jb + c) * n] : zero;
    }
    __syncthreads();
    ZTile z[2][4];
    const double2 *Xw = X + 16 * warp + lr;
#pragma unroll
    for (int q = 0; q < 8; q++) {
      const double2 a0 = Xw[(4 * q + lk) * ldR], a1 = Xw[8 + (4 * q + lk) * ldR];
#pragma unroll
      for (int tj = 0; tj < 4; tj++)
        if (q <= 2 * tj + 1) {
          const double2 b = D[4 * q + lk + (8 * tj + lr) * ldT];
          z[0][tj].mma(a0, b);
          z[1][tj].mma(a1, b);
        }
    }
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
      for (int tj = 0; tj < 4; tj++)
#pragma unroll
        for (int x = 0; x < 2; x++) {
          const int r = r0 + 16 * warp + 8 * h + lr, c = 8 * tj + 2 * lk + x;
          if (r < n && c < nb)
            F[r + (long long)(jb + c) * n] = make_double2(z[h][tj].r[x], z[h][tj].i[x]);
        }
    return;
  }
  const bool left = y >= nright;
  const int s0 = left ? (y - nright) * kTile : c1 + y * kTile;
  const int ns = left ? min(kTile, jb - s0) : min(kTile, n - s0);
  if (tid < nb) sw[tid] = swap[f.own0 + jb + tid] - jb;
  __syncthreads();
  if (tid < nb) {
    src[tid] = swap_source(tid, sw, nb);
    const int d = sw[tid];
    dst[tid] = d >= nb ? d : -1;  // rows of the panel's top block come from src
    dsrc[tid] = d >= nb ? swap_source(d, sw, nb) : -1;
  }
  if (!left)
    for (int e = tid; e < NB * NB; e += kGemmThreads) {
      const int r = e % NB, c = e / NB;
      D[r + c * ldD] = r == c ? one : (c < r && r < nb) ? F[jb + r + (long long)(jb + c) * n] : zero;
    }
  __syncthreads();
  // top rows after the interchanges to X; the displaced rows wait in registers
  double2 dv[kTile / 4];
#pragma unroll
  for (int q = 0; q < kTile / 4; q++) {
    const int c = warp + 4 * q;
    const double2 *col = F + (long long)(s0 + c) * n + jb;
    X[lane + c * ldT] = (lane < nb && c < ns) ? col[src[lane]] : zero;
    dv[q] = (lane < nb && c < ns && dst[lane] >= 0) ? col[dsrc[lane]] : zero;
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < kTile / 4; q++) {
    const int c = warp + 4 * q;
    double2 *col = F + (long long)(s0 + c) * n + jb;
    if (lane < nb && c < ns) {
      if (dst[lane] >= 0) col[dst[lane]] = dv[q];
      if (left) col[lane] = X[lane + c * ldT];
    }
  }
  if (left) return;
  // inv(L) (32 x 32) X(32 x 64): a warp takes 16 columns
  ZTile z[4][2];
#pragma unroll
  for (int q = 0; q < 8; q++) {
    const double2 b0 = X[4 * q + lk + (16 * warp + lr) * ldT];
    const double2 b1 = X[4 * q + lk + (16 * warp + 8 + lr) * ldT];
#pragma unroll
    for (int ti = 0; ti < 4; ti++)
      if (q <= 2 * ti + 1) {
        const double2 a = D[8 * ti + lr + (4 * q + lk) * ldD];
        z[ti][0].mma(a, b0);
        z[ti][1].mma(a, b1);
      }
  }
#pragma unroll
  for (int ti = 0; ti < 4; ti++)
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
      for (int x = 0; x < 2; x++) {
        const int r = 8 * ti + lr, c = 16 * warp + 8 * h + 2 * lk + x;
        if (r < nb && c < ns)
          F[jb + r + (long long)(s0 + c) * n] = make_double2(z[ti][h].r[x], z[ti][h].i[x]);
      }
}

// ---------------------------------------------------------------------------
// products
// ---------------------------------------------------------------------------
// 32 x 32 tiles of C -= A B, tile columns [c0, c0 + cn) (t2 tiles per front at
// most), four warps of 16 x 16 (2 x 2 tensor-core tiles of complex 8 x 8; at five CTAs
// an SM as fast as 64 x 64 tiles of 4 x 4 where those are full, and 10 to 40 % faster
// where the fronts end in part tiles: 15.3 against 19.0 ms over a factorisation of
// 331 GFLOP), A and B staged by cp.async in double-buffered chunks of 8; 8 x 8 tiles
// past the edge are skipped.  SCHUR: F22 = the children's updates - L21 U12 from the
// factor store, K = k (jb unused).  Otherwise the trailing update after panel jb of a
// larger front, K = its columns, on rows and columns beyond the panel except F22, in
// place in the work buffer.
template <bool SCHUR>
__global__ void __launch_bounds__(kGemmThreads, 5)
    k_sp_gemm(const int *__restrict__ fronts, const SpFront *__restrict__ fr,
              double2 *__restrict__ work, const double2 *__restrict__ fac, int jb, int t2, int c0,
              int cn, const int *__restrict__ pull, const double2 *__restrict__ wchild) {
  constexpr int NT = kGt / 16;
  extern __shared__ double2 sh[];
  const SpFront f = fr[fronts[blockIdx.x / t2]];
  const int tile = blockIdx.x % t2;
  const int k = f.k, m = f.m, n = k + m;
  const double2 *A, *B;
  double2 *C;
  int M, K, lda, ldb;
  int corner;  // C(r, c) with r, c >= corner is left alone
  if (SCHUR) {
    M = corner = m;
    K = k;
    A = fac + f.fac0 + k;
    lda = n;
    B = fac + f.fac0 + (long long)n * k;
    ldb = k;
    C = work + f.work0 + (long long)k * (n + 1);
  } else {
    if (jb >= k) return;
    K = min(sp::kNb, k - jb);
    const int c1 = jb + K;
    M = n - c1;
    A = work + f.work0 + c1 + (long long)jb * n;
    B = work + f.work0 + jb + (long long)c1 * n;
    lda = ldb = n;
    C = work + f.work0 + (long long)c1 * (n + 1);
    corner = k - c1;
  }
  int m0, n0;
  if (!sp::gemm_tile(M, corner, tile, c0, cn, &m0, &n0)) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, lr = lane >> 2, lk = lane & 3;
  const int wm = kGt / 2 * (warp & 1), wn = kGt / 2 * (warp >> 1);
  const int mt = min(NT, max(0, (M - m0 - wm + 7) / 8)), nt = min(NT, max(0, (M - n0 - wn + 7) / 8));
  auto stage = [&](int ch) {
    double2 *As = sh + (ch & 1) * kGemmStage, *Bs = As + kKc * kGemmLda;
    const int k0 = ch * kKc;
#pragma unroll
    for (int q = 0; q < kKc * kGt / kGemmThreads; q++) {
      const int e = tid + q * kGemmThreads;
      {
        const int r = e % kGt, c = e / kGt;
        const bool ok = m0 + r < M && k0 + c < K;
        cp16(As + r + c * kGemmLda, ok ? A + m0 + r + (long long)(k0 + c) * lda : A, ok);
      }
      {
        const int r = e % kKc, c = e / kKc;
        const bool ok = n0 + c < M && k0 + r < K;
        cp16(Bs + r + c * kGemmLdb, ok ? B + k0 + r + (long long)(n0 + c) * ldb : B, ok);
      }
    }
    cp_commit();
  };
  ZTile z[NT][NT];
  const int nch = (K + kKc - 1) / kKc;
  if (nch > 0) stage(0);
  for (int ch = 0; ch < nch; ch++) {
    if (ch + 1 < nch) {
      stage(ch + 1);
      cp_wait<1>();
    } else {
      cp_wait<0>();
    }
    __syncthreads();
    const double2 *As = sh + (ch & 1) * kGemmStage, *Bs = As + kKc * kGemmLda;
#pragma unroll
    for (int kk = 0; kk < kKc; kk += 4) {
      double2 b[NT];
#pragma unroll
      for (int tj = 0; tj < NT; tj++) b[tj] = Bs[kk + lk + (wn + 8 * tj + lr) * kGemmLdb];
#pragma unroll
      for (int ti = 0; ti < NT; ti++) {
        if (ti < mt) {
          const double2 a = As[wm + 8 * ti + lr + (kk + lk) * kGemmLda];
#pragma unroll
          for (int tj = 0; tj < NT; tj++)
            if (tj < nt) z[ti][tj].mma(a, b[tj]);
        }
      }
    }
    __syncthreads();
  }
  if (SCHUR) {
    const Children ch(f, fr, pull, wchild);
    int row[2][NT], col[2][2 * NT];  // places in the children's boundaries
#pragma unroll
    for (int s = 0; s < 2; s++) {
#pragma unroll
      for (int ti = 0; ti < NT; ti++) {
        const int r = m0 + wm + 8 * ti + lr;
        row[s][ti] = ch.base[s] && r < M ? ch.map[s][k + r] : -1;
      }
#pragma unroll
      for (int q = 0; q < 2 * NT; q++) {
        const int c = n0 + wn + 8 * (q >> 1) + 2 * lk + (q & 1);
        col[s][q] = ch.base[s] && c < M ? ch.map[s][k + c] : -1;
      }
    }
#pragma unroll
    for (int ti = 0; ti < NT; ti++)
#pragma unroll
      for (int q = 0; q < 2 * NT; q++) {
        const int r = m0 + wm + 8 * ti + lr, c = n0 + wn + 8 * (q >> 1) + 2 * lk + (q & 1);
        double2 v = make_double2(0.0, 0.0);
        if (row[0][ti] >= 0 && col[0][q] >= 0) v = ch.base[0][row[0][ti] + col[0][q] * ch.ld[0]];
        if (row[1][ti] >= 0 && col[1][q] >= 0) {
          const double2 w = ch.base[1][row[1][ti] + col[1][q] * ch.ld[1]];
          v.x += w.x;
          v.y += w.y;
        }
        const ZTile &t = z[ti][q >> 1];
        if (r < M && c < M)
          C[r + (long long)c * n] = make_double2(v.x - t.r[q & 1], v.y - t.i[q & 1]);
      }
    return;
  }
#pragma unroll
  for (int ti = 0; ti < NT; ti++)
#pragma unroll
    for (int tj = 0; tj < NT; tj++)
#pragma unroll
      for (int x = 0; x < 2; x++) {
        const int r = m0 + wm + 8 * ti + lr, c = n0 + wn + 8 * tj + 2 * lk + x;
        if (r < M && c < M && !(r >= corner && c >= corner)) {
          double2 *o = C + r + (long long)c * n;
          *o = make_double2(o->x - z[ti][tj].r[x], o->y - z[ti][tj].i[x]);
        }
      }
}

// ---------------------------------------------------------------------------
// a larger front's factors to the store, and its row permutation
// ---------------------------------------------------------------------------
__global__ void k_sp_store(const int *__restrict__ fronts, const SpFront *__restrict__ fr,
                           const double2 *__restrict__ work, double2 *__restrict__ fac,
                           const int *__restrict__ swap, int *__restrict__ perm) {
  const SpFront f = fr[fronts[blockIdx.x]];
  const long long n = (long long)f.k + f.m;
  const double2 *F = work + f.work0;
  double2 *L = fac + f.fac0, *U = L + n * f.k;
  const long long stride = (long long)gridDim.y * blockDim.x;
  for (long long q = blockIdx.y * blockDim.x + threadIdx.x; q < n * f.k; q += stride) L[q] = F[q];
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  for (int j = blockIdx.y * nw + (threadIdx.x >> 5); j < f.m; j += gridDim.y * nw)
    for (int i = lane; i < f.k; i += 32) U[i + (long long)j * f.k] = F[i + (f.k + j) * n];
  for (long long r = blockIdx.y * blockDim.x + threadIdx.x; r < f.k; r += stride)
    perm[f.own0 + r] = swap_source((int)r, swap + f.own0, f.k);
}

size_t lu_smem(int k) { return sizeof(double2) * (size_t)k * (k | 1); }
size_t trsm_smem(int kmax) {
  const size_t kp = (kmax + 7) & ~7;
  return sizeof(double2) * (kp + 5) * (kStrip + 2);
}
constexpr size_t kApplySmem = sizeof(double2) * (kTile + sp::kNb) * (sp::kNb + 4);
constexpr size_t kPanelSmem = sizeof(double2) * sp::kNb * kSmLd;
constexpr size_t kGemmSmem = sizeof(double2) * 2 * kGemmStage;

}  // namespace

cudaError_t sparse_factor_attributes() {
  cudaError_t e;
  if ((e = cudaFuncSetAttribute(k_sp_lu, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)lu_smem(sp::kSmallK))))
    return e;
  if ((e = cudaFuncSetAttribute(k_sp_trsm, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)trsm_smem(sp::kSmallK))))
    return e;
  if ((e = cudaFuncSetAttribute(k_sp_panel<8, 1, kSmThreads, true>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPanelSmem)) ||
      (e = cudaFuncSetAttribute(k_sp_panel<8, 2, kSmThreads, true>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPanelSmem)))
    return e;
  if ((e = cudaFuncSetAttribute(k_sp_panel_apply, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)kApplySmem)))
    return e;
  return cudaSuccess;
}

// nf of level l's fronts (with k <= kSmallK or larger) on group g's streams
static cudaError_t factor_group(SparseLU *s, int l, const int *fronts, int nf, bool small,
                                double2 *W, const double2 *Wc, int nsm, int g) {
  if (nf <= 0) return cudaSuccess;
  const cudaStream_t st = s->st[g];
  cudaError_t e;
  auto tiles = [](int rows) { return (rows + kTile - 1) / kTile; };
  if (small && s->lev_ksmall[l] > 0) {
    const int ks = s->lev_ksmall[l], ms = s->lev_msmall[l];
    k_sp_lu<<<nf, kLuThreads, lu_smem(ks), st>>>(fronts, s->d_fr, W, s->d_fac, s->d_perm,
                                                 s->d_swap, s->d_info);
    if (ms > 0)
      k_sp_trsm<<<dim3(nf, 2 * ((ms + kStrip - 1) / kStrip)), kTrsmThreads, trsm_smem(ks), st>>>(
          fronts, s->d_fr, W, s->d_fac, s->d_perm);
  }
  if (!small) {
    const int kmax = s->lev_kmax[l], mmax = s->lev_mmax[l], nmax = s->lev_nmax[l];
    // FEM25_PANEL_WIDTH caps the sub-panel width (8, 4, 2; 1: the any-size kernel)
    const char *env = std::getenv("FEM25_PANEL_WIDTH");
    const int cap = env ? std::atoi(env) : 8;
    bool pending = false;
    for (int jb = 0; jb < kmax; jb += sp::kNb) {
      const int rows = kmax - jb;
      constexpr int PT = kPanelThreads, ST = kSmThreads;
      if (rows <= ST && cap >= 8)
        k_sp_panel<8, 1, ST, true>
            <<<nf, ST, kPanelSmem, st>>>(fronts, s->d_fr, W, jb, s->d_swap, s->d_info);
      else if (rows <= kSmRows && cap >= 8)
        k_sp_panel<8, 2, ST, true>
            <<<nf, ST, kPanelSmem, st>>>(fronts, s->d_fr, W, jb, s->d_swap, s->d_info);
      else if (rows <= PT && cap >= 8)
        k_sp_panel<8, 1, PT, false>
            <<<nf, PT, 0, st>>>(fronts, s->d_fr, W, jb, s->d_swap, s->d_info);
      else if (rows <= 2 * PT && cap >= 8)
        k_sp_panel<8, 2, PT, false>
            <<<nf, PT, 0, st>>>(fronts, s->d_fr, W, jb, s->d_swap, s->d_info);
      else if (rows <= 4 * PT && cap >= 4)
        k_sp_panel<4, 4, PT, false>
            <<<nf, PT, 0, st>>>(fronts, s->d_fr, W, jb, s->d_swap, s->d_info);
      else if (rows <= 8 * PT && cap >= 2)
        k_sp_panel<2, 8, PT, false>
            <<<nf, PT, 0, st>>>(fronts, s->d_fr, W, jb, s->d_swap, s->d_info);
      else
        k_sp_panel_any<<<nf, kPanelThreads, 0, st>>>(fronts, s->d_fr, W, jb, s->d_swap, s->d_info);
      // the interchanges and rows of U need the last panel's whole update
      if (pending && (e = cudaStreamWaitEvent(st, s->updated[g], 0))) return e;
      const int right = nmax - jb;  // >= columns beyond the panel of any front
      k_sp_panel_apply<<<dim3(nf, tiles(right) + tiles(jb) + tiles(mmax) + 1), kGemmThreads,
                         kApplySmem, st>>>(fronts, s->d_fr, W, jb, s->d_swap);
      if (kmax <= jb + sp::kNb) break;  // the last panel: only F22 lies beyond it
      const int tr = (right + kGt - 1) / kGt;
      // the next panel's columns on this stream, the others beside it
      k_sp_gemm<false><<<(unsigned)(nf * tr), kGemmThreads, kGemmSmem, st>>>(
          fronts, s->d_fr, W, s->d_fac, jb, tr, 0, 1, nullptr, nullptr);
      if (tr > 1) {
        if ((e = cudaEventRecord(s->applied[g], st)) ||
            (e = cudaStreamWaitEvent(s->side[g], s->applied[g], 0)))
          return e;
        k_sp_gemm<false>
            <<<(unsigned)(nf * tr * (tr - 1)), kGemmThreads, kGemmSmem, s->side[g]>>>(
                fronts, s->d_fr, W, s->d_fac, jb, tr * (tr - 1), 1, tr - 1, nullptr, nullptr);
        if ((e = cudaEventRecord(s->updated[g], s->side[g]))) return e;
        pending = true;
      }
    }
    if (pending && (e = cudaStreamWaitEvent(st, s->updated[g], 0))) return e;
    const unsigned ysb = (unsigned)std::max(1, std::min(256, 8 * nsm / nf));
    k_sp_store<<<dim3(nf, ysb), 256, 0, st>>>(fronts, s->d_fr, W, s->d_fac, s->d_swap, s->d_perm);
  }
  const int mmax = small ? s->lev_msmall[l] : s->lev_mmax[l];
  if (mmax > 0) {
    const int tm = (mmax + kGt - 1) / kGt;
    k_sp_gemm<true><<<(unsigned)((long long)nf * tm * tm), kGemmThreads, kGemmSmem, st>>>(
        fronts, s->d_fr, W, s->d_fac, -1, tm * tm, 0, tm, s->d_pull, Wc);
  }
  return cudaSuccess;
}

cudaError_t sparse_factor_level(SparseLU *s, int l, const double2 *csr, double2 *W,
                                const double2 *Wc, int nsm, cudaStream_t st) {
  const int nfl = (int)s->lev[l].size(), nsmall = s->lev_nsmall[l], nbig = nfl - nsmall;
  const int *dfr = s->d_lev_fronts + s->lev_off[l];
  // more CTAs per front where the level has few fronts
  const unsigned ysplit = (unsigned)std::max(1, std::min(256, 8 * nsm / std::max(nfl, 1)));
  k_sp_pull<<<dim3(nfl, ysplit), 256, 0, st>>>(dfr, s->d_fr, s->d_pull, Wc, W);
  const long long ne = s->lev_ent0[l + 1] - s->lev_ent0[l];
  if (ne > 0)
    k_sp_entries<<<(int)std::min<long long>((ne + 255) / 256, (long long)nsm * 16), 256, 0, st>>>(
        ne, s->d_ent_idx + s->lev_ent0[l], s->d_ent_loc + s->lev_ent0[l], csr, W);
  // The fronts in groups, each on a stream of its own: a group's pivot searches (one
  // CTA a front) run beside another's products, and within a group the next panel
  // beside the update of the columns behind it.  A factorisation of 331 GFLOP and a
  // solve, measured while k_sp_pull still wrote F22: 38.7 ms on one stream, 37.4 in
  // groups, 36.2 with the side streams, 35.7 with the groups' streams first in
  // priority (2 to 4 groups within 1 %, 8 slower); 34.7 now.
  cudaError_t e;
  const int groups = std::min(sp::kStreams, nfl);
  if ((e = cudaEventRecord(s->ready, st))) return e;
  for (int g = 0; g < groups; g++) {
    cudaStream_t sg = s->st[g];
    if ((e = cudaStreamWaitEvent(sg, s->ready, 0))) return e;
    const int a0 = (int)((long long)nsmall * g / groups), a1 = (int)((long long)nsmall * (g + 1) / groups);
    const int b0 = (int)((long long)nbig * g / groups), b1 = (int)((long long)nbig * (g + 1) / groups);
    if ((e = factor_group(s, l, dfr + a0, a1 - a0, true, W, Wc, nsm, g)) ||
        (e = factor_group(s, l, dfr + nsmall + b0, b1 - b0, false, W, Wc, nsm, g)) ||
        (e = cudaEventRecord(s->done[g], sg)) || (e = cudaStreamWaitEvent(st, s->done[g], 0)))
      return e;
  }
  return cudaGetLastError();
}

}  // namespace fem25
