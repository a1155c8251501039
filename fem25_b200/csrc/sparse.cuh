// Structures of the sparse direct solve shared by its analysis and solve
// (sparse_solve.cu) and its factorisation (sparse_factor.cu).
#pragma once
#include <algorithm>
#include <string>
#include <vector>

#include "ctx.cuh"

namespace fem25 {

namespace sp {
constexpr int kLeafElems = 2;  // elements per leaf of the dissection
constexpr int kNb = 32;        // columns of a panel and of an inverted diagonal block
constexpr int kSmallK = 96;    // fronts with at most this many own DOFs: F11 in shared memory
constexpr int kStreams = 3;    // groups of a level's fronts factored side by side
}  // namespace sp

struct SpFront {
  int k, m;             // own (fully summed) and boundary DOFs
  int parent;           // -1: root
  int child[2];         // -1: none
  int level;            // depth in the dissection tree (root 0)
  long long own0;       // first own DOF in own[] (= elimination position)
  long long bnd0;       // first boundary DOF in bnd[]
  long long map0;       // its two pull maps in pull[], n entries each (see k_sp_pull)
  long long fac0;       // factor store: L block [n][k] (ld n), then U12 [k][m] (ld k)
  long long work0;      // offset of its n x n front in its level's work buffer
};

// Factor store of a front: L11 \ U11 over L21 as n x k (ld n), then U12 as
// k x m (ld k).  Each 32 x 32 diagonal block of L11 \ U11 holds the inverses of
// its two triangles instead (strictly lower: inv(L), unit diagonal implied;
// upper with diagonal: inv(U)): every later use of the triangles is a product.
struct SparseLU {
  bool analysed = false, factored = false;
  int nfront = 0, nlevel = 0;
  std::vector<SpFront> fr;
  std::vector<std::vector<int>> lev;   // front ids per level, kSmallK fronts first
  std::vector<int> lev_nsmall;         // per level: fronts with k <= kSmallK
  std::vector<int> lev_ksmall, lev_msmall;      // their largest own and boundary counts
  std::vector<int> lev_kmax, lev_mmax, lev_nmax;  // the same and the order over all fronts
  std::vector<long long> lev_work;     // work elements per level
  std::vector<long long> lev_ent0;     // first CSR-entry record of each level
  long long fac_elems = 0, max_work = 0;
  // device
  SpFront *d_fr = nullptr;
  int *d_own = nullptr, *d_bnd = nullptr, *d_pull = nullptr;
  int *d_lev_fronts = nullptr;         // all levels' front ids, concatenated
  std::vector<long long> lev_off;      // offset of each level in d_lev_fronts
  int *d_ent_idx = nullptr;            // CSR entries by level, and their
  long long *d_ent_loc = nullptr;      // offsets in the level's work buffer
  double2 *d_fac = nullptr;            // factor store
  int *d_perm = nullptr;               // [NDOF] row j of a front's P F11 is its row perm[j]
  int *d_swap = nullptr;               // [NDOF] interchanges of the panels being factored
  double2 *d_work[2] = {nullptr, nullptr};
  int *d_info = nullptr;               // first zero pivot (front + 1), 0 = none
  // per group of fronts: its stream, a side stream for the updates that the next
  // panel does not wait for, and the events between them and the caller's stream
  cudaStream_t st[sp::kStreams] = {}, side[sp::kStreams] = {};
  cudaEvent_t done[sp::kStreams] = {}, applied[sp::kStreams] = {}, updated[sp::kStreams] = {};
  cudaEvent_t ready = nullptr;
};

// Numeric factorisation of one level's fronts (sparse_factor.cu): W holds the
// level's fronts, Wc its children's.
cudaError_t sparse_factor_level(SparseLU *s, int level, const double2 *csr, double2 *W,
                                const double2 *Wc, int nsm, cudaStream_t st);
cudaError_t sparse_factor_attributes();

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 cfms(double2 acc, double2 a, double2 b) {  // acc - a b
  return make_double2(acc.x - a.x * b.x + a.y * b.y, acc.y - a.x * b.y - a.y * b.x);
}

// FP64 tensor-core product of warp tiles, D(8x8) += A(8x4) B(4x8): lane l holds
// A[l / 4][l % 4], B[l % 4][l / 4] and D[l / 4][2 (l % 4) + {0, 1}].
__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1},{%2},{%3},{%0,%1};"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

// 8 x 8 complex accumulator of a warp
struct ZTile {
  double r[2] = {0.0, 0.0}, i[2] = {0.0, 0.0};
  __device__ __forceinline__ void mma(double2 a, double2 b) {
    dmma(r, a.x, b.x);
    dmma(i, a.x, b.y);
    dmma(r, -a.y, b.y);
    dmma(i, a.y, b.x);
  }
};

// 16-byte asynchronous copy to shared memory, zero-filled when !ok
__device__ __forceinline__ void cp16(double2 *dst, const double2 *src, bool ok) {
  const int bytes = ok ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                   (unsigned)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

}  // namespace fem25
