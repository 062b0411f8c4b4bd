// icp.cuh — one registration_icp rung as a routine of a CTA or of a cluster of
// CTAs (matching/icp.rs:308-440, 599-778).
//
// A pass has two halves. First every moving point finds its match: the point
// moved by the current pose (f64, R p + tau) and its nearest target inside the
// strict radius (exact, lowest index on ties), most of them without a search
// (icp_match). Then the correspondence count, the squared error and the 27
// normal-equation terms (21 of the lower triangle of J^T J, 6 of J^T r) are
// summed in f64 (icp_sums). The order of every sum is fixed: 128 partial sums,
// partial v over the points v, v + 128, ... in ascending order, whatever the
// number of threads; then a warp shuffle tree and a fixed-order sum over the
// four warps' totals, both compensated (TwoSum, the rounding errors carried and
// added once), so a rung is bit-for-bit reproducible run to run and does not
// depend on the block and cluster size it ran at. Open3D's convergence test
// follows, and one warp runs Eigen's pivoted LDLT (f64) and the Rz Ry Rx update.
//
// The points are the reference numerics (Numerics::REFERENCE, f64 point loops,
// World assembly); the difference from the CPU oracle is the summation order
// of the per-pass sums and the pose being re-applied to the source each pass
// (T S) where the reference moves the previous pass's points (U P).
#pragma once

#include "traverse.cuh"

namespace sherd {

constexpr int ICP_BLOCK = 128;  // partial sums of a pass
constexpr int ICP_SUMS = 29;    // count, err2, jtj[21], jtr[6]
constexpr int ICP_TERMS = 9;    // row[6], r, d2, 1: what a point adds products of

struct IcpShared {
  double red[ICP_BLOCK / 32][ICP_SUMS];
  double carry[ICP_BLOCK / 32][ICP_SUMS];  // the rounding errors of red's warp sums
  double sums[ICP_SUMS];
  double t[16];
  double tp[16];  // the pose of the pass before
  double x[6], mats[3][9], prod[9], u[16];  // plane_step's working values
  float turn;     // a bound on |R - Rp| of the two poses' rotations
  unsigned todo, next;  // the chunks listed to look at, the next of them
};

// What a rung keeps of its source from pass to pass, one slot per item in
// flight: per point the last match (a target slot, or -1) and how far it stands
// (icp_match), and per chunk of 32 points its centre and radius and, while none
// of its points has a match, a bound for all of them. `chunks` and `balls` may be
// null; every chunk is then looked at point by point.
struct IcpChunk {
  float slack;  // every point of the chunk is at least this far from every target point; -1: no bound
  float debt;   // the moves of the chunk since its points' slacks were last brought up to date
};
template <class H>
struct IcpMemory {
  H *hint;
  float *slack;
  IcpChunk *chunks;
  float4 *balls;
};

// Slot `k` of a memory with room for n points a slot.
template <class H>
__host__ __device__ inline IcpMemory<H> memory_slot(const IcpMemory<H> &m, size_t k, size_t n) {
  const size_t c = k * ((n + 31) / 32);
  return {m.hint + k * n, m.slack + k * n, m.chunks ? m.chunks + c : nullptr,
          m.balls ? m.balls + c : nullptr};
}

// The shared memory of a rung on blocks of G groups of 128 threads, in clusters
// of C.
template <int G, int C>
struct IcpBlock {
  IcpShared s;
  uint32_t queue[4 * G * 64];  // the points that need a search, 64 per warp or all together
  uint32_t list[ICP_BLOCK * G];   // the chunks to look at, and what they owe
  float owed[ICP_BLOCK * G];
  // a round of points' terms
  double tile[G > 2 ? ICP_TERMS : 1][G > 2 ? ICP_BLOCK * G : 1];
  double part[C > 1 ? ICP_SUMS : 1][C > 1 ? ICP_BLOCK : 1];  // every CTA's partial sums
};

// Static for a block on its own; a cluster's is above the 48 KB a static one may
// have, so its kernels are launched with it as dynamic shared memory.
template <int G, int C>
__device__ __forceinline__ IcpBlock<G, C> &rung_memory() {
  if constexpr (C == 1) {
    __shared__ IcpBlock<G, 1> b;
    return b;
  } else {
    extern __shared__ __align__(16) unsigned char rung_dynamic[];
    return *reinterpret_cast<IcpBlock<G, C> *>(rung_dynamic);
  }
}

// ---- clusters ---------------------------------------------------------------
// A rung with few items in flight runs on a cluster of C CTAs: the points'
// matches and the 29 sums are shared out over the CTAs, the totals written to
// every CTA's shared memory.

template <int C>
__device__ __forceinline__ uint32_t cta_rank() {
  if constexpr (C == 1) return 0;
  uint32_t r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}

// A barrier over the block (C = 1) or the cluster; writes before it, to global
// and to any CTA's shared memory, are seen after it.
template <int C>
__device__ __forceinline__ void rung_sync() {
  if constexpr (C == 1) {
    __syncthreads();
  } else {
    __syncwarp();
    asm volatile(
        "barrier.cluster.arrive.release.aligned;\n\t"
        "barrier.cluster.wait.acquire.aligned;" ::
            : "memory");
  }
}

// The address of `p` (in this CTA's shared memory) in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t peer_address(const void *p, uint32_t rank) {
  uint32_t a = uint32_t(__cvta_generic_to_shared(p)), out;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(out) : "r"(a), "r"(rank));
  return out;
}
__device__ __forceinline__ void peer_store(double *p, uint32_t rank, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(peer_address(p, rank)), "d"(v) : "memory");
}
__device__ __forceinline__ void peer_store(unsigned *p, uint32_t rank, unsigned v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(peer_address(p, rank)), "r"(v) : "memory");
}

__device__ void matmul4(const double *a, const double *b, double *o) {
  double r[16];
  for (int i = 0; i < 4; ++i)
    for (int j = 0; j < 4; ++j) {
      double s = a[4 * i] * b[j];
      for (int k = 1; k < 4; ++k) s += a[4 * i + k] * b[4 * k + j];
      r[4 * i + j] = s;
    }
  for (int i = 0; i < 16; ++i) o[i] = r[i];
}

// The point-to-plane update of a pass (icp.rs:408-440), T <- U T for the sums s
// by the calling warp (all 32 lanes): U from Eigen's pivoted LDLT
// (icp::eigen_pivots and icp::solve_ldlt, icp.rs:661-753) and
// icp::euler_zyx (icp.rs:770-778); the identity when there is no
// correspondence, no normal or no finite solution.
//
// Lane r holds row r of the permuted 6x6 system in registers, so the rows'
// updates and the five divisions of a column run side by side; every value is
// formed by the operations of the sequential loop, in its order. On one thread,
// with the matrices in local memory, the step took 20 us of every pass (a tenth
// of a 6000-point pass at 128 threads); this one is bound by its chain of six
// dependent f64 divisions.
__device__ __noinline__ void plane_step(const double *s, bool has_normals, double *t,
                                        IcpShared &sh) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  if (lane < 16) sh.u[lane] = lane % 5 == 0 ? 1.0 : 0.0;
  __syncwarp();
  if (s[0] != 0.0 && has_normals) {
    // The pivot order: a selection sort of the original diagonal by magnitude.
    double dv[6];
    int pm[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      pm[k] = k;
      dv[k] = fabs(s[2 + k * (k + 1) / 2 + k]);
    }
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      int b = k;
      double bv = dv[k];
#pragma unroll
      for (int i = k + 1; i < 6; ++i)
        if (dv[i] > bv) {
          b = i;
          bv = dv[i];
        }
#pragma unroll
      for (int i = k + 1; i < 6; ++i)
        if (i == b) {
          const double d = dv[k];
          dv[k] = dv[i];
          dv[i] = d;
          const int q = pm[k];
          pm[k] = pm[i];
          pm[i] = q;
        }
    }
    const int r = lane < 6 ? lane : 5;
    int pr = pm[0];
#pragma unroll
    for (int k = 1; k < 6; ++k)
      if (r == k) pr = pm[k];
    double row[6], d[6], own = 0.0;
#pragma unroll
    for (int l = 0; l < 6; ++l) {
      const int hi = max(pr, pm[l]), lo = min(pr, pm[l]);
      row[l] = s[2 + hi * (hi + 1) / 2 + lo];
    }
    double y = -s[23 + pr];
    // Column by column; lanes r >= k form their entry of column k (the entries
    // above the diagonal are never read).
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      double v = row[k];
#pragma unroll
      for (int j = 0; j < k; ++j) v -= row[j] * (d[j] * __shfl_sync(FULL, row[j], k));
      d[k] = __shfl_sync(FULL, v, k);
      row[k] = d[k] != 0.0 && lane > k ? v / d[k] : v;
      if (r == k) own = d[k];
    }
#pragma unroll
    for (int j = 0; j < 5; ++j) {
      const double yj = __shfl_sync(FULL, y, j);
      if (lane > j) y -= row[j] * yj;
    }
    y = fabs(own) > 2.2250738585072014e-308 ? y / own : 0.0;
    double yy[6];
    bool finite = true;
#pragma unroll
    for (int i = 5; i >= 0; --i) {
      yy[i] = __shfl_sync(FULL, y, i);
#pragma unroll
      for (int j = i + 1; j < 6; ++j) yy[i] -= __shfl_sync(FULL, row[i], j) * yy[j];
      finite = finite && isfinite(yy[i]);
    }
    if (finite) {  // the same for the warp
      if (lane == 0) {
#pragma unroll
        for (int k = 0; k < 6; ++k) sh.x[pm[k]] = yy[k];
      }
      __syncwarp();
      if (lane < 3) {  // Rx, Ry, Rz
        double sn, cs;
        sincos(sh.x[lane], &sn, &cs);
        double *m = sh.mats[lane];
        const int i = lane == 0 ? 1 : 0, j = lane == 2 ? 1 : 2;
        const double up = lane == 1 ? sn : -sn;
        for (int k = 0; k < 9; ++k) m[k] = k % 4 == 0 ? 1.0 : 0.0;
        m[4 * i] = cs;
        m[4 * j] = cs;
        m[3 * i + j] = up;
        m[3 * j + i] = -up;
      }
      __syncwarp();
      const int i = lane / 3, j = lane % 3;
      if (lane < 9) {
        const double *a = sh.mats[2] + 3 * i, *b = sh.mats[1] + j;
        sh.prod[lane] = (a[0] * b[0] + a[1] * b[3]) + a[2] * b[6];
      }
      __syncwarp();
      if (lane < 9) {
        const double *a = sh.prod + 3 * i, *b = sh.mats[0] + j;
        sh.u[4 * i + j] = (a[0] * b[0] + a[1] * b[3]) + a[2] * b[6];
      } else if (lane < 12) {
        sh.u[4 * (lane - 9) + 3] = sh.x[lane - 6];
      }
    }
  }
  __syncwarp();
  double v = 0.0;
  if (lane < 16) {
    sh.tp[lane] = t[lane];
    const double *a = sh.u + (lane & 12), *b = t + (lane & 3);
    v = a[0] * b[0];
    for (int k = 1; k < 4; ++k) v += a[k] * b[4 * k];
  }
  __syncwarp();
  if (lane < 16) t[lane] = v;
  __syncwarp();
}

// The rotation of the SVD of m with a reflection on the smallest singular
// value undone, R = U diag(1, 1, det(U) det(V)) V^T: the rotation part of
// Eigen's umeyama (icp.rs:585-590). One-sided Jacobi (Hestenes): plane
// rotations of the columns of a = m V until every two are orthogonal; then
// a_j = sigma_j u_j, with u2 taken as u0 x u1. R is unique whenever the
// second singular value is not zero.
__device__ __noinline__ void svd_rotation(const double m[3][3], double r[3][3]) {
  double a[3][3], v[3][3] = {{1.0, 0.0, 0.0}, {0.0, 1.0, 0.0}, {0.0, 0.0, 1.0}};
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) a[i][j] = m[i][j];
  for (int sweep = 0; sweep < 30; ++sweep) {
    bool turned = false;
    for (int p = 0; p < 2; ++p)
      for (int q = p + 1; q < 3; ++q) {
        double al = (a[0][p] * a[0][p] + a[1][p] * a[1][p]) + a[2][p] * a[2][p];
        double be = (a[0][q] * a[0][q] + a[1][q] * a[1][q]) + a[2][q] * a[2][q];
        double ga = (a[0][p] * a[0][q] + a[1][p] * a[1][q]) + a[2][p] * a[2][q];
        if (!(fabs(ga) > 1e-15 * sqrt(al * be))) continue;
        turned = true;
        double ze = (be - al) / (2.0 * ga);
        double tt = (ze >= 0.0 ? 1.0 : -1.0) / (fabs(ze) + sqrt(1.0 + ze * ze));
        double c = 1.0 / sqrt(1.0 + tt * tt), sn = c * tt;
        for (int i = 0; i < 3; ++i) {
          double x = a[i][p], y = a[i][q];
          a[i][p] = c * x - sn * y;
          a[i][q] = sn * x + c * y;
          x = v[i][p];
          y = v[i][q];
          v[i][p] = c * x - sn * y;
          v[i][q] = sn * x + c * y;
        }
      }
    if (!turned) break;
  }
  double sv[3];
  int ord[3] = {0, 1, 2};
  for (int j = 0; j < 3; ++j) sv[j] = sqrt((a[0][j] * a[0][j] + a[1][j] * a[1][j]) + a[2][j] * a[2][j]);
  for (int x = 0; x < 2; ++x)
    for (int y = 0; y < 2 - x; ++y)
      if (sv[ord[y]] < sv[ord[y + 1]]) {
        int t = ord[y];
        ord[y] = ord[y + 1];
        ord[y + 1] = t;
      }
  const double smax = sv[ord[0]];
  double u[3][3], w[3][3];
  bool have[3];
  for (int k = 0; k < 3; ++k) {
    int j = ord[k];
    for (int i = 0; i < 3; ++i) w[i][k] = v[i][j];
    have[k] = smax > 0.0 && sv[j] > 1e-12 * smax;
    for (int i = 0; i < 3; ++i) u[i][k] = have[k] ? a[i][j] / sv[j] : 0.0;
  }
  if (!have[0]) {
    for (int i = 0; i < 3; ++i)
      for (int j = 0; j < 3; ++j) r[i][j] = i == j ? 1.0 : 0.0;
    return;
  }
  if (!have[1]) {  // any unit vector orthogonal to u0
    int e = fabs(u[0][0]) <= fabs(u[1][0]) ? (fabs(u[0][0]) <= fabs(u[2][0]) ? 0 : 2)
                                          : (fabs(u[1][0]) <= fabs(u[2][0]) ? 1 : 2);
    double ev[3] = {0.0, 0.0, 0.0};
    ev[e] = 1.0;
    double c[3] = {u[1][0] * ev[2] - u[2][0] * ev[1], u[2][0] * ev[0] - u[0][0] * ev[2],
                   u[0][0] * ev[1] - u[1][0] * ev[0]};
    double nc = sqrt((c[0] * c[0] + c[1] * c[1]) + c[2] * c[2]);
    for (int i = 0; i < 3; ++i) u[i][1] = c[i] / nc;
  }
  // u2 = u0 x u1 always: for rank 3 the SVD's own u2 is +-(u0 x u1) and the
  // det(U) det(V) factor below absorbs the sign; for rank 2, a2 / sigma2 is
  // round-off.
  u[0][2] = u[1][0] * u[2][1] - u[2][0] * u[1][1];
  u[1][2] = u[2][0] * u[0][1] - u[0][0] * u[2][1];
  u[2][2] = u[0][0] * u[1][1] - u[1][0] * u[0][1];
  auto det3 = [](const double x[3][3]) {
    return x[0][0] * (x[1][1] * x[2][2] - x[1][2] * x[2][1]) -
           x[0][1] * (x[1][0] * x[2][2] - x[1][2] * x[2][0]) +
           x[0][2] * (x[1][0] * x[2][1] - x[1][1] * x[2][0]);
  };
  const double d = det3(u) * det3(w) < 0.0 ? -1.0 : 1.0;
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j)
      r[i][j] = (u[i][0] * w[j][0] + u[i][1] * w[j][1]) + d * u[i][2] * w[j][2];
}

// icp::umeyama without scaling (icp.rs:527-592) from a point-to-point pass's
// sums: s[0] count, s[2..5) and s[5..8) the sums of the moved source and of
// the target points, s[8..17) the covariance already scaled by 1/n. T <- U T
// (thread 0 only); identity when there is no correspondence.
__device__ __noinline__ void point_step(IcpShared &sh) {
  const double *s = sh.sums;
  double u[16];
  for (int i = 0; i < 16; ++i) u[i] = (i % 5 == 0) ? 1.0 : 0.0;
  if (s[0] != 0.0) {
    const double one_over_n = 1.0 / s[0];
    double mp[3], mq[3], sigma[3][3], r[3][3];
    for (int k = 0; k < 3; ++k) {
      mp[k] = s[2 + k] * one_over_n;
      mq[k] = s[5 + k] * one_over_n;
    }
    for (int i = 0; i < 3; ++i)
      for (int j = 0; j < 3; ++j) sigma[i][j] = s[8 + 3 * i + j];
    svd_rotation(sigma, r);
    for (int i = 0; i < 3; ++i) {
      for (int j = 0; j < 3; ++j) u[4 * i + j] = r[i][j];
      u[4 * i + 3] = mq[i] - ((r[i][0] * mp[0] + r[i][1] * mp[1]) + r[i][2] * mp[2]);
    }
  }
  matmul4(u, sh.t, sh.t);
}

// Knuth's TwoSum: s = fl(a + b) and the exact rounding error e, a + b = s + e
// (no multiply-add is contracted in this build, so the identity holds).
__device__ __forceinline__ void two_sum(double a, double b, double &s, double &e) {
  s = a + b;
  double bp = s - a;
  e = (a - (s - bp)) + (b - bp);
}

// The sums of N values over the warp, compensated, all N at once: the shuffle
// tree adds the 32 lanes' partials pairwise (l with l ^ 16, then 8, 4, 2, 1)
// and carries every addition's rounding error (TwoSum) beside it. While more
// than one value is left, a lane keeps half of them and hands its partner the
// others, so N sums (a power of two) cost about N + 5 exchanges instead of
// 5 N, each the same pairwise tree (TwoSum's sum and error do not depend on
// the order of its two arguments). On return v[0] and c[0] are the sum and the
// carried error of value `idx`.
template <int N, int O, int M>
__device__ __forceinline__ void warp_sums_compensated(double (&v)[M], double (&c)[M], int lane,
                                                      int &idx) {
  static_assert((N & (N - 1)) == 0, "N a power of two");
  const unsigned FULL = 0xffffffffu;
  if constexpr (O > 0) {
    constexpr int HALF = N > 1 ? N / 2 : 1;
    const bool up = N > 1 && (lane & O);
#pragma unroll
    for (int j = 0; j < HALF; ++j) {
      const int k = N > 1 ? j + HALF : j;
      const double keep = up ? v[k] : v[j], give = up ? v[j] : v[k];
      const double ckeep = up ? c[k] : c[j], cgive = up ? c[j] : c[k];
      const double y = __shfl_xor_sync(FULL, give, O), cy = __shfl_xor_sync(FULL, cgive, O);
      double s, e;
      two_sum(keep, y, s, e);
      v[j] = s;
      c[j] = (ckeep + cy) + e;
    }
    if (up) idx += HALF;
    warp_sums_compensated<HALF, O / 2>(v, c, lane, idx);
  }
}

// The warp totals of a group's partials of sums k0..k0+N-1 into sh.red and
// sh.carry.
template <int N>
__device__ __forceinline__ void store_warp_sums(const double (&acc)[N], int k0, IcpShared &sh) {
  const int lane = threadIdx.x & 31, warp = (threadIdx.x >> 5) & 3;
  constexpr int P = N <= 1 ? 1 : N <= 2 ? 2 : N <= 4 ? 4 : N <= 8 ? 8 : 16;  // padded with zeros
  static_assert(N <= P, "at most 16 sums at a time");
  double v[P], c[P];
#pragma unroll
  for (int k = 0; k < P; ++k) {
    v[k] = k < N ? acc[k < N ? k : 0] : 0.0;
    c[k] = 0.0;
  }
  int idx = 0;
  warp_sums_compensated<P, 16>(v, c, lane, idx);
  if (idx < N && k0 + idx < ICP_SUMS) {
    sh.red[warp][k0 + idx] = v[0];
    sh.carry[warp][k0 + idx] = c[0];
  }
}

// A source point's match (a target slot, or -1) as the pass keeps it: an int,
// or 16 bits (0xFFFF for none) when every target of the batch has fewer than
// 65535 points, which halves the bytes the ladder writes and re-reads.
__device__ __forceinline__ int hint_get(const int *h, uint32_t i) { return h[i]; }
__device__ __forceinline__ int hint_get(const uint16_t *h, uint32_t i) {
  uint16_t v = h[i];
  return v == 0xFFFFu ? -1 : int(v);
}
__device__ __forceinline__ void hint_set(int *h, uint32_t i, int s) { h[i] = s; }
__device__ __forceinline__ void hint_set(uint16_t *h, uint32_t i, int s) {
  h[i] = s < 0 ? uint16_t(0xFFFFu) : uint16_t(s);
}

// Bounds of a square root from above and below: sqrt.approx is within 2^-23
// of the root, the factors are far wider.
__device__ __forceinline__ float root_approx(float x) {
  float y;
  asm("sqrt.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float root_above(double x) {
  return root_approx(__double2float_ru(x)) * 1.000001f;
}

__device__ __forceinline__ float warp_min(float x) {
#pragma unroll
  for (int o = 16; o; o >>= 1) x = fminf(x, __shfl_xor_sync(0xffffffffu, x, o));
  return x;
}

// Lowers a bound (non-negative, or -1) to v: as integers the bits of
// non-negative floats keep their order and those of -1 are below them.
__device__ __forceinline__ void atomic_min_slack(float *p, float v) {
  atomicMin(reinterpret_cast<int *>(p), v < 0.0f ? __float_as_int(-1.0f) : __float_as_int(v));
}

// The ball around the warp's 32 points: the centre of their box, and a radius
// no point is outside of.
__device__ __forceinline__ void chunk_ball(const double4 &p, float4 *out, int lane) {
  const float x = float(p.x), y = float(p.y), z = float(p.z);
  const float cx = 0.5f * (warp_min(x) - warp_min(-x)), cy = 0.5f * (warp_min(y) - warp_min(-y)),
              cz = 0.5f * (warp_min(z) - warp_min(-z));
  const double dx = p.x - cx, dy = p.y - cy, dz = p.z - cz;
  const float r = -warp_min(-root_above((dx * dx + dy * dy) + dz * dz));
  if (lane == 0) *out = make_float4(cx, cy, cz, r);
}

// Hints another CTA of the cluster wrote are read past L1.
template <int C, class H>
__device__ __forceinline__ int hint_load(const H *h, uint32_t i) {
  if constexpr (C == 1) return hint_get(h, i);
  return __ldcg(h + i);
}

// ---- matches ------------------------------------------------------------------

// nearest_within_sq that also says how far the point may move before its
// match can change: `slack` receives a lower bound on the distance from the
// query to every target point but the match (to every point when there is
// none): the nearest of what was scored and of the boxes that were left out.
// (Box distances come from the f32-rounded query; the boxes' padding, or far
// from the cloud the 1e-5, covers that.)
__device__ __noinline__ int nearest_guarded(const CloudView &c, double qx, double qy, double qz,
                                            double r2, int hint, float &slack,
                                            uint32_t &status) {
  double best = r2;
  int best_s = -1;
  uint32_t best_i = MISS;
  slack = -1.0f;
  if (c.n == 0 || !(r2 >= 0.0)) return -1;
  float other = f_inf();  // squared, the nearest thing that is not the match
  float bnd;              // the search radius squared, padded
  auto set_bound = [&]() {
    const float b = __double2float_ru(best);
    bnd = b + 1e-5f * b + 1e-30f;
  };
  auto score = [&](int s, const double4 &p) {
    const double dx = qx - p.x, dy = qy - p.y, dz = qz - p.z;
    const double d2 = (dx * dx + dy * dy) + dz * dz;
    const uint32_t id = uint32_t(p.w);
    if (!(d2 > r2) && (best_s < 0 || d2 < best || (d2 == best && id < best_i))) {
      if (best_s >= 0) other = fminf(other, __double2float_rd(best));
      best = d2;
      best_s = s;
      best_i = id;
      set_bound();
    } else {
      other = fminf(other, __double2float_rd(d2));
    }
  };
  set_bound();
  if (hint >= 0) {
    score(hint, ldg4(c.pts + hint));
    if (best_s < 0) other = f_inf();  // beyond the radius: the walk meets it again or prunes its box
  }
  const float qc[3] = {float(qx), float(qy), float(qz)};
  auto leaf = [&](int first, int count) {
    // Both points of a leaf are read before either is scored.
    static_assert(POINT_LEAF <= 2, "a leaf holds one or two points");
    const double4 p0 = ldg4(c.pts + first), p1 = ldg4(c.pts + first + (count - 1));
    if (first != best_s) score(first, p0);
    if (count > 1 && first + 1 != best_s) score(first + 1, p1);
  };
  if (c.root_leaf)
    leaf(0, c.root_leaf);
  else
    wide_walk(
        c.wide, qc, 2u * c.n + 64u, leaf, [&]() { return bnd; },
        [&](float k) { other = fminf(other, k); }, status);
  slack = root_approx(other) * 0.99999f;
  return best_s;
}

// The matches under the pose sh.t into m.hint[] (a target slot, or -1), for the
// chunks of 32 points rank, rank + C, ... (interleaved, because hard chunks lie
// together). Every thread of the CTA calls it.
//
// A point whose match of the last pass provably still holds is not searched
// for: slack[i] is a lower bound on its distance, where it was then, to every
// other target point; it has moved by |x - xp| since, so every other point is
// at least slack[i] - |x - xp| away, and while that is more than its distance
// to the old match, the match is unchanged (with no match: while it is more
// than the radius, there is still none). The bounds are rounded the safe way,
// so the matches are those of a search of every point; slack[i] is kept for
// where the point is now. The others are queued and searched, the old match as
// the first bound. In the first pass (`fresh`) every point
// is searched for and nothing is read from the memory.
//
// A chunk without matches is passed over as a whole by the same rule: its
// points have moved by no more than its centre has plus its radius times the
// change of the rotation. What it moves while it is passed over is its debt,
// taken off its points' slacks when it is next looked at. The chunks left to look
// at are listed, and the warps take them from the list one by one.
template <int G, int C, class H>
__device__ __forceinline__ void icp_match(const double4 *src, uint32_t ns, const CloudView &tgt,
                                          double r2, bool fresh, IcpBlock<G, C> &b,
                                          const IcpMemory<H> &m, uint32_t &status) {
  const unsigned FULL = 0xffffffffu;
  IcpShared &sh = b.s;
  const int lane = threadIdx.x & 31;
  constexpr int WARPS = 4 * G;
  const int warp = threadIdx.x >> 5;
  const float r_up = root_above(r2);
  auto move_of = [&](const double4 &p, double &x, double &y, double &z) {
    double xp, yp, zp;
    apply_pose(sh.t, p.x, p.y, p.z, x, y, z);
    apply_pose(sh.tp, p.x, p.y, p.z, xp, yp, zp);
    const double mx = x - xp, my = y - yp, mz = z - zp;
    return root_above((mx * mx + my * my) + mz * mz);
  };
  auto search_for = [&](uint32_t i) {
    const double4 p = ldg4(src + i);
    double x, y, z;
    apply_pose(sh.t, p.x, p.y, p.z, x, y, z);
    float sl;
    const int s = nearest_guarded(tgt, x, y, z, r2, fresh ? -1 : hint_get(m.hint, i), sl, status);
    hint_set(m.hint, i, s);
    m.slack[i] = sl;
    if (m.chunks) atomic_min_slack(&m.chunks[i >> 5].slack, s < 0 ? sl : -1.0f);
  };
  constexpr bool DEALT = G == 4;
  uint32_t *queue = b.queue + 64 * warp;
  int n_q = 0;
  auto search = [&](bool drain) {
    while (n_q >= 32 || (drain && n_q > 0)) {
      const int take = min(n_q, 32);
      n_q -= take;
      if (lane < take) search_for(queue[n_q + lane]);
      __syncwarp();
    }
  };
  const uint32_t chunks = (ns + 31u) / 32u;
  for (uint32_t base = 0; base < chunks; base += ICP_BLOCK * G * C) {
    if (threadIdx.x == 0) sh.todo = sh.next = 0;
    __syncthreads();
    const uint32_t mine = base + threadIdx.x * C + cta_rank<C>();
    bool look = mine < chunks;
    float debt = 0.0f;
    if (look && !fresh && m.chunks) {
      IcpChunk &ch = m.chunks[mine];
      debt = ch.debt;
      if (ch.slack >= 0.0f) {
        const float4 ball = m.balls[mine];
        double x, y, z;
        const float move = move_of(make_double4(ball.x, ball.y, ball.z, 0.0), x, y, z);
        const float mag = fabsf(float(x)) + fabsf(float(y)) + fabsf(float(z)) + ball.w;
        const float bound = (move + sh.turn * ball.w) * 1.00001f + 1e-9f * mag;
        const float left = __fsub_rd(ch.slack, bound);
        if (left > r_up) {
          look = false;
          ch.slack = left;
          ch.debt = debt + bound;
        }
      }
    }
    const unsigned wanted = __ballot_sync(FULL, look);
    if (wanted) {
      unsigned at = 0;
      if (lane == 0) at = atomicAdd(&sh.todo, unsigned(__popc(wanted)));
      at = __shfl_sync(FULL, at, 0) + __popc(wanted & ((1u << lane) - 1u));
      if (look) {
        b.list[at] = mine;
        b.owed[at] = debt;
      }
    }
    __syncthreads();
    const unsigned n_todo = sh.todo;
    // One chunk, the warp's lanes on its points; returns who needs a search.
    auto test = [&](unsigned k) {
      const uint32_t c = b.list[k], i = 32u * c + lane;
      const float owed = b.owed[k];
      const bool in = i < ns;
      bool need = in;
      float bound = f_inf();  // this point's share of the chunk's bound
      if (fresh) {
        if (m.chunks) {
          const double4 p = ldg4(src + min(i, ns - 1u));
          chunk_ball(p, m.balls + c, lane);
        }
      } else if (in) {
        const float sl0 = m.slack[i];
        const int s = hint_get(m.hint, i);
        const double4 p = ldg4(src + i);
        double x, y, z;
        const float sl = __fsub_rd(__fsub_rd(sl0, owed * 1.00001f), move_of(p, x, y, z));
        if (s >= 0) {
          const double4 q = ldg4(tgt.pts + s);
          const double dx = x - q.x, dy = y - q.y, dz = z - q.z;
          const double d2 = (dx * dx + dy * dy) + dz * dz;
          if (root_above(d2) < sl) {
            need = false;
            if (d2 <= r2) {
              m.slack[i] = sl;
              bound = -1.0f;
            } else {  // out of the radius, and every other point farther still
              hint_set(m.hint, i, -1);
              m.slack[i] = bound = root_approx(__double2float_rd(d2)) * 0.999999f;
            }
          }
        } else if (sl > r_up) {
          need = false;
          m.slack[i] = bound = sl;
        }
      }
      if (m.chunks) {
        // The searches still to come lower it.
        bound = warp_min(bound);
        if (lane == 0) m.chunks[c] = IcpChunk{bound, 0.0f};
      }
      return __ballot_sync(FULL, need);
    };
    if constexpr (!DEALT) {
      // Many items in flight: the warps take chunks one by one, and search
      // whenever they have 32 points.
      for (;;) {
        unsigned k = 0;
        if (lane == 0) k = atomicAdd(&sh.next, 1u);
        k = __shfl_sync(FULL, k, 0);
        if (k >= n_todo) break;
        const unsigned mask = test(k);
        if (mask >> lane & 1u) queue[n_q + __popc(mask & ((1u << lane) - 1u))] = 32u * b.list[k] + lane;
        n_q += __popc(mask);
        __syncwarp();
        search(false);
      }
      __syncthreads();  // the list is used up
    } else {
      // Few items: what counts is how long the longest warp takes. Two chunks a
      // warp, then what they leave to search for is dealt out evenly. (With many
      // items in flight the two barriers cost more than the balance is worth: a
      // pot's ladder took 74 ms this way against 64.)
      for (unsigned k0 = 0; k0 < n_todo; k0 += 2 * WARPS) {
        if (threadIdx.x == 0) sh.next = 0;
        __syncthreads();
        for (unsigned q = 0; q < 2; ++q) {
          const unsigned k = k0 + WARPS * q + warp;
          if (k >= n_todo) break;  // the same for the warp
          const unsigned mask = test(k);
          if (!mask) continue;
          unsigned at = 0;
          if (lane == 0) at = atomicAdd(&sh.next, unsigned(__popc(mask)));
          at = __shfl_sync(FULL, at, 0) + __popc(mask & ((1u << lane) - 1u));
          if (mask >> lane & 1u) b.queue[at] = 32u * b.list[k] + lane;
        }
        __syncthreads();
        const unsigned total = sh.next, share = (total + WARPS - 1) / WARPS;
        for (unsigned e = lane; e < share; e += 32)
          if (warp * share + e < total) search_for(b.queue[warp * share + e]);
        __syncthreads();
      }
    }
  }
  if (!DEALT) search(true);
}

// ---- sums -----------------------------------------------------------------------

// Sum k's total from the warps' partial sums, in warp order: the final sum of
// the partials is compensated (TwoSum over the warps' sums, their carried
// errors added once at the end), so the total is the partials' exact sum up to a
// last rounding whatever their magnitudes.
__device__ __forceinline__ double block_total(const IcpShared &sh, int k) {
  double v = sh.red[0][k], c = sh.carry[0][k];
  for (int w = 1; w < ICP_BLOCK / 32; ++w) {
    double s, e;
    two_sum(v, sh.red[w][k], s, e);
    v = s;
    c = (c + sh.carry[w][k]) + e;
  }
  return v + c;
}

// sh.sums[lo..hi) of this CTA.
__device__ __forceinline__ void reduce_sums(IcpShared &sh, int lo, int hi) {
  __syncthreads();
  if (int(threadIdx.x) >= lo && int(threadIdx.x) < hi)
    sh.sums[threadIdx.x] = block_total(sh, threadIdx.x);
  __syncthreads();
}

// The two terms (indices into row[6], r, d2, 1) whose product sum k adds up:
// 0 the count, 1 the squared error, then J^T J's lower triangle and J^T r.
__host__ __device__ constexpr int term_a(int k) {
  if (k < 2) return k == 0 ? 8 : 7;
  if (k >= 23) return k - 23;
  int row = 0, q = k - 2;
  while (q > row) q -= ++row;
  return row;
}
__host__ __device__ constexpr int term_b(int k) {
  if (k < 2) return 8;
  if (k >= 23) return 6;
  int row = 0, q = k - 2;
  while (q > row) q -= ++row;
  return q;
}

// One point's products of sums B..B+N-1 added to acc.
template <int B, int N>
__device__ __forceinline__ void add_terms(const double (&c)[ICP_TERMS], double (&acc)[N]) {
#pragma unroll
  for (int k = 0; k < N; ++k)
    if (B + k < ICP_SUMS) acc[k] += c[term_a(B + k)] * c[term_b(B + k)];
}
// The same, its terms read from the tile column `col`.
template <int G, int B, int N, int W>
__device__ __forceinline__ void add_tile(const double (&tile)[ICP_TERMS][W], int col,
                                         double (&acc)[N]) {
  double c[ICP_TERMS];
#pragma unroll
  for (int k = 0; k < ICP_TERMS; ++k) c[k] = tile[k][col];
  add_terms<B, N>(c, acc);
}

// One point's terms for the sums (the squared distance re-formed exactly as the
// search formed it); zeros, which add nothing, where there is no correspondence.
template <class H, int C>
__device__ __forceinline__ bool point_terms(const double4 *src, uint32_t ns, const CloudView &tgt,
                                            double r2, const double *t, const H *hint, uint32_t i,
                                            double (&e)[ICP_TERMS]) {
#pragma unroll
  for (int k = 0; k < ICP_TERMS; ++k) e[k] = 0.0;
  const int s = i < ns ? hint_load<C>(hint, i) : -1;
  if (s < 0) return false;
  const double4 p = ldg4(src + i);
  const double4 q = ldg4(tgt.pts + s);
  double x, y, z;
  apply_pose(t, p.x, p.y, p.z, x, y, z);
  const double dx = x - q.x, dy = y - q.y, dz = z - q.z;
  const double d2 = (dx * dx + dy * dy) + dz * dz;
  if (!(d2 < r2)) return false;
  e[7] = d2;
  e[8] = 1.0;
  if (tgt.nrm) {
    const double4 n = ldg4(tgt.nrm + s);
    e[0] = y * n.z - z * n.y;
    e[1] = z * n.x - x * n.z;
    e[2] = x * n.y - y * n.x;
    e[3] = n.x;
    e[4] = n.y;
    e[5] = n.z;
    e[6] = (x - q.x) * n.x + (y - q.y) * n.y + (z - q.z) * n.z;
  }
  return true;
}

// The pass's 29 sums over the correspondences in hint[] into sh.sums of every
// CTA, by one of three schemes.
//
// 256 threads (many items in flight): warp w of a group holds partials 32 w to
// 32 w + 31 of the group's half of the sums, which chunks w, w + 4, ... add to,
// and goes over those of them that have a match. Both groups form a chunk's
// terms; sharing them through shared memory took a barrier every 256 points and
// all the chunks between (a pot's ladder of 1792 items: 61.8 ms, 51.7 this way).
//
// 512 threads: rounds of 512 points, each thread forming one point's terms into
// the shared tile, then thread v of group g adding the round's points v, v + 128,
// ... to partial v of the group's quarter of the sums.
//
// A cluster: the partials are dealt out over the CTAs, 128 / C each with the
// points that are theirs, and every CTA gets all of them for the last steps; its
// threads hold NS sums of one partial. (With the sums dealt out instead, every
// CTA needs every point's terms: forming them again in each CTA took 60 k cycles
// a pass of 6000 points on clusters of 8, reading them from the other CTAs'
// shared memory 75 k.)
template <int G, int C, class H>
__device__ __forceinline__ void icp_sums(const double4 *src, uint32_t ns, const CloudView &tgt,
                                         double r2, bool valid, IcpBlock<G, C> &b,
                                         const IcpMemory<H> &m) {
  IcpShared &sh = b.s;
  double e[ICP_TERMS];
  if constexpr (G == 2) {
    constexpr int NS = (ICP_SUMS + 1) / 2;
    const int lane = threadIdx.x & 31, w = (threadIdx.x >> 5) & 3, g = threadIdx.x >> 7;
    double acc[NS];
#pragma unroll
    for (int k = 0; k < NS; ++k) acc[k] = 0.0;
    const uint32_t chunks = valid ? (ns + 31u) / 32u : 0u;
    for (uint32_t base = w; base < chunks; base += 4 * 32) {
      const uint32_t mine = base + 4 * lane;
      unsigned some = __ballot_sync(0xffffffffu, mine < chunks && (!m.chunks || m.chunks[mine].slack < 0.0f));
      while (some) {
        const int q = __ffs(some) - 1;
        some &= some - 1u;
        if (point_terms<H, C>(src, ns, tgt, r2, sh.t, m.hint, 32u * (base + 4 * q) + lane, e)) {
          if (g == 0)
            add_terms<0, NS>(e, acc);
          else
            add_terms<NS, NS>(e, acc);
        }
      }
    }
    store_warp_sums<NS>(acc, g * NS, sh);
  } else if constexpr (C == 1) {
    constexpr int NS = (ICP_SUMS + G - 1) / G;
    const int g = threadIdx.x >> 7, v = threadIdx.x & 127;
    double acc[NS];
#pragma unroll
    for (int k = 0; k < NS; ++k) acc[k] = 0.0;
    for (uint32_t base = 0; valid && base < ns; base += ICP_BLOCK * G) {
      if (m.chunks) {  // a round of chunks without matches (the same for the block)
        bool some = false;
#pragma unroll
        for (int u = 0; u < 4 * G; ++u)
          if (base + 32u * u < ns) some = some || __ldcg(&m.chunks[(base >> 5) + u].slack) < 0.0f;
        if (!some) continue;
      }
      const bool ok = point_terms<H, C>(src, ns, tgt, r2, sh.t, m.hint, base + threadIdx.x, e);
#pragma unroll
      for (int k = 0; k < ICP_TERMS; ++k) b.tile[k][threadIdx.x] = e[k];
      if (!__syncthreads_or(ok)) continue;  // no correspondence in the round
#pragma unroll
      for (int u = 0; u < G; ++u) {
        const int col = v + ICP_BLOCK * u;
        if (g == 0) add_tile<G, 0, NS>(b.tile, col, acc);
        if (g == 1) add_tile<G, NS, NS>(b.tile, col, acc);
        if (g == 2) add_tile<G, 2 * NS, NS>(b.tile, col, acc);
        if (g == 3) add_tile<G, 3 * NS, NS>(b.tile, col, acc);
      }
      __syncthreads();
    }
    store_warp_sums<NS>(acc, g * NS, sh);
  } else {
    constexpr int V = ICP_BLOCK / C;          // partials of a CTA
    constexpr int J = ICP_BLOCK * G / V;      // 128-point blocks a round, and shares of the sums
    constexpr int NS = (ICP_SUMS + J - 1) / J;
    const int v = threadIdx.x % V, j = threadIdx.x / V, k0 = j * NS;
    const uint32_t own = V * cta_rank<C>() + v;
    double acc[NS];
    const double *ta[NS], *tb[NS];
#pragma unroll
    for (int k = 0; k < NS; ++k) {
      acc[k] = 0.0;
      ta[k] = b.tile[term_a(min(k0 + k, ICP_SUMS - 1))] + v;
      tb[k] = b.tile[term_b(min(k0 + k, ICP_SUMS - 1))] + v;
    }
    for (uint32_t base = 0; valid && base < ns; base += ICP_BLOCK * J) {
      const bool ok = point_terms<H, C>(src, ns, tgt, r2, sh.t, m.hint, base + ICP_BLOCK * j + own, e);
#pragma unroll
      for (int k = 0; k < ICP_TERMS; ++k) b.tile[k][threadIdx.x] = e[k];
      if (!__syncthreads_or(ok)) continue;
#pragma unroll 8
      for (int q = 0; q < J; ++q)
#pragma unroll
        for (int k = 0; k < NS; ++k) acc[k] += ta[k][V * q] * tb[k][V * q];
      __syncthreads();
    }
#pragma unroll
    for (int k = 0; k < NS; ++k)
      if (k0 + k < ICP_SUMS)
        for (uint32_t r = 0; r < C; ++r) peer_store(&b.part[k0 + k][own], r, acc[k]);
    rung_sync<C>();
    constexpr int NK = (ICP_SUMS + G - 1) / G;
    const int g = threadIdx.x >> 7;
    double all[NK];
#pragma unroll
    for (int k = 0; k < NK; ++k)
      all[k] = g * NK + k < ICP_SUMS ? b.part[g * NK + k][threadIdx.x & 127] : 0.0;
    store_warp_sums<NK>(all, g * NK, sh);
  }
  __syncthreads();
  if (threadIdx.x < ICP_SUMS) sh.sums[threadIdx.x] = block_total(sh, threadIdx.x);
  __syncthreads();
}

// The sums of a point-to-point pass over the correspondences in hint[]:
// MOMENTS gives count, err2 and the sums of the moved source and matched target
// points (s[0..8)); otherwise the 9 covariance terms ((q - mean_q) / n)(p -
// mean_p)^T (s[8..17)), centred as umeyama centres them (icp.rs:548-570). The first 128
// threads of each CTA call it.
template <bool MOMENTS, int C, class H>
__device__ __forceinline__ void p2p_accumulate(const double4 *src, uint32_t ns,
                                               const CloudView &tgt, const double *t, double r2,
                                               bool valid, const H *hint, const double *mean,
                                               double one_over_n, IcpShared &sh) {
  constexpr int N = MOMENTS ? 8 : 9, B = MOMENTS ? 0 : 8;
  double acc[N];
#pragma unroll
  for (int k = 0; k < N; ++k) acc[k] = 0.0;
  if (valid) {
    for (uint32_t i = threadIdx.x; i < ns; i += ICP_BLOCK) {
      int s = hint_load<C>(hint, i);
      if (s < 0) continue;
      double4 p = src[i];
      double x, y, z;
      apply_pose(t, p.x, p.y, p.z, x, y, z);
      double4 q = tgt.pts[s];
      double dx = x - q.x, dy = y - q.y, dz = z - q.z;
      double d2 = (dx * dx + dy * dy) + dz * dz;
      if (!(d2 < r2)) continue;
      if (MOMENTS) {
        acc[0] += 1.0;
        acc[1] += d2;
        acc[2] += x;
        acc[3] += y;
        acc[4] += z;
        acc[5] += q.x;
        acc[6] += q.y;
        acc[7] += q.z;
      } else {
        double a[3] = {x - mean[0], y - mean[1], z - mean[2]};
        double b[3] = {(q.x - mean[3]) * one_over_n, (q.y - mean[4]) * one_over_n,
                       (q.z - mean[5]) * one_over_n};
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
          for (int c = 0; c < 3; ++c) acc[3 * r + c] += b[r] * a[c];
      }
    }
  }
  store_warp_sums<N>(acc, B, sh);
}

// A bound on how far two rotations move a unit vector apart (the Frobenius
// norm of their difference).
__device__ __forceinline__ float rotation_change(const double *t, const double *tp) {
  double s = 0.0;
  for (int r = 0; r < 3; ++r)
    for (int c = 0; c < 3; ++c) {
      const double d = t[4 * r + c] - tp[4 * r + c];
      s += d * d;
    }
  return root_above(s);
}

// One correspondence pass (icp::correspondences + icp::normal_equations) over
// `src` under the pose sh.t; leaves the totals in sh.sums. `m` carries the
// matches from pass to pass (icp_match). Every thread of the cluster calls it,
// sh.tp and sh.turn set.
template <int G, int C, class H>
__device__ __forceinline__ void icp_pass(const double4 *src, uint32_t ns, const CloudView &tgt,
                                         double r2, bool valid, IcpBlock<G, C> &b,
                                         const IcpMemory<H> &m, bool fresh, uint32_t &status,
                                         bool point_to_point = false) {
  IcpShared &sh = b.s;
  if (valid)
    icp_match<G, C>(src, ns, tgt, r2, fresh, b, m, status);
  rung_sync<C>();
  if (point_to_point) {  // every CTA forms all the sums
    if (threadIdx.x < ICP_BLOCK)
      p2p_accumulate<true, C>(src, ns, tgt, sh.t, r2, valid, m.hint, nullptr, 0.0, sh);
    reduce_sums(sh, 0, 8);
    double one_over_n = sh.sums[0] != 0.0 ? 1.0 / sh.sums[0] : 0.0;
    double mean[6];
    for (int k = 0; k < 6; ++k) mean[k] = sh.sums[2 + k] * one_over_n;
    if (threadIdx.x < ICP_BLOCK)
      p2p_accumulate<false, C>(src, ns, tgt, sh.t, r2, valid, m.hint, mean, one_over_n, sh);
    reduce_sums(sh, 8, 17);
    // Every CTA has read every match: only now may one of them write the next
    // pass's (the point-to-plane sums have this barrier before their exchange).
    if constexpr (C > 1) rung_sync<C>();
    return;
  }
  icp_sums<G, C>(src, ns, tgt, r2, valid, b, m);
}

// Open3D's (fitness, inlier_rmse) from the pass sums (icp.rs:385-391).
__device__ __forceinline__ void fit_rmse(const double *s, uint32_t ns, double &fit, double &rmse) {
  if (s[0] == 0.0) {
    fit = 0.0;
    rmse = 0.0;
    return;
  }
  fit = s[0] / double(ns);
  rmse = sqrt(s[1] / s[0]);
}

// icp::register (icp.rs:308-356) for the pose in b.s.t of every CTA; every
// thread of the cluster calls it, after a barrier. On return b.s.t holds the
// refined pose and *out is written. `keep`: the rung before ran over the same
// clouds and its last pass at this pose, so its matches still stand.
template <int G, int C, class H>
__device__ void icp_rung_block(const double4 *src, uint32_t ns, const CloudView &tgt,
                               double distance, int max_iter, IcpBlock<G, C> &b,
                               const IcpMemory<H> &m, sherd_registration *out, uint32_t &status,
                               bool point_to_point = false, bool keep = false) {
  IcpShared &sh = b.s;
  const uint32_t rank = cta_rank<C>();
  if (ns == 0 || tgt.n == 0) {
    if (rank == 0 && threadIdx.x == 0) {
      for (int k = 0; k < 16; ++k) out->transform[k] = sh.t[k];
      out->fitness = 0.0;
      out->inlier_rmse = 0.0;
      out->correspondences = 0;
      out->iterations = 0;
      out->converged = 0;
    }
    __syncthreads();
    return;
  }
  const bool valid = distance > 0.0;  // a NaN radius is not valid either
  const double r2 = distance * distance;
  if (threadIdx.x < 16) sh.tp[threadIdx.x] = sh.t[threadIdx.x];
  if (threadIdx.x == 0) sh.turn = 0.0f;
  __syncthreads();
  icp_pass<G, C>(src, ns, tgt, r2, valid, b, m, !keep, status, point_to_point);
  double fit, rmse;
  fit_rmse(sh.sums, ns, fit, rmse);
  uint32_t iterations = 0;
  bool converged = false;
  for (int it = 0; it < max_iter; ++it) {
    if (point_to_point) {
      if (threadIdx.x < 16) sh.tp[threadIdx.x] = sh.t[threadIdx.x];
      if (threadIdx.x < 32) __syncwarp();
      if (threadIdx.x == 0) point_step(sh);
    } else if (threadIdx.x < 32) {
      plane_step(sh.sums, tgt.nrm != nullptr, sh.t, sh);
    }
    if (threadIdx.x == 0) sh.turn = rotation_change(sh.t, sh.tp);
    __syncthreads();
    icp_pass<G, C>(src, ns, tgt, r2, valid, b, m, false, status, point_to_point);
    ++iterations;
    double nfit, nrmse;
    fit_rmse(sh.sums, ns, nfit, nrmse);
    converged = fabs(nfit - fit) < 1e-6 && fabs(nrmse - rmse) < 1e-6;
    fit = nfit;
    rmse = nrmse;
    if (converged) break;
  }
  if (rank == 0) {
    if (threadIdx.x < 16) out->transform[threadIdx.x] = sh.t[threadIdx.x];
    if (threadIdx.x == 0) {
      out->fitness = fit;
      out->inlier_rmse = rmse;
      out->correspondences = (unsigned long long)sh.sums[0];
      out->iterations = iterations;
      out->converged = converged ? 1u : 0u;
    }
  }
  __syncthreads();
}

}  // namespace sherd
