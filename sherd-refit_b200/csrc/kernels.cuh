// kernels.cuh — the __global__ entry points of the backend.
#pragma once

#include "verify.cuh"

namespace sherd {

struct Pose16 {
  double m[16];
};

// ---- Executor-shaped batch kernels (one thread per query) -------------------

__global__ void k_first_hit(MeshView m, const float *org, const float *dir, uint32_t n, float *t,
                            uint32_t *prim, uint32_t *status) {
  uint32_t st = 0;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    F3 o = {org[3 * i], org[3 * i + 1], org[3 * i + 2]};
    F3 d = {dir[3 * i], dir[3 * i + 1], dir[3 * i + 2]};
    first_hit(m, o, d, t[i], prim[i], st);
  }
  if (st) atomicOr(status, st);
}

// The block's share [first, first + count) of n queries.
__device__ __forceinline__ uint32_t block_share(uint32_t n, uint32_t &first) {
  const uint32_t per = (n + gridDim.x - 1) / gridDim.x;
  first = uint32_t(min((unsigned long long)per * blockIdx.x, (unsigned long long)n));
  return min(per, n - first);
}

// Bound by the latency of the walks: a lane's faces shared by its warp, 150,000
// queries 136 -> 66 us (a thread per query with its own loop over a leaf's faces).
__global__ void __launch_bounds__(128) k_bounded_all(const __grid_constant__ MeshView m,
                                                     const double *pts, uint32_t n,
                                                     const __grid_constant__ Pose16 pose,
                                                     float window, double *out, uint32_t *status) {
  __shared__ unsigned next;
  __shared__ WalkSlots slots[4];
  if (threadIdx.x == 0) next = 0;
  __syncthreads();
  uint32_t st = 0, first;
  const uint32_t count = block_share(n, first);
  face_walks(
      &next, count, slots[threadIdx.x >> 5],
      [&](uint32_t k, FaceWalk &w) {
        const size_t i = first + k;
        double x, y, z;
        apply_pose(pose.m, pts[3 * i], pts[3 * i + 1], pts[3 * i + 2], x, y, z);
        return walk_start(w, &m, {float(x), float(y), float(z)}, window);
      },
      [&](uint32_t k, const FaceWalk &w) {
        out[size_t(first) + k] = w.best == f_inf() ? d_inf() : double(w.best);
      },
      st);
  if (st) atomicOr(status, st);
}

// DistReduce::Min: every query searches with the best distance so far as its
// window; the minimum is order-independent, so this is the CPU's scan.
__global__ void k_bounded_min(MeshView m, const double *pts, uint32_t n, Pose16 pose,
                              unsigned *best_key, uint32_t *status) {
  uint32_t st = 0;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    double x, y, z;
    apply_pose(pose.m, pts[3 * i], pts[3 * i + 1], pts[3 * i + 2], x, y, z);
    float window = key2f(*((volatile unsigned *)best_key));
    float d = mesh_distance(m, {float(x), float(y), float(z)}, window, st);
    if (d != f_inf()) atomicMin(best_key, f2key(d));
  }
  if (st) atomicOr(status, st);
}

__global__ void k_nn_within(CloudView c, const double *q, uint32_t n, double r2, uint32_t *idx,
                            double *d2, uint32_t *status) {
  uint32_t st = 0;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    double best;
    int s = nearest_within_sq(c, q[3 * i], q[3 * i + 1], q[3 * i + 2], r2, best, st);
    idx[i] = s < 0 ? MISS : uint32_t(c.pts[s].w);
    d2[i] = s < 0 ? d_inf() : best;
  }
  if (st) atomicOr(status, st);
}

__global__ void k_nn_below(CloudView c, const double *q, uint32_t n, double bound, uint32_t *idx,
                           double *dist, uint32_t *status) {
  uint32_t st = 0;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    double d = 0.0;
    int s = nearest_below(c, q[3 * i], q[3 * i + 1], q[3 * i + 2], bound, d, st);
    idx[i] = s < 0 ? MISS : uint32_t(c.pts[s].w);
    dist[i] = s < 0 ? d_inf() : d;
  }
  if (st) atomicOr(status, st);
}

// ---- preprocessing rays -------------------------------------------------------

// mesh::geometry::face_geometry (mesh/geometry.rs:70-96).
__global__ void k_face_geometry(const double *v, const uint32_t *f, uint32_t nf, double *normals,
                                double *areas, double *centroids) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nf) return;
  const double *a = v + 3 * size_t(f[3 * i]), *b = v + 3 * size_t(f[3 * i + 1]),
               *c = v + 3 * size_t(f[3 * i + 2]);
  double e1[3] = {b[0] - a[0], b[1] - a[1], b[2] - a[2]};
  double e2[3] = {c[0] - a[0], c[1] - a[1], c[2] - a[2]};
  double n[3] = {e1[1] * e2[2] - e1[2] * e2[1], e1[2] * e2[0] - e1[0] * e2[2],
                 e1[0] * e2[1] - e1[1] * e2[0]};
  double len = sqrt((n[0] * n[0] + n[1] * n[1]) + n[2] * n[2]);
  double den = len > 1e-12 ? len : 1e-12;
  if (normals)
    for (int k = 0; k < 3; ++k) normals[3 * i + k] = n[k] / den;
  if (areas) areas[i] = 0.5 * len;
  if (centroids)
    for (int k = 0; k < 3; ++k) centroids[3 * i + k] = (a[k] + b[k] + c[k]) / 3.0;
}

// thickness::cast_inward_rays (thickness.rs:115-132) fused with the filter of
// thickness_from_hits (thickness.rs:139-162, looking_back 185-204): valid hit
// distances are appended to ok[], the ones whose face looks back to far[].
__global__ void k_thickness_rays(MeshView m, const double *centroids, const double *normals,
                                 uint32_t nf, uint32_t stride, uint32_t n, float *t_out,
                                 uint32_t *prim_out, float *ok, float *far, unsigned *counts,
                                 uint32_t *status) {
  uint32_t st = 0;
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    uint32_t face = k * stride;
    const double *c = centroids + 3 * size_t(face), *nn = normals + 3 * size_t(face);
    double d[3] = {-nn[0], -nn[1], -nn[2]};
    F3 o = {float(c[0] + d[0] * 1e-3), float(c[1] + d[1] * 1e-3), float(c[2] + d[2] * 1e-3)};
    F3 dir = {float(d[0]), float(d[1]), float(d[2])};
    float t;
    uint32_t prim;
    first_hit(m, o, dir, t, prim, st);
    if (t_out) t_out[k] = t;
    if (prim_out) prim_out[k] = prim;
    if (!(isfinite(t) && prim < nf)) continue;
    ok[atomicAdd(&counts[0], 1u)] = t;
    const double *hit = normals + 3 * size_t(prim);
    double dd = -((hit[0] * nn[0] + hit[1] * nn[1]) + hit[2] * nn[2]);
    if (dd > 0.7) far[atomicAdd(&counts[1], 1u)] = t;
  }
  if (st) atomicOr(status, st);
}

// The same filter over given hits (the injected mode).
__global__ void k_thickness_filter(const double *normals, uint32_t nf, const uint32_t *idx,
                                   const float *t_hit, const uint32_t *prim, uint32_t n, float *ok,
                                   float *far, unsigned *counts) {
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    float t = t_hit[k];
    uint32_t p = prim[k];
    if (!(isfinite(t) && p < nf)) continue;
    ok[atomicAdd(&counts[0], 1u)] = t;
    const double *hit = normals + 3 * size_t(p), *from = normals + 3 * size_t(idx[k]);
    double dd = -((hit[0] * from[0] + hit[1] * from[1]) + hit[2] * from[2]);
    if (dd > 0.7) far[atomicAdd(&counts[1], 1u)] = t;
  }
}

// thickness::hist_mode (thickness.rs:212-262) over an ascending array, in one
// block: numpy's percentile(90) interpolation in the array's dtype, 60 equal
// bins over [0, p90] with numpy's edge corrections, the first fullest bin.
__global__ void k_hist_mode(const float *sorted, uint32_t n, float *out) {
  __shared__ unsigned counts[60];
  __shared__ float edges[61];
  __shared__ float range[2];
  if (threadIdx.x < 60) counts[threadIdx.x] = 0;
  if (threadIdx.x == 0) {
    float p90;
    if (n == 1) {
      p90 = sorted[0];
    } else {
      double vi = double(n - 1) * (90.0 / 100.0);
      double prev = floor(vi);
      uint32_t i = uint32_t(prev);
      double gamma = vi - prev;
      float a = sorted[i], b = sorted[i + 1 < n ? i + 1 : n - 1];
      float diff = b - a;
      p90 = gamma >= 0.5 ? b - diff * float(1.0 - gamma) : a + diff * float(gamma);
    }
    float first = 0.0f, last = p90;
    if (p90 == 0.0f) {
      first = -0.5f;
      last = 0.5f;
    }
    float step = (last - first) / 60.0f;
    for (int k = 0; k <= 60; ++k) edges[k] = float(k) * step + first;
    edges[60] = last;
    range[0] = first;
    range[1] = last;
  }
  __syncthreads();
  float first = range[0], last = range[1], denom = last - first;
  for (uint32_t j = threadIdx.x; j < n; j += blockDim.x) {
    float v = sorted[j];
    if (!(v >= first && v <= last)) continue;
    unsigned i = unsigned(((v - first) / denom) * 60.0f);
    if (i == 60u) i -= 1;
    if (v < edges[i]) i -= 1;
    if (i != 59u && v >= edges[i + 1]) i += 1;
    atomicAdd(&counts[i], 1u);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int k = 0;
    for (int i = 1; i < 60; ++i)
      if (counts[i] > counts[k]) k = i;
    *out = 0.5f * (edges[k] + edges[k + 1]);
  }
}

struct ConeConsts {
  double cos_a, sin_a;
  double cp[6], sp[6];
};

// segment::classify_faces (segment.rs:318-376): seven rays per face, a warp per
// ray and 32 faces: warp k of a block of seven casts the k-th ray of its 32 faces,
// and their votes meet in shared memory. (A thread that cast its face's seven rays
// in turn left a 66 144-face mesh 14 warps an SM, each as long as seven walks:
// 1.26 ms, 0.61 ms this way.)
constexpr int CONE_BLOCK = 7 * 32;
__global__ void __launch_bounds__(CONE_BLOCK) k_cone_votes(MeshView m, const double *centroids,
                                                           const double *normals, const double *ns,
                                                           const double *hit_normals, uint32_t nf,
                                                           double thick, ConeConsts cc, uint8_t *good,
                                                           uint32_t *status) {
  __shared__ unsigned votes[32];
  const int lane = threadIdx.x & 31, k = threadIdx.x >> 5;
  uint32_t st = 0;
  const float min_hit = float(0.1 * thick);
  const float thick_f = float(thick);
  for (uint32_t base = blockIdx.x * 32u; base < nf; base += gridDim.x * 32u) {
    if (k == 0) votes[lane] = 0;
    __syncthreads();
    const uint32_t i = base + lane;
    if (i < nf) {
      const double *n = ns + 3 * size_t(i), *fnv = normals + 3 * size_t(i),
                   *c = centroids + 3 * size_t(i);
      bool finite = isfinite(n[0]) && isfinite(n[1]) && isfinite(n[2]);
      double a[3] = {1.0, 0.0, 0.0};
      if (!(fabs(n[0]) < 0.9)) {
        a[0] = 0.0;
        a[1] = 1.0;
      }
      double cr[3] = {n[1] * a[2] - n[2] * a[1], n[2] * a[0] - n[0] * a[2],
                      n[0] * a[1] - n[1] * a[0]};
      double len = sqrt((cr[0] * cr[0] + cr[1] * cr[1]) + cr[2] * cr[2]);
      if (finite && len > 0.0) {
        F3 o = {float(c[0] - fnv[0] * 1e-3), float(c[1] - fnv[1] * 1e-3),
                float(c[2] - fnv[2] * 1e-3)};
        double d[3];
        if (k == 0) {
          d[0] = -n[0];
          d[1] = -n[1];
          d[2] = -n[2];
        } else {
          double e1[3] = {cr[0] / len, cr[1] / len, cr[2] / len};
          double e2[3] = {n[1] * e1[2] - n[2] * e1[1], n[2] * e1[0] - n[0] * e1[2],
                          n[0] * e1[1] - n[1] * e1[0]};
          double cp = cc.cp[k - 1], sp = cc.sp[k - 1];
          for (int q = 0; q < 3; ++q) d[q] = -(cc.cos_a * n[q]) + cc.sin_a * (cp * e1[q] + sp * e2[q]);
        }
        F3 dir = {float(d[0]), float(d[1]), float(d[2])};
        float dh;
        uint32_t prim;
        first_hit(m, o, dir, dh, prim, st);
        if (prim != MISS && isfinite(dh) && prim < nf && !(dh <= min_hit)) {
          float ratio = dh / thick_f;
          if (!(ratio <= 0.5f || ratio >= 1.8f)) {
            const double *h = hit_normals + 3 * size_t(prim);
            double al = (h[0] * d[0] + h[1] * d[1]) + h[2] * d[2];
            if (al > 0.7) atomicAdd(&votes[lane], 1u);
          }
        }
      }
    }
    __syncthreads();
    if (k == 0 && i < nf) good[i] = uint8_t(votes[lane]);
    __syncthreads();
  }
  if (st) atomicOr(status, st);
}

// ---- ICP -----------------------------------------------------------------------

// Executor::icp_rung: one block of 128 G threads, or one cluster of C of them,
// per candidate.
template <int G, int C>
__global__ void __launch_bounds__(ICP_BLOCK *G, 4 / G)
    k_icp_rung(const double4 *src, uint32_t ns, CloudView tgt, const double *inits,
               sherd_icp_options opt, IcpMemory<int> mem, sherd_registration *out,
               uint32_t *status) {
  IcpBlock<G, C> &b = rung_memory<G, C>();
  uint32_t st = 0;
  const uint32_t cand = blockIdx.x / C;
  if (threadIdx.x < 16) {
    double v = inits[16 * size_t(cand) + threadIdx.x];
    b.s.t[threadIdx.x] = v;
    // A non-finite start (which only a caller passing device-resident poses can hand over,
    // the host-buffer entry refusing it first) is reported; the rung itself stays in bounds
    // (no distance compares below a NaN radius, so it finds no correspondence).
    if (!isfinite(v)) st |= ST_RANGE;
  }
  __syncthreads();
  icp_rung_block<G, C>(src, ns, tgt, opt.max_correspondence_distance, opt.max_iteration, b,
                       memory_slot(mem, cand, ns), out + cand, st,
                       opt.estimation == SHERD_POINT_TO_POINT);
  rung_sync<C>();  // no CTA of a cluster ends while another may write to it
  if (st) atomicOr(status, st);
}

// Executor::coarse_scores (cpu.rs:46-68, 136-169): one warp per pose, its
// lanes over the points, the agreeing points counted by ballot.
__global__ void k_coarse_scores(CloudView tgt, const double *pts, const double *nrm, uint32_t n,
                                const double *poses, uint32_t k, double radius,
                                double normal_agree, double *out, uint32_t *status) {
  uint32_t st = 0;
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t h = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; h < k; h += warps) {
    const double *t = poses + 16 * size_t(h);
    uint32_t agree = 0;
    for (uint32_t base = 0; base < n; base += 32) {
      uint32_t i = base + lane;
      bool ok = false;
      if (i < n) {
        double x, y, z;
        apply_pose(t, pts[3 * size_t(i)], pts[3 * size_t(i) + 1], pts[3 * size_t(i) + 2], x, y, z);
        double d;
        int s = nearest_below(tgt, x, y, z, radius, d, st);
        if (s >= 0) {
          double u, v, w;
          rotate_pose(t, nrm[3 * size_t(i)], nrm[3 * size_t(i) + 1], nrm[3 * size_t(i) + 2], u, v, w);
          double4 m = ldg4(tgt.nrm + s);
          ok = (m.x * u + m.y * v) + m.z * w > normal_agree;
        }
      }
      agree += __popc(__ballot_sync(0xFFFFFFFFu, ok));
    }
    if (lane == 0) out[h] = n ? double(agree) / double(n) : 0.0;
  }
  if (st) atomicOr(status, st);
}

// verify::penetration_share (verify.rs:509-527): points inside the mesh and
// deeper than `pen`, counted per warp by ballot.
__global__ void k_penetration_share(MeshView m, const double *pts, uint32_t n, Pose16 pose,
                                    double pen, unsigned long long *count, uint32_t *status) {
  uint32_t st = 0;
  unsigned long long mine = 0;
  for (uint32_t base = blockIdx.x * blockDim.x; base < n; base += gridDim.x * blockDim.x) {
    uint32_t i = base + threadIdx.x;
    bool deeper = false;
    if (i < n) {
      double x, y, z;
      apply_pose(pose.m, pts[3 * size_t(i)], pts[3 * size_t(i) + 1], pts[3 * size_t(i) + 2], x, y, z);
      F3 p = {float(x), float(y), float(z)};
      bool in_box = !(p.x < m.lo[0] || p.x > m.hi[0] || p.y < m.lo[1] || p.y > m.hi[1] ||
                      p.z < m.lo[2] || p.z > m.hi[2]);
      if (in_box && inside_mesh(m, p))
        deeper = double(mesh_distance(m, p, f_inf(), st)) > pen;
    }
    unsigned ballot = __ballot_sync(0xFFFFFFFFu, deeper);
    if ((threadIdx.x & 31) == 0) mine += __popc(ballot);
  }
  if ((threadIdx.x & 31) == 0 && mine) atomicAdd(count, mine);
  if (st) atomicOr(status, st);
}

// ---- the batched stage-2 path ----------------------------------------------------

// The forms k_ladder is built in. The first three are a block of 256 threads per
// item with a register budget for so many resident CTAs per SM; the batch picks
// one per point-count bucket (the autotuner in sherd.cu). The others are blocks
// of 512 threads, alone or in clusters of 2, 4 and 8 per item, for batches with
// fewer items than such blocks fill the device (ladder_form in sherd.cu).
constexpr int LADDER_VARIANTS = 3;
constexpr int LADDER_MINB[LADDER_VARIANTS] = {3, 4, 5};
// The variant a bucket runs until the autotuner has timed it (and when it has
// too few items to time).
constexpr int LADDER_DEFAULT = 1;

// How a running kernel hears of sherd_abort: the host's flag is mapped memory,
// a read of it crosses the bus (about 0.8 us each, one after the other for the
// whole device: a warp that polled it when it started made 4736 warps wait 3.8 ms
// for their first chunk), so one thread at a time reads it, every POLL_NS, and
// the rest read its copy on the device. The copy is cleared with the status word.
struct StopCtl {
  const uint32_t *host;       // host-mapped; non-zero asks the kernel to stop (null: never)
  uint32_t *seen;             // the device's copy
  unsigned long long *polled; // when it was last refreshed (global_ns)
};
constexpr unsigned long long POLL_NS = 20000;

__device__ __forceinline__ bool stop_asked(const StopCtl &c) {
  if (!c.host) return false;
  if (*((volatile uint32_t *)c.seen)) return true;
  const unsigned long long last = *((volatile unsigned long long *)c.polled), now = global_ns();
  if (now - last < POLL_NS || atomicCAS(c.polled, last, now) != last) return false;
  if (!*((volatile const uint32_t *)c.host)) return false;
  *((volatile uint32_t *)c.seen) = 1u;
  return true;
}

struct QueueCtl {
  unsigned *head;             // next queue position to take
  const uint32_t *order;      // item indices, most expensive first
  uint32_t n;                 // queue length
  StopCtl stop;
  unsigned long long budget_ns;
};

// Takes the next queue entry for the whole block, or returns false when the
// queue is empty, the host asked to stop or the time budget is spent.
__device__ __forceinline__ bool take(const QueueCtl &q, unsigned long long start, unsigned &slot,
                                     uint32_t &st) {
  __shared__ unsigned s_item;
  if (threadIdx.x == 0) {
    unsigned item = 0xFFFFFFFFu;
    if (stop_asked(q.stop)) {
      st |= ST_ABORTED;
    } else if (q.budget_ns && global_ns() - start > q.budget_ns) {
      st |= ST_TIMEOUT;
    } else {
      unsigned pos = atomicAdd(q.head, 1u);
      if (pos < q.n) item = q.order[pos];
    }
    s_item = item;
  }
  __syncthreads();
  slot = s_item;
  __syncthreads();
  return slot != 0xFFFFFFFFu;
}

// take() for a cluster of C blocks: the first block's answer for all of them.
template <int C>
__device__ __forceinline__ bool take_shared(const QueueCtl &q, unsigned long long start,
                                            unsigned &slot, uint32_t &st) {
  if constexpr (C == 1) {
    return take(q, start, slot, st);
  } else {
    __shared__ unsigned s_got;
    if (cta_rank<C>() == 0) {
      unsigned got;
      take(q, start, got, st);
      if (threadIdx.x < C) peer_store(&s_got, threadIdx.x, got);
    }
    rung_sync<C>();
    slot = s_got;
    rung_sync<C>();
    return slot != 0xFFFFFFFFu;
  }
}

// R 5.6's point-to-plane rungs r_lo..r_hi-1 of the four per (pair, start)
// (ladder.rs:142-161): from the item's start pose when r_lo is 0, else from
// its rung r_lo - 1, on one block of 128 G threads or a cluster of C of them per
// item. With skip_partial, items an early rejection left partial are passed over.
template <class H, int G, int C, int MINB>
__global__ void __launch_bounds__(ICP_BLOCK *G, MINB) k_ladder(const PairView *pairs,
                                                      const sherd_work_item *items, QueueCtl q,
                                                      IcpMemory<H> mem, size_t stride,
                                                      sherd_candidate *out, int r_lo, int r_hi,
                                                      int skip_partial, uint32_t *status) {
  IcpBlock<G, C> &b = rung_memory<G, C>();
  uint32_t st = 0;
  const IcpMemory<H> mine = memory_slot(mem, blockIdx.x / C, stride);
  unsigned long long start = global_ns();
  unsigned it;
  // A CTA's shared memory may be written by another once it is known to run.
  if constexpr (C > 1) rung_sync<C>();
  while (take_shared<C>(q, start, it, st)) {
    const sherd_work_item &w = items[it];
    const PairView &pr = pairs[w.pair];
    sherd_candidate *c = out + it;
    if (skip_partial && c->scores.partial) continue;  // the same for every block of the item
    if (threadIdx.x < 16)
      b.s.t[threadIdx.x] = r_lo == 0 ? w.init[threadIdx.x] : c->rungs[r_lo - 1].transform[threadIdx.x];
    if (threadIdx.x == 0 && cta_rank<C>() == 0 && r_lo == 0) {
      c->pair = w.pair;
      c->start = w.start;
    }
    __syncthreads();
    const double k[4] = {0.2, 0.08, 0.08, 0.04};
    for (int r = r_lo; r < r_hi; ++r) {
      const double distance = k[r] * pr.sc.t * pr.sc.icp;
      // Rungs 1 and 3 follow a rung over the same clouds (0 and 2): when that
      // rung ran in this launch, its matches still stand.
      const bool keep = (r & 1) && r > r_lo;
      const bool reg = r < 2;
      icp_rung_block<G, C>(reg ? pr.reg_src : pr.frac_src, reg ? pr.n_reg : pr.n_frac,
                           reg ? pr.reg_tgt : pr.frac_tgt, distance, 30, b, mine,
                           &c->rungs[r], st, false, keep);
    }
  }
  if (st) atomicOr(status, st);
}

// R 6 + R 6.5 at each item's rung `pose_rung` pose (verify.rs:590-638): the
// last rung, or rung 1 for R 5.6's early-rejection check (full = 0). With
// `inv` set, the penetration half is left to the wavefront kernels below and
// the inverse pose of every item is written for them. With skip_partial,
// items an early rejection left partial are passed over.
__global__ void __launch_bounds__(VER_BLOCK, 3) k_verify_items(const PairView *pairs,
                                                            const sherd_work_item *items,
                                                            QueueCtl q, sherd_params p,
                                                            unsigned *scratch, size_t stride,
                                                            sherd_candidate *out, int full,
                                                            double *inv, int pose_rung,
                                                            int skip_partial, uint32_t *status) {
  __shared__ VerShared sh;
  uint32_t st = 0;
  unsigned long long start = global_ns();
  unsigned *mine = scratch + stride * blockIdx.x;
  unsigned it;
  while (take(q, start, it, st)) {
    const PairView &pr = pairs[items[it].pair];
    sherd_candidate *c = out + it;
    if (skip_partial && c->scores.partial) continue;  // the same for the whole block
    if (threadIdx.x < 16) sh.t[threadIdx.x] = c->rungs[pose_rung].transform[threadIdx.x];
    __syncthreads();
    if (pr.scratch_floats > stride) {
      if (threadIdx.x == 0) {
        st |= ST_SCRATCH;
        c->status = uint32_t(-SHERD_E_INVALID);
      }
      __syncthreads();
      continue;
    }
    verify_block(pr, full != 0, p, mine, sh, &c->scores, &c->accepted, st, inv == nullptr,
                 inv ? inv + 16 * size_t(it) : nullptr);
  }
  if (st) atomicOr(status, st);
}

// k_verify_items for few items, the penetration left to the wavefront kernels: the
// four scores of an item (the two fracture sides, the seam, the continuity) on a
// block each, of 1024 threads, side by side. What an item takes is then its
// longest score's few rounds of queries, where one 256-thread block went through
// all four: ten items 1.26 ms, 0.35 ms this way. With more blocks than two per SM
// the SMs are full either way and the persistent form stays (verify_in_parts).
constexpr int PART_BLOCK = 1024;
__global__ void __launch_bounds__(PART_BLOCK) k_verify_parts(const PairView *pairs,
                                                             const sherd_work_item *items,
                                                             unsigned *scratch, size_t stride,
                                                             sherd_candidate *out, int full,
                                                             double *inv, int pose_rung,
                                                             StopCtl stop, uint32_t *status) {
  __shared__ VerShared sh;
  uint32_t st = 0;
  // Asked to stop (in the ladder, say): as a queue would, nothing more is begun.
  if (__syncthreads_or(threadIdx.x == 0 && stop_asked(stop))) {
    if (threadIdx.x == 0) atomicOr(status, ST_ABORTED);
    return;
  }
  const uint32_t it = blockIdx.x >> 2, part = blockIdx.x & 3u;
  const PairView &pr = pairs[items[it].pair];
  sherd_candidate *c = out + it;
  unsigned *mine = scratch + stride * blockIdx.x;
  if (threadIdx.x < 16) sh.t[threadIdx.x] = c->rungs[pose_rung].transform[threadIdx.x];
  __syncthreads();
  if (threadIdx.x == 0) pose_inverse(sh.t, sh.inv);
  __syncthreads();
  const sherd_scales &sc = pr.sc;
  double x = 0.0, y = 0.0, z = 0.0;
  if (part == 0) {
    if (threadIdx.x < 16) inv[16 * size_t(it) + threadIdx.x] = sh.inv[threadIdx.x];
    one_side(pr.b.pf, pr.b.n_pf, sh.t, pr.a.frac, pr.b.frac_area, sc, mine, sh, x, y, z, st);
  } else if (part == 1) {
    one_side(pr.a.pf, pr.a.n_pf, sh.inv, pr.b.frac, pr.a.frac_area, sc, mine, sh, x, y, z, st);
  } else if (part == 2) {
    x = seam_score(pr, sh, st);
  } else {
    x = 1.0;
    y = -1.0;
    if (full) {
      unsigned long long *steps = reinterpret_cast<unsigned long long *>(mine);
      continuity(pr, steps, steps + pr.b.n_margin, sh, x, y, st);
    }
  }
  if (threadIdx.x == 0) {
    sherd_scores &s = c->scores;
    if (part == 0) {
      s.tight_b = x;
      s.gap_b = y;
      s.contact_b = z;
    } else if (part == 1) {
      s.tight_a = x;
      s.gap_a = y;
      s.contact_a = z;
    } else if (part == 2) {
      s.seam = x;
    } else {
      s.cont = x;
      s.cont_n = y;
    }
  }
  if (st) atomicOr(status, st);
}

// The rest of an item's scores, as verify_block leaves them.
__global__ void k_verify_join(const PairView *pairs, const sherd_work_item *items,
                              sherd_candidate *out, int full, uint32_t n) {
  const uint32_t it = blockIdx.x * blockDim.x + threadIdx.x;
  if (it >= n) return;
  const PairView &pr = pairs[items[it].pair];
  sherd_scores &s = out[it].scores;
  s.tight = fmin(s.tight_a, s.tight_b);
  s.gap = fmax(s.gap_a, s.gap_b);
  s.contact = fmin(s.contact_a, s.contact_b);
  s.gap_limit = pr.sc.gap / pr.sc.t;
  s.tight_delta = pr.sc.tight / pr.sc.t;
  s.pen = 0.0;
  s.pen_depth = 0.0;
  s.pen_unavailable =
      full && (!pr.a.has_mesh || !pr.b.has_mesh || !(pr.a.watertight && pr.b.watertight)) ? 1u : 0u;
  s.partial = full ? 0u : 1u;
  s.brk = 0.0;
  s.brk_best = 0.0;
}

// R 5.6's early rejection (pair.rs:315-340) after the fracture and seam
// scores at rung 1: an item below the tight limit keeps those partial scores,
// is rejected, and its pc_frac rungs stay unrun (the rung-1 pose, zero
// counts); the others are cleared to go on.
__global__ void k_early_mark(sherd_candidate *cands, const uint32_t *order, uint32_t n,
                             double limit) {
  uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  sherd_candidate &c = cands[order[k]];
  if (c.status) return;
  if (c.scores.tight < limit) {
    for (int r = 2; r < 4; ++r) {
      sherd_registration &g = c.rungs[r];
      for (int k = 0; k < 16; ++k) g.transform[k] = c.rungs[1].transform[k];
      g.fitness = 0.0;
      g.inlier_rmse = 0.0;
      g.correspondences = 0;
      g.iterations = 0;
      g.converged = 0;
    }
    c.accepted = 0;
  } else {
    c.scores.partial = 0;
  }
}

// ---- the penetration wavefront of the batched path ------------------------------
//
// R 6.4 for every (item, side) of a batch at once: side 0 is B's surface
// samples moved by T against A's mesh, side 1 A's moved by T^-1 against B's.
// The samples of all units are one flat list of 32-point chunks that warps
// take from a global counter, so no block ever waits at a barrier for its
// slowest lane. Each warp keeps two shared queues: the points of its chunks
// that fall in the mesh's box, and the ones the parity test calls inside; a
// queue is drained 32 entries at a time, so the parity and depth queries run
// with every lane of the warp busy. A unit's count, deepest depth and minimum
// distance are combined with global atomics, which makes them independent of
// the order the points are taken in, as R 6.4's statistics are.

struct PenState {
  unsigned *deeper;    // per unit: points deeper than sc.pen
  unsigned *deep;      // per unit: f2key(deepest depth) + 1, 0 when nothing is inside
  unsigned *best;      // per unit: f2key(smallest distance) for the nothing-inside case
  const uint32_t *chunk0;  // per unit: its first chunk in the flat list (n_units + 1)
  const uint32_t *coarse;  // the unit of every 256th chunk (chunk k << 8)
  uint32_t n_units, n_chunks;
  uint32_t run;  // chunks per run of the inside pass
};

struct PenUnit {
  const double4 *pts;
  uint32_t n;
  const MeshView *mesh;
  const double *pose;
  double pen;
  bool avail;
};

__device__ __forceinline__ PenUnit pen_unit(const PairView *pairs, const sherd_work_item *items,
                                            const sherd_candidate *cands, const double *inv,
                                            uint32_t u) {
  uint32_t item = u >> 1, side = u & 1u;
  const PairView &pr = pairs[items[item].pair];
  PenUnit x;
  x.avail = pr.a.has_mesh && pr.b.has_mesh && pr.a.watertight && pr.b.watertight &&
            !cands[item].scores.partial;
  x.pts = side ? pr.a.s : pr.b.s;
  x.n = side ? pr.a.n_s : pr.b.n_s;
  x.mesh = side ? &pr.b.mesh : &pr.a.mesh;
  x.pose = side ? inv + 16 * size_t(item) : cands[item].rungs[3].transform;
  x.pen = pr.sc.pen;
  return x;
}

// The unit a chunk belongs to: the unit of the last 256-chunk mark before it,
// then forward over the units that start at or before it (units without
// chunks included).
__device__ __forceinline__ uint32_t unit_of_chunk(const PenState &ps, uint32_t chunk) {
  uint32_t u = __ldg(ps.coarse + (chunk >> 8));
  while (__ldg(ps.chunk0 + u + 1) <= chunk) ++u;
  return u;
}

struct WarpQueue {
  unsigned long long box[64];
  unsigned long long in[64];
  int n_box, n_in;
};

__device__ __forceinline__ void wq_push(unsigned long long *q, int *count, bool pred,
                                        unsigned long long v) {
  unsigned mask = __ballot_sync(0xffffffffu, pred);
  int lane = threadIdx.x & 31;
  int base = *count;
  if (pred) q[base + __popc(mask & ((1u << lane) - 1u))] = v;
  __syncwarp();
  if (lane == 0) *count = base + __popc(mask);
  __syncwarp();
}

// Pops up to 32 entries; returns whether this lane got one.
__device__ __forceinline__ bool wq_pop(unsigned long long *q, int *count, unsigned long long &v) {
  int lane = threadIdx.x & 31;
  int n = *count;
  int take = n < 32 ? n : 32;
  bool got = lane < take;
  if (got) v = q[n - take + lane];
  __syncwarp();
  if (lane == 0) *count = n - take;
  __syncwarp();
  return got;
}

// k_pen_inside takes its chunks in runs: so many consecutive chunks (of one unit,
// mostly) per atomic, the unit of each following from the previous one. A unit is
// then shared by a few dozen warps rather than hundreds, so the running deepest
// depth its points are checked against is known early, and few points need their
// depth searched exactly (64 chunks measured best on large batches). A batch with
// fewer chunks than would give every warp RUNS_PER_WARP runs takes shorter ones:
// one pair's 12 500 chunks in runs of 64 kept 195 warps of 5920 busy (6.6 ms; in
// runs of one 0.6 ms).
constexpr uint32_t RUN_INSIDE = 64, RUNS_PER_WARP = 4;

struct ChunkRun {
  uint32_t next = 0, end = 0;       // chunks [next, end) still to do
  uint32_t unit = 0, unit_end = 0;  // the unit of `next` and the first chunk after it
  uint32_t taken = 0;               // runs taken (whether to stop is asked every 8)
};

__device__ __forceinline__ bool next_chunk(ChunkRun &r, const PenState &ps, unsigned *head,
                                           const StopCtl &stop_ctl, unsigned long long budget,
                                           unsigned long long start, uint32_t &chunk, uint32_t &u,
                                           uint32_t &st) {
  if (r.next >= r.end) {
    uint32_t c = 0xFFFFFFFFu;
    if ((threadIdx.x & 31) == 0) {
      bool stop = false;
      if ((r.taken++ & 7u) == 0u) {
        if (stop_asked(stop_ctl)) {
          st |= ST_ABORTED;
          stop = true;
        } else if (budget && global_ns() - start > budget) {
          st |= ST_TIMEOUT;
          stop = true;
        }
      }
      if (!stop) c = atomicAdd(head, ps.run);
    }
    c = __shfl_sync(0xffffffffu, c, 0);
    if (c >= ps.n_chunks) return false;
    r.next = c;
    r.end = min(c + ps.run, ps.n_chunks);
    r.unit = unit_of_chunk(ps, c);
    r.unit_end = __ldg(ps.chunk0 + r.unit + 1);
  }
  chunk = r.next++;
  while (chunk >= r.unit_end) {
    ++r.unit;
    r.unit_end = __ldg(ps.chunk0 + r.unit + 1);
  }
  u = r.unit;
  return true;
}

__device__ __forceinline__ F3 unit_point(const PenUnit &x, uint32_t i) {
  double4 q = ldg4(x.pts + i);
  double a, b, c;
  apply_pose(x.pose, q.x, q.y, q.z, a, b, c);
  return {float(a), float(b), float(c)};
}

// The +axis ray parity of every active lane's point (RayScene::crossings,
// spatial/bvh.rs:160-175, under crossings_axis's rule), the 32 lanes sharing
// the work: each lane's grid cell is a run of entries, the runs of the warp are
// laid end to end (a prefix sum of their lengths), and every round each lane
// tests the next entry of that flattened list for its owner (the last lane
// whose run starts at or before it). Rounds therefore keep every lane busy
// however unevenly the cells are filled, and the lanes of one owner read its
// run's rectangles as consecutive, coalesced loads. A crossing toggles the
// owner's bit in the warp's parity word; `axis` is the same for the warp.
__device__ __forceinline__ uint32_t warp_crossings(const MeshView *m, F3 p, int axis, bool active,
                                                   unsigned *par_word) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const unsigned long long tri = reinterpret_cast<unsigned long long>(active ? m->tri : nullptr);
  uint32_t b = 0, len = 0;
  unsigned long long rect = 0, slot = 0;
  if (active && m->nf) {
    const AxisGrid &g = m->grid[axis];
    float pc[3] = {p.x, p.y, p.z};
    float pu = pc[(axis + 1) % 3], pv = pc[(axis + 2) % 3];
    float fu = floorf((pu - g.lo_u) * g.inv_cell), fv = floorf((pv - g.lo_v) * g.inv_cell);
    if (fu >= 0.0f && fv >= 0.0f && fu < float(g.nu) && fv < float(g.nv)) {
      size_t cell = size_t(fu) * g.nv + size_t(fv);
      b = __ldg(g.start + cell);
      len = __ldg(g.start + cell + 1) - b;
      rect = reinterpret_cast<unsigned long long>(g.rect);
      slot = reinterpret_cast<unsigned long long>(g.slot);
    }
  }
  uint32_t incl = len;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t y = __shfl_up_sync(FULL, incl, o);
    if (lane >= o) incl += y;
  }
  const uint32_t off = incl - len, total = __shfl_sync(FULL, incl, 31);
  if (lane == 0) *par_word = 0u;
  __syncwarp();
  const F3 d = {axis == 0 ? 1.0f : 0.0f, axis == 1 ? 1.0f : 0.0f, axis == 2 ? 1.0f : 0.0f};
  for (uint32_t base = 0; base < total; base += 32) {
    const uint32_t w = base + lane;
    int j = 0;  // the last lane whose run starts at or before w (off[0] = 0 <= w)
#pragma unroll
    for (int step = 16; step; step >>= 1)
      if (__shfl_sync(FULL, off, j + step) <= w) j += step;
    const float qx = __shfl_sync(FULL, p.x, j), qy = __shfl_sync(FULL, p.y, j),
                qz = __shfl_sync(FULL, p.z, j);
    const uint32_t bj = __shfl_sync(FULL, b, j), oj = __shfl_sync(FULL, off, j);
    const float4 *rj = reinterpret_cast<const float4 *>(__shfl_sync(FULL, rect, j));
    const uint32_t *sj = reinterpret_cast<const uint32_t *>(__shfl_sync(FULL, slot, j));
    const float4 *tj = reinterpret_cast<const float4 *>(__shfl_sync(FULL, tri, j));
    if (w < total) {
      const size_t k = size_t(bj) + (w - oj);
      const float qc[3] = {qx, qy, qz};
      const float qu = qc[(axis + 1) % 3], qv = qc[(axis + 2) % 3];
      const float4 r = __ldg(rj + k);
      if (!(qu < r.x || qu > r.y || qv < r.z || qv > r.w)) {
        const float4 *t = tj + 3 * size_t(__ldg(sj + k));
        const float4 a = __ldg(t), b = __ldg(t + 1), c = __ldg(t + 2);
        if (moller_trumbore_edges({qx, qy, qz}, d, {a.x, a.y, a.z}, {b.x - a.x, b.y - a.y, b.z - a.z},
                                  {c.x - a.x, c.y - a.y, c.z - a.z}) >= 0.0f)
          atomicXor(par_word, 1u << j);
      }
    }
  }
  __syncwarp();
  const uint32_t bits = *par_word;
  __syncwarp();
  return (bits >> lane) & 1u;
}

// RayScene::inside (spatial/bvh.rs:146-157) for every lane's point at once, by
// warp_crossings: the majority of the three parities, the third ray cast only
// for the lanes whose first two disagree.
__device__ __forceinline__ bool warp_inside(const MeshView *m, F3 p, bool active,
                                            unsigned *par_word) {
  const uint32_t a = warp_crossings(m, p, 0, active, par_word);
  const uint32_t b = warp_crossings(m, p, 1, active, par_word);
  const bool third = active && a != b;
  uint32_t c = 0;
  if (__any_sync(0xffffffffu, third)) c = warp_crossings(m, p, 2, third, par_word);
  return active && (a == b ? a != 0u : c != 0u);
}

// Inside or not and, inside, the depth. A block takes INSIDE_BLOCK queries at a
// time: the parities by its warps, then the depths of those inside as walks.
// Bound by the latency of a block's three steps: 20,000 queries 178 -> 19 us (a
// thread per query scanning its own cells, then walking while the others of its
// warp, outside, waited).
constexpr int INSIDE_BLOCK = 128;
__global__ void __launch_bounds__(INSIDE_BLOCK) k_inside(const __grid_constant__ MeshView m,
                                                         const double *pts, uint32_t n,
                                                         const __grid_constant__ Pose16 pose,
                                                         sherd_inside_outcome *out, uint32_t *status) {
  __shared__ unsigned next, found, parity[INSIDE_BLOCK / 32];
  __shared__ unsigned char queue[INSIDE_BLOCK];
  __shared__ float4 at[INSIDE_BLOCK];
  __shared__ WalkSlots slots[INSIDE_BLOCK / 32];
  const int warp = threadIdx.x >> 5;
  uint32_t st = 0;
  for (size_t first = size_t(blockIdx.x) * INSIDE_BLOCK; first < n;
       first += size_t(gridDim.x) * INSIDE_BLOCK) {
    if (threadIdx.x == 0) next = found = 0;
    __syncthreads();
    const size_t i = first + threadIdx.x;
    F3 p = {0.0f, 0.0f, 0.0f};
    bool in_box = false;
    if (i < n) {
      double x, y, z;
      apply_pose(pose.m, pts[3 * i], pts[3 * i + 1], pts[3 * i + 2], x, y, z);
      p = {float(x), float(y), float(z)};
      in_box = !(p.x < m.lo[0] || p.x > m.hi[0] || p.y < m.lo[1] || p.y > m.hi[1] ||
                 p.z < m.lo[2] || p.z > m.hi[2]);
    }
    const bool inside = warp_inside(&m, p, in_box, parity + warp);
    if (inside) {
      at[threadIdx.x] = make_float4(p.x, p.y, p.z, 0.0f);
      queue[atomicAdd(&found, 1u)] = (unsigned char)threadIdx.x;
    } else if (i < n) {
      out[i] = {0.0f, 0u};
    }
    __syncthreads();
    face_walks(
        &next, found, slots[warp],
        [&](uint32_t k, FaceWalk &w) {
          const float4 q = at[queue[k]];
          return walk_start(w, &m, {q.x, q.y, q.z}, f_inf());
        },
        [&](uint32_t k, const FaceWalk &w) { out[first + queue[k]] = {w.best, 1u}; }, st);
    __syncthreads();
  }
  if (st) atomicOr(status, st);
}

__global__ void k_pen_init(PenState ps) {
  for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u < ps.n_units; u += gridDim.x * blockDim.x) {
    ps.deeper[u] = 0;
    ps.deep[u] = 0;
    ps.best[u] = f2key(3.4028234663852886e38f);
  }
}

// Box test, parity, depth: the first pass of one_penetration (verify.rs:541-568).
__global__ void __launch_bounds__(256, PEN_INSIDE_MINB) k_pen_inside(const PairView *pairs, const sherd_work_item *items,
                                                    const sherd_candidate *cands, const double *inv,
                                                    PenState ps, unsigned *head,
                                                    StopCtl stop_ctl,
                                                    unsigned long long budget, uint32_t *status) {
  __shared__ WarpQueue wqs[8];
  __shared__ unsigned parity[8];
  __shared__ WalkSlots walk_slots[8];
  WalkSlots &slots = walk_slots[threadIdx.x >> 5];
  WarpQueue &q = wqs[threadIdx.x >> 5];
  unsigned *par_word = parity + (threadIdx.x >> 5);
  int lane = threadIdx.x & 31;
  if (lane == 0) q.n_box = q.n_in = 0;
  __syncwarp();
  uint32_t st = 0;
  unsigned long long start = global_ns();
  // An inside point's depth D (its distance to the mesh) enters the unit's
  // statistics twice: whether D > pen, and the unit's deepest D. Both are
  // exact without the full nearest-face search of every point. With w the
  // largest f32 <= pen (so D > pen exactly when D > w): the bound grid or a
  // walk that stops at the first face within w decides "deeper"; then the
  // point can only raise the running maximum M if no face lies within M, and
  // only then is D itself searched (within w when not deeper, unbounded
  // otherwise; the same value mesh_distance gives). M only ever holds depths
  // of inside points, so the last point to raise it holds the true maximum.
  auto depth_stage = [&](bool drain) {
    while (q.n_in >= 32 || (drain && q.n_in > 0)) {
      unsigned long long e = 0;
      const bool got = wq_pop(q.in, &q.n_in, e);
      const uint32_t u = uint32_t(e >> 32);
      const MeshView *m = nullptr;
      F3 p = {0.0f, 0.0f, 0.0f};
      float w = 0.0f, top = 0.0f;
      if (got) {
        PenUnit x = pen_unit(pairs, items, cands, inv, u);
        m = x.mesh;
        p = unit_point(x, uint32_t(e));
        w = __double2float_rd(x.pen);
      }
      const bool deeper =
          warp_walks<true>(m, p, w, got && mesh_may_reach(*m, p, w), slots, st) == f_inf();
      bool raise = got, look = false;
      if (got) {
        if (deeper) atomicAdd(&ps.deeper[u], 1u);
        const unsigned key = *((volatile unsigned *)&ps.deep[u]);
        if (key != 0u) {
          top = key2f(key - 1u);
          if (!deeper && top >= w)
            raise = false;  // D <= w <= M
          else
            look = mesh_may_reach(*m, p, top);
        }
      }
      if (warp_walks<true>(m, p, top, look, slots, st) != f_inf()) raise = false;  // D <= M
      const float depth = warp_walks<false>(m, p, deeper ? f_inf() : w, raise, slots, st);
      if (raise) atomicMax(&ps.deep[u], f2key(depth) + 1u);
    }
  };
  auto parity_stage = [&](bool drain) {
    while (q.n_box >= 32 || (drain && q.n_box > 0)) {
      unsigned long long e = 0;
      bool got = wq_pop(q.box, &q.n_box, e);
      F3 p = {0.0f, 0.0f, 0.0f};
      const MeshView *m = nullptr;
      if (got) {
        uint32_t u = uint32_t(e >> 32), i = uint32_t(e);
        PenUnit x = pen_unit(pairs, items, cands, inv, u);
        p = unit_point(x, i);
        m = x.mesh;
      }
      bool inside = warp_inside(m, p, got, par_word);
      wq_push(q.in, &q.n_in, inside, e);
      depth_stage(false);
    }
  };
  ChunkRun run;
  uint32_t chunk, u;
  while (next_chunk(run, ps, head, stop_ctl, budget, start, chunk, u, st)) {
    PenUnit x = pen_unit(pairs, items, cands, inv, u);
    uint32_t i = (chunk - ps.chunk0[u]) * 32u + lane;
    bool in_box = false;
    if (x.avail && i < x.n) {
      F3 p = unit_point(x, i);
      const MeshView &m = *x.mesh;
      in_box = !(p.x < m.lo[0] || p.x > m.hi[0] || p.y < m.lo[1] || p.y > m.hi[1] ||
                 p.z < m.lo[2] || p.z > m.hi[2]);
    }
    wq_push(q.box, &q.n_box, in_box, (unsigned long long)u << 32 | i);
    parity_stage(false);
  }
  parity_stage(true);
  depth_stage(true);
  if (st) atomicOr(status, st);
}

// ---- the minimum distance of the nothing-inside units (verify.rs:569-579) ----
//
// A closest-face walk takes 20 nodes on average and thousands at worst, so a
// warp that walks 32 queries at once waits for the longest of them: 15 times the
// mean. Here every lane holds a walk of its own and takes one node a round; when
// enough lanes have finished theirs, the warp refills them from its queue. A
// walk's bound is the smallest distance its unit has so far, read again as it
// goes (the unit is only asked for its minimum), so an early answer ends the
// walks beside it. The result is the smallest of the points' distances whatever
// the order. For the same reason a walk can be split: with the queue empty, a lane
// without work takes over the oldest subtree another lane has stacked (the walks
// of a point thousands of nodes from its answer would otherwise end the kernel
// alone, 2 us a node).

// Lanes that may be idle before a warp refills them.
#ifndef MIN_REFILL
#define MIN_REFILL 4
#endif
// Rounds between two looks at what the other walks of the unit have found.
#ifndef MIN_LOOK
#define MIN_LOOK 8
#endif

struct MinWalk {
  const MeshView *m;
  unsigned *best;  // f2key of the unit's smallest distance so far
  F3 p;
  unsigned key;    // what it was when last looked at
  float bound2;    // the padded square of it that boxes are held against
  int node, sb, sp;  // the node to visit, the stack's entries [sb, sp)
  uint32_t visits;
};

__device__ __forceinline__ void min_bound(MinWalk &w, unsigned key) {
  w.key = key;
  const float b = key2f(key);
  const float s = b + 4e-6f * b + w.m->pad;
  w.bound2 = s * s;
}
__device__ __forceinline__ void min_look(MinWalk &w) {
  min_bound(w, *((volatile unsigned *)w.best));
}

// The faces of the leaves the warp's walks have come to, shared out over its
// lanes: leaf `count` faces at `first` of each lane (0: none), laid end to end.
// A lane's own loop over its faces has the others wait for up to twelve
// face tests, a load and a division each; 32 at a time they take about three
// rounds. Returns the smallest distance of the lane's faces to its point.
__device__ __forceinline__ float warp_leaves(const MeshView *m, F3 p, uint32_t first, uint32_t count,
                                             unsigned *slot) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  uint32_t incl = count;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(FULL, incl, o);
    if (lane >= o) incl += y;
  }
  const uint32_t off = incl - count, total = __shfl_sync(FULL, incl, 31);
  if (!total) return f_inf();
  slot[lane] = f2key(f_inf());
  __syncwarp();
  const unsigned long long tri = reinterpret_cast<unsigned long long>(count ? m->tri : nullptr);
  for (uint32_t base = 0; base < total; base += 32) {
    const uint32_t w = base + lane;
    int j = 0;  // the last lane whose faces start at or before w
#pragma unroll
    for (int step = 16; step; step >>= 1)
      if (__shfl_sync(FULL, off, j + step) <= w) j += step;
    const F3 q = {__shfl_sync(FULL, p.x, j), __shfl_sync(FULL, p.y, j), __shfl_sync(FULL, p.z, j)};
    const uint32_t fj = __shfl_sync(FULL, first, j), oj = __shfl_sync(FULL, off, j);
    const float4 *t = reinterpret_cast<const float4 *>(__shfl_sync(FULL, tri, j)) + 3 * size_t(fj + (w - oj));
    if (w < total) {
      const float4 a = __ldg(t), b = __ldg(t + 1), c = __ldg(t + 2);
      const float d = tri_distance(q, {a.x, a.y, a.z}, {b.x, b.y, b.z}, {c.x, c.y, c.z});
      if (d < f_inf()) atomicMin(&slot[j], f2key(d));
    }
  }
  __syncwarp();
  const float d = key2f(slot[lane]);
  __syncwarp();
  return d;
}

__device__ __forceinline__ void min_found(MinWalk &w, float d) {
  const unsigned key = f2key(d);
  if (d < f_inf() && key < w.key) {
    atomicMin(w.best, key);
    min_bound(w, key);
  }
}

// One node of every lane's walk (`active`: it has one); false where it has ended.
// mesh_walk with its state kept by the caller and the leaves shared out.
__device__ __forceinline__ bool min_step(MinWalk &w, bool active, int *stack_n, float *stack_k,
                                         unsigned *slot, uint32_t &st) {
  if (active && ++w.visits > 2u * w.m->nf + 64u) {
    st |= ST_STACK;
    active = false;
  }
  int next = -1;
  uint32_t first = 0, faces = 0;
  if (active) {
    const Child2 n = load_node(w.m->nodes, w.node);
    const float pc[3] = {w.p.x, w.p.y, w.p.z};
    const float k[2] = {box_dist2(n.lo0, n.hi0, pc), box_dist2(n.lo1, n.hi1, pc)};
    const bool in0 = k[0] <= w.bound2, in1 = k[1] <= w.bound2;
    // The leaves of a node are one run of slots (the left one's end where the
    // right one's begin).
    const bool leaf0 = in0 && n.cnt[0], leaf1 = in1 && n.cnt[1];
    first = leaf0 ? n.ref[0] : n.ref[1];
    faces = (leaf0 ? n.cnt[0] : 0) + (leaf1 ? n.cnt[1] : 0);
    const bool go0 = in0 && !n.cnt[0], go1 = in1 && !n.cnt[1];
    if (go0 && go1) {
      const bool second = k[1] < k[0];
      next = second ? n.ref[1] : n.ref[0];
      if (w.sp < STACK) {
        stack_n[w.sp] = second ? n.ref[0] : n.ref[1];
        stack_k[w.sp++] = second ? k[0] : k[1];
      } else {
        st |= ST_STACK;
      }
    } else if (go0 || go1) {
      next = go0 ? n.ref[0] : n.ref[1];
    }
  }
  if (__any_sync(0xffffffffu, faces != 0)) {
    const float d = warp_leaves(w.m, w.p, first, faces, slot);
    if (faces) min_found(w, d);
  }
  if (!active) return false;
  if ((w.visits & (MIN_LOOK - 1)) == 0) min_look(w);
  if (next < 0) {
    while (w.sp > w.sb) {
      --w.sp;
      if (stack_k[w.sp] <= w.bound2) {
        next = stack_n[w.sp];
        break;
      }
    }
  }
  w.node = next;
  return next >= 0;
}

// Starts the walk of point i of unit u; false when there is nothing to walk.
__device__ __forceinline__ bool min_start(MinWalk &w, const PairView *pairs,
                                          const sherd_work_item *items, const sherd_candidate *cands,
                                          const double *inv, const PenState &ps, uint32_t u,
                                          uint32_t i) {
  const PenUnit x = pen_unit(pairs, items, cands, inv, u);
  w.m = x.mesh;
  w.best = &ps.best[u];
  w.p = unit_point(x, i);
  w.node = w.sb = w.sp = 0;
  w.visits = 0;
  min_look(w);
  if (w.m->root_leaf) {
    for (uint32_t f = 0; f < w.m->root_leaf; ++f) {
      F3 a, b, c;
      uint32_t id;
      tri_at(*w.m, f, a, b, c, id);
      min_found(w, tri_distance(w.p, a, b, c));
    }
    return false;
  }
  return w.m->nf != 0;
}

// The walks of a warp: `refill(have)` tops the queue up when fewer than 32 of
// its entries are left (false once there is nothing more to queue).
// A walk ends after `limit` nodes, answered or not.
template <class Refill>
__device__ __forceinline__ void min_walks(const PairView *pairs, const sherd_work_item *items,
                                          const sherd_candidate *cands, const double *inv,
                                          const PenState &ps, WarpQueue &q, unsigned *slot,
                                          uint32_t limit, Refill &&refill, uint32_t &st) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  int stack_n[STACK];
  float stack_k[STACK];
  MinWalk w = {};
  bool active = false, more = true;
  for (;;) {
    const unsigned idle = __ballot_sync(FULL, !active);
    if (__popc(idle) >= MIN_REFILL) {
      while (more && q.n_box < 32) more = refill();
      const int have = q.n_box, rank = __popc(idle & ((1u << lane) - 1u));
      __syncwarp();
      if (!active && rank < have) {
        const unsigned long long e = q.box[have - 1 - rank];
        active = min_start(w, pairs, items, cands, inv, ps, uint32_t(e >> 32), uint32_t(e));
      }
      __syncwarp();
      if (lane == 0) q.n_box = have - min(have, __popc(idle));
      __syncwarp();
      if (have < __popc(idle)) {
        // The queue is empty: lanes without work take over stacked subtrees.
        const unsigned poor = __ballot_sync(FULL, !active),
                       rich = __ballot_sync(FULL, active && w.sp > w.sb);
        const unsigned below = (1u << lane) - 1u;
        const int pairs_n = min(__popc(poor), __popc(rich));
        const bool give = active && w.sp > w.sb && __popc(rich & below) < pairs_n;
        const bool get = !active && __popc(poor & below) < pairs_n;
        const int from = get ? int(__fns(rich, 0, __popc(poor & below) + 1)) : lane;
        int gn = 0;
        float gk = 0.0f;
        if (give) {
          gn = stack_n[w.sb];
          gk = stack_k[w.sb++];
        }
        const int node = __shfl_sync(FULL, gn, from);
        const float key_k = __shfl_sync(FULL, gk, from);
        const unsigned long long m = __shfl_sync(FULL, reinterpret_cast<unsigned long long>(w.m), from),
                                 best = __shfl_sync(FULL, reinterpret_cast<unsigned long long>(w.best), from);
        const F3 p = {__shfl_sync(FULL, w.p.x, from), __shfl_sync(FULL, w.p.y, from),
                      __shfl_sync(FULL, w.p.z, from)};
        const unsigned key = __shfl_sync(FULL, w.key, from), visits = __shfl_sync(FULL, w.visits, from);
        if (get) {
          w.m = reinterpret_cast<const MeshView *>(m);
          w.best = reinterpret_cast<unsigned *>(best);
          w.p = p;
          w.node = node;
          w.sb = w.sp = 0;
          w.visits = visits;
          min_bound(w, key);
          active = key_k <= w.bound2;
        }
      }
      if (!__any_sync(FULL, active) && q.n_box == 0 && !more) return;
    }
    active = min_step(w, active, stack_n, stack_k, slot, st) && w.visits < limit;
  }
}

// 32 points spread over each nothing-inside unit give it a first bound; with
// none yet, the bound is what the walks beside a walk have found. Any face's
// distance is a bound, so a walk stops after SEED_VISITS nodes: a pose so far off that
// f32 cannot tell the mesh's faces apart has its points visit all of them, one
// warp a unit (118 ms on a collection with such poses, 1.4 with the limit).
constexpr uint32_t SEED_VISITS = 512;
__global__ void __launch_bounds__(256) k_pen_seed(const PairView *pairs, const sherd_work_item *items,
                                                  const sherd_candidate *cands, const double *inv,
                                                  PenState ps, uint32_t *status) {
  __shared__ WarpQueue wqs[8];
  __shared__ unsigned slots[8][32];
  WarpQueue &q = wqs[threadIdx.x >> 5];
  const uint32_t lane = threadIdx.x & 31, warps = (gridDim.x * blockDim.x) >> 5;
  uint32_t st = 0, u = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (lane == 0) q.n_box = q.n_in = 0;
  __syncwarp();
  min_walks(
      pairs, items, cands, inv, ps, q, slots[threadIdx.x >> 5], SEED_VISITS,
      [&]() {
        if (u >= ps.n_units) return false;
        const PenUnit x = pen_unit(pairs, items, cands, inv, u);
        const bool want = x.avail && ps.deep[u] == 0 && lane < x.n;
        const uint32_t i = uint32_t((unsigned long long)lane * x.n / 32u);
        wq_push(q.box, &q.n_box, want, (unsigned long long)u << 32 | i);
        u += warps;
        return true;
      },
      st);
  if (st) atomicOr(status, st);
}

// Every point of the nothing-inside units; one farther from the mesh's box than
// the unit's bound, or out of reach by the bound grid, cannot lower it (the bound
// only shrinks, so it still cannot when its walk would start). The warps stride
// over the chunks, so that at any time they are all on a few units and each
// finds the bound the others have brought down: in runs of 8 or 16 chunks a warp,
// with many units under way at once and their bounds still wide, the pass took
// 4 to 5 times as long (177 and 230 ms against 44 on a two-wall collection).
__global__ void __launch_bounds__(256) k_pen_min(const PairView *pairs, const sherd_work_item *items,
                                                 const sherd_candidate *cands, const double *inv,
                                                 PenState ps, StopCtl stop_ctl,
                                                 unsigned long long budget, uint32_t *status) {
  __shared__ WarpQueue wqs[8];
  __shared__ unsigned slots[8][32];
  WarpQueue &q = wqs[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  if (lane == 0) q.n_box = q.n_in = 0;
  __syncwarp();
  uint32_t st = 0, taken = 0;
  const unsigned long long start = global_ns();
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  uint32_t chunk = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  min_walks(
      pairs, items, cands, inv, ps, q, slots[threadIdx.x >> 5], MISS,
      [&]() {
        if (chunk >= ps.n_chunks) return false;
        if ((taken++ & 127u) == 0u) {
          if (lane == 0) {
            if (stop_asked(stop_ctl))
              st |= ST_ABORTED;
            else if (budget && global_ns() - start > budget)
              st |= ST_TIMEOUT;
          }
          if (__shfl_sync(0xffffffffu, st & (ST_ABORTED | ST_TIMEOUT), 0)) return false;
        }
        const uint32_t u = unit_of_chunk(ps, chunk), i = (chunk - ps.chunk0[u]) * 32u + lane;
        chunk += warps;
        if (ps.deep[u] != 0) return true;
        const PenUnit x = pen_unit(pairs, items, cands, inv, u);
        bool want = false;
        F3 p = {0.0f, 0.0f, 0.0f};
        if (x.avail && i < x.n) {
          p = unit_point(x, i);
          const float pc[3] = {p.x, p.y, p.z};
          const float window = key2f(*((volatile unsigned *)&ps.best[u]));
          const float gap = sqrtf(box_dist2(x.mesh->lo, x.mesh->hi, pc));
          want = !(gap > window + 1e-5f * window + x.mesh->pad) && mesh_may_reach(*x.mesh, p, window);
        }
        // Points that a far pose has rounded to the same f32 place are one query (the
        // walks of such poses are the pass's longest: f32 hardly tells the mesh's
        // faces apart, and a walk visits them all). The order is spatial, so a point's
        // twin is the lane before, which is walked, is a twin itself or cannot lower
        // the bound. (Three collections of 8,448 items with such poses: 349, 150 and
        // 187 ms, with this 134, 72 and 17. Twins across chunks gained nothing more.)
        const float bx = __shfl_up_sync(0xffffffffu, p.x, 1), by = __shfl_up_sync(0xffffffffu, p.y, 1),
                    bz = __shfl_up_sync(0xffffffffu, p.z, 1);
        const bool twin = lane > 0 && bx == p.x && by == p.y && bz == p.z;
        wq_push(q.box, &q.n_box, want && !twin, (unsigned long long)u << 32 | i);
        return true;
      },
      st);
  if (st) atomicOr(status, st);
}

// penetration_scores (verify.rs:483-498) from the two units of each item, and
// the verdict (verify.rs:632-638).
__global__ void k_pen_finalize(const PairView *pairs, const sherd_work_item *items,
                               sherd_candidate *cands, PenState ps, sherd_params p, uint32_t n_items) {
  uint32_t it = blockIdx.x * blockDim.x + threadIdx.x;
  if (it >= n_items) return;
  const PairView &pr = pairs[items[it].pair];
  sherd_candidate &c = cands[it];
  if (c.status || c.scores.partial) return;  // an early rejection's scores are final
  sherd_scores &s = c.scores;
  bool avail = pr.a.has_mesh && pr.b.has_mesh && pr.a.watertight && pr.b.watertight;
  if (avail) {
    double frac[2], mins[2];
    for (int side = 0; side < 2; ++side) {
      uint32_t u = 2 * it + side;
      uint32_t n = side ? pr.a.n_s : pr.b.n_s;
      if (n == 0) {
        frac[side] = 0.0;
        mins[side] = 0.0;
        continue;
      }
      frac[side] = double(ps.deeper[u]) / double(n);
      mins[side] = ps.deep[u] ? -double(key2f(ps.deep[u] - 1u)) : double(key2f(ps.best[u]));
    }
    // side 0 is pen_b / min_b, side 1 pen_a / min_a
    s.pen = fmax(frac[1], frac[0]);
    s.pen_depth = fmax(-mins[1], -mins[0]) / pr.sc.t;
  }
  const sherd_scales &sc = pr.sc;
  c.accepted = (s.tight >= p.min_tight && s.gap * sc.t <= sc.gap && s.pen <= p.max_pen &&
                s.seam >= p.min_seam && s.cont_n >= p.min_cont_n)
                   ? 1u
                   : 0u;
}

}  // namespace sherd
