// segment.cuh — R 3.4's shell/fracture segmentation (fragment/segment.rs:189-631)
// on the device.
//
// The steps and the arrays between them:
//   voxel keys of the face centroids -> (radix sort) -> representatives, the
//   lowest face of every t/8 voxel, ascending -> each face's nearest
//   representative (point LBVH, lowest index on a tie) -> radius balls around
//   the representatives over the centroid LBVH (smoothed normals, majority
//   filter, shell reference normals) -> cone votes -> islands (lock-free
//   union-find over the face adjacency, component areas summed in face order)
//   -> boundary growth passes.
//
// Bit-exactness to a sequential restatement: a radius ball is collected in
// shared memory, sorted by face index and summed in that order, a thread a sum
// (PointTree::within returns its members ascending, kdtree.rs:219-245); a
// component's area is summed by one thread in face order (components.rs:
// 180-185). Everything else is a per-face decision or an exact reduction.
#pragma once

#include "kernels.cuh"

namespace sherd {

constexpr uint32_t VOXEL_LIMIT = 1u << 21;

enum BallMode { BALL_NORMALS = 0, BALL_MAJORITY = 1, BALL_SHELL_NORMALS = 2 };

// The exact per-axis minimum of the centroids, as order-preserving keys.
__global__ void k_min_bound(const double *c, uint32_t n, unsigned long long *mb) {
  unsigned long long m[3] = {~0ull, ~0ull, ~0ull};
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    for (int k = 0; k < 3; ++k) m[k] = min(m[k], d2key(c[3 * size_t(i) + k]));
  for (int k = 0; k < 3; ++k) {  // one atomic a warp: all of them meet on three words
    for (int o = 16; o; o >>= 1) m[k] = min(m[k], __shfl_xor_sync(0xffffffffu, m[k], o));
    if ((threadIdx.x & 31) == 0) atomicMin(mb + k, m[k]);
  }
}

// voxel_representatives (segment.rs:217-259): floor((c - (min - 1)) / spacing)
// per axis, packed 21 bits an axis so that the key order is the tuple order.
__global__ void k_voxel_keys(const double *c, uint32_t n, const unsigned long long *mb,
                             double spacing, unsigned long long *key, uint32_t *idx,
                             uint32_t *status) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  unsigned long long k = 0;
  for (int a = 0; a < 3; ++a) {
    double lo = key2d(mb[a]) - 1.0;
    double v = floor((c[3 * size_t(i) + a] - lo) / spacing);
    if (!(v >= 0.0 && v < double(VOXEL_LIMIT))) {
      atomicOr(status, ST_RANGE);
      v = 0.0;
    }
    k = (k << 21) | (unsigned long long)v;
  }
  key[i] = k;
  idx[i] = i;
}

__global__ void k_run_heads(const unsigned long long *key, uint32_t n, uint8_t *head) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) head[i] = i == 0 || key[i] != key[i - 1];
}

__global__ void k_gather_points(const double *src, const uint32_t *idx, uint32_t n, double *dst) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  for (int k = 0; k < 3; ++k) dst[3 * size_t(i) + k] = src[3 * size_t(idx[i]) + k];
}

// coarse_grid's near (segment.rs:189-200): the representative nearest each
// centroid, an index into the ascending representative list.
__global__ void k_nearest_rep(CloudView reps, const double *c, uint32_t n, uint32_t *near,
                              uint32_t *status) {
  uint32_t st = 0;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    double d2;
    int s = nearest_within_sq(reps, c[3 * size_t(i)], c[3 * size_t(i) + 1], c[3 * size_t(i) + 2],
                              d_inf(), d2, st);
    near[i] = s < 0 ? 0u : uint32_t(reps.pts[s].w);
  }
  if (st) atomicOr(status, st);
}

__device__ __forceinline__ float ball_bound(const CloudView &c, double radius) {
  return float(radius) * (1.0f + 1e-6f) + c.pad;
}

__device__ __forceinline__ bool in_ball(const double *q, double4 p, double r2) {
  double ex = q[0] - p.x, ey = q[1] - p.y, ez = q[2] - p.z;
  return (ex * ex + ey * ey) + ez * ez <= r2;
}

// A radius ball: every centroid with d2 <= r2 (inclusive, d2 = ((dx dx + dy dy) +
// dz dz)), sorted by face index and summed in that order.
//   BALL_NORMALS / BALL_SHELL_NORMALS: ball_normals (segment.rs:267-296),
//     m = sum A FN / max(sum A, 1e-12), m / max(|m|, 1e-12), and whether the
//     ball is non-empty; the shell form keeps only faces with frac == 0.
//   BALL_MAJORITY: majority_filter (segment.rs:402-427), wet > 0.5 total.
//
// A group of T threads takes a representative: it walks the tree up to T nodes at
// a time from a shared stack, appends the members, sorts them, and adds up their
// products, formed by all threads, one after the other by a thread per sum. One
// warp does a ball of up to BALL_CAP members; the representatives with larger
// ones are listed, and a block of 512 threads each does those. On a mesh of
// 66 144 faces (24 k representatives of 15 to 120 members, a few of thousands
// where its rings meet) the five passes of segmentation and breaklines took
// 8.8 ms with a counting pass and blocks whose first thread walked and summed
// alone, and take 0.7 ms this way.
constexpr uint32_t BALL_CAP = 512;     // members of a warp's ball
constexpr uint32_t BALL_STACK = 512;   // nodes waiting
constexpr int BALL_WARPS = 4;
constexpr int BALL_BLOCK = 512;
constexpr uint32_t BALL_BLOCK_STACK = 2048;

// Entries kept free for going down one node at a time, which adds one a level: a
// Karras tree's path takes each of the 63 code bits, and where codes are equal
// each of the 32 index bits, at most once.
constexpr int BALL_RESERVE = 63 + 32 + 1;

// Nodes to take at a time: each may put two back, and from one at a time on the
// stack grows by no more than the tree's depth.
__host__ __device__ __forceinline__ int ball_width(int sp, uint32_t stack, int most) {
  const int room = int(stack) - BALL_RESERVE - sp, width = room < most ? room : most;
  return width < 1 ? 1 : width < sp ? width : sp;
}

struct BallSums {
  int mode;
  const double *normals, *areas;
  const uint8_t *frac;
  double *out3;
  uint8_t *flag;
};

// Member j's terms of the four sums: the normal times the area and the area, or
// the area of a fracture face and the area.
__device__ __forceinline__ void ball_terms(const BallSums &w, uint32_t j, double (&t)[4]) {
  const double a = w.areas[j];
  if (w.mode == BALL_MAJORITY) {
    t[0] = w.frac[j] ? a : 0.0;
    t[1] = a;
    t[2] = t[3] = 0.0;
  } else {
    const double *nn = w.normals + 3 * size_t(j);
    t[0] = nn[0] * a;
    t[1] = nn[1] * a;
    t[2] = nn[2] * a;
    t[3] = a;
  }
}

__device__ __forceinline__ void ball_result(const BallSums &w, uint32_t r, uint32_t n,
                                            const double *sum) {
  if (w.mode == BALL_MAJORITY) {
    w.flag[r] = sum[0] > 0.5 * sum[1];
    return;
  }
  double m[3];
  const double den = fmax(sum[3], 1e-12);
  for (int c = 0; c < 3; ++c) m[c] = sum[c] / den;
  const double norm = fmax(sqrt((m[0] * m[0] + m[1] * m[1]) + m[2] * m[2]), 1e-12);
  for (int c = 0; c < 3; ++c) w.out3[3 * size_t(r) + c] = m[c] / norm;
  w.flag[r] = n > 0;
}

// Whether centroid slot s is a member, and its face.
__device__ __forceinline__ bool ball_member(const BallSums &w, const CloudView &all, const double *q,
                                            double r2, int s, uint32_t &j) {
  const double4 p = ldg4(all.pts + s);
  j = uint32_t(p.w);
  return in_ball(q, p, r2) && !(w.mode == BALL_SHELL_NORMALS && w.frac[j]);
}

// The children of a node whose boxes come within the bound: a leaf range
// (cnt > 0), a node (cnt = 0), or neither (cnt = -1).
__device__ __forceinline__ void ball_children(const CloudView &all, int node, const float *qf,
                                              float b2, int (&ref)[2], int (&cnt)[2]) {
  const Child2 nd = load_node(all.nodes, node);
  const bool in[2] = {box_dist2(nd.lo0, nd.hi0, qf) <= b2, box_dist2(nd.lo1, nd.hi1, qf) <= b2};
  for (int c = 0; c < 2; ++c) {
    ref[c] = nd.ref[c];
    cnt[c] = in[c] ? nd.cnt[c] : -1;
  }
}

__device__ __forceinline__ void ball_swap(uint32_t *idx, uint32_t i, uint32_t size, uint32_t stride) {
  const uint32_t lo = 2 * i - (i & (stride - 1)), hi = lo + stride;
  const uint32_t x = idx[lo], y = idx[hi];
  if ((x > y) == ((lo & size) == 0)) {
    idx[lo] = y;
    idx[hi] = x;
  }
}

struct BallWarp {
  double part[4][32];
  double sum[4];
  uint32_t idx[BALL_CAP];
  int stack[BALL_STACK];
};

__global__ void __launch_bounds__(BALL_WARPS * 32)
    k_ball_warp(CloudView all, const double *cent, const uint32_t *rep, uint32_t n_rep,
                double radius, BallSums w, uint32_t *large, uint32_t *n_large, uint32_t *status) {
  const unsigned FULL = 0xffffffffu;
  __shared__ BallWarp mem[BALL_WARPS];
  BallWarp &b = mem[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  const double r2 = radius * radius;
  const float bound = ball_bound(all, radius), b2 = bound * bound;
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  uint32_t st = 0;
  for (uint32_t r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < n_rep; r += warps) {
    const double *c0 = cent + 3 * size_t(rep[r]);
    const double q[3] = {c0[0], c0[1], c0[2]};
    const float qf[3] = {float(q[0]), float(q[1]), float(q[2])};
    uint32_t n = 0;  // members so far
    auto take = [&](bool has, int slot) {
      uint32_t j = 0;
      const bool in = has && ball_member(w, all, q, r2, slot, j);
      const unsigned got = __ballot_sync(FULL, in);
      const uint32_t at = n + __popc(got & below);
      if (in && at < BALL_CAP) b.idx[at] = j;
      n += __popc(got);
    };
    int sp = 0;
    if (all.root_leaf) {
      for (uint32_t s = 0; s < all.root_leaf; s += 32) take(s + lane < all.root_leaf, int(s + lane));
    } else {
      if (lane == 0) b.stack[0] = 0;
      sp = 1;
    }
    __syncwarp();
    while (sp > 0 && n <= BALL_CAP) {
      const int width = ball_width(sp, BALL_STACK, 32);
      int ref[2], cnt[2] = {-1, -1};
      sp -= width;
      const int node = lane < width ? b.stack[sp + lane] : 0;
      __syncwarp();
      if (lane < width) ball_children(all, node, qf, b2, ref, cnt);
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        for (int k = 0; __any_sync(FULL, cnt[c] > k); ++k) take(cnt[c] > k, ref[c] + k);
        const unsigned open = __ballot_sync(FULL, cnt[c] == 0);
        const int at = sp + __popc(open & below);
        if (cnt[c] == 0 && at < int(BALL_STACK)) b.stack[at] = ref[c];
        sp += __popc(open);
        if (sp > int(BALL_STACK)) {  // the same for the warp
          st |= ST_STACK;
          sp = int(BALL_STACK);
        }
      }
      __syncwarp();
    }
    if (n > BALL_CAP) {
      if (lane == 0) large[atomicAdd(n_large, 1u)] = r;
      __syncwarp();
      continue;
    }
    uint32_t pw = 1;
    while (pw < n) pw <<= 1;
    for (uint32_t i = n + lane; i < pw; i += 32) b.idx[i] = 0xFFFFFFFFu;
    __syncwarp();
    for (uint32_t size = 2; size <= pw; size <<= 1)
      for (uint32_t stride = size >> 1; stride > 0; stride >>= 1) {
        for (uint32_t i = lane; i < pw / 2; i += 32) ball_swap(b.idx, i, size, stride);
        __syncwarp();
      }
    double sum = 0.0;
    for (uint32_t base = 0; base < n; base += 32) {
      if (base + lane < n) {
        double t[4];
        ball_terms(w, b.idx[base + lane], t);
        for (int c = 0; c < 4; ++c) b.part[c][lane] = t[c];
      }
      __syncwarp();
      if (lane < 4) {
        const uint32_t m = min(32u, n - base);
        for (uint32_t t = 0; t < m; ++t) sum += b.part[lane][t];
      }
      __syncwarp();
    }
    if (lane < 4) b.sum[lane] = sum;
    __syncwarp();
    if (lane == 0) ball_result(w, r, n, b.sum);
    __syncwarp();
  }
  if (st && lane == 0) atomicOr(status, st);
}

// The listed representatives, a block each; `cap` (a power of two) member slots in
// dynamic shared memory. Reports the largest ball and the most leaf ranges any
// of them met, whatever the capacity (a ball above it is left undone).
__global__ void __launch_bounds__(BALL_BLOCK)
    k_ball_block(CloudView all, const double *cent, const uint32_t *rep, const uint32_t *list,
                 uint32_t n_list, double radius, BallSums w, uint32_t cap, uint32_t *max_members,
                 uint32_t *max_ranges, uint32_t *status) {
  extern __shared__ __align__(16) unsigned char ball_dynamic[];
  double *part = reinterpret_cast<double *>(ball_dynamic);               // 4 x BALL_BLOCK
  int *stack = reinterpret_cast<int *>(part + 4 * BALL_BLOCK);           // BALL_BLOCK_STACK
  uint32_t *idx = reinterpret_cast<uint32_t *>(stack + BALL_BLOCK_STACK);  // cap
  __shared__ uint32_t s_n, s_sp, s_ranges;
  __shared__ double s_sum[4];
  const uint32_t tid = threadIdx.x;
  uint32_t st = 0;
  const double r2 = radius * radius;
  const float bound = ball_bound(all, radius), b2 = bound * bound;
  for (uint32_t e = blockIdx.x; e < n_list; e += gridDim.x) {
    const uint32_t r = list[e];
    const double *c0 = cent + 3 * size_t(rep[r]);
    const double q[3] = {c0[0], c0[1], c0[2]};
    const float qf[3] = {float(q[0]), float(q[1]), float(q[2])};
    auto take = [&](int first, int count) {
      for (int s = first; s < first + count; ++s) {
        uint32_t j;
        if (!ball_member(w, all, q, r2, s, j)) continue;
        const uint32_t at = atomicAdd(&s_n, 1u);
        if (at < cap) idx[at] = j;
      }
    };
    if (tid == 0) {
      s_n = 0;
      s_ranges = 0;
      s_sp = all.root_leaf ? 0u : 1u;
      stack[0] = 0;
    }
    __syncthreads();
    if (all.root_leaf && tid == 0) {
      s_ranges = 1;
      take(0, int(all.root_leaf));
    }
    for (;;) {
      const int sp = int(min(s_sp, BALL_BLOCK_STACK));
      if (sp == 0) break;
      const int width = ball_width(sp, BALL_BLOCK_STACK, BALL_BLOCK);
      const bool mine = int(tid) < width;
      const int node = mine ? stack[sp - width + tid] : 0;
      __syncthreads();
      if (tid == 0) s_sp = uint32_t(sp - width);
      __syncthreads();
      if (mine) {
        int ref[2], cnt[2];
        ball_children(all, node, qf, b2, ref, cnt);
        for (int c = 0; c < 2; ++c) {
          if (cnt[c] > 0) {
            atomicAdd(&s_ranges, 1u);
            take(ref[c], cnt[c]);
          } else if (cnt[c] == 0) {
            const uint32_t at = atomicAdd(&s_sp, 1u);
            if (at < BALL_BLOCK_STACK)
              stack[at] = ref[c];
            else
              st |= ST_STACK;
          }
        }
      }
      __syncthreads();
    }
    __syncthreads();
    const uint32_t n = s_n;
    if (tid == 0) {
      atomicMax(max_members, n);
      atomicMax(max_ranges, s_ranges);
    }
    if (n <= cap) {  // the same for the block
      uint32_t pw = 1;
      while (pw < n) pw <<= 1;
      for (uint32_t i = n + tid; i < pw; i += BALL_BLOCK) idx[i] = 0xFFFFFFFFu;
      __syncthreads();
      for (uint32_t size = 2; size <= pw; size <<= 1)
        for (uint32_t stride = size >> 1; stride > 0; stride >>= 1) {
          for (uint32_t i = tid; i < pw / 2; i += BALL_BLOCK) ball_swap(idx, i, size, stride);
          __syncthreads();
        }
      double sum = 0.0;
      for (uint32_t base = 0; base < n; base += BALL_BLOCK) {
        if (base + tid < n) {
          double t[4];
          ball_terms(w, idx[base + tid], t);
          for (int c = 0; c < 4; ++c) part[c * BALL_BLOCK + tid] = t[c];
        }
        __syncthreads();
        if (tid < 4) {
          const uint32_t m = min(uint32_t(BALL_BLOCK), n - base);
          for (uint32_t t = 0; t < m; ++t) sum += part[tid * BALL_BLOCK + t];
        }
        __syncthreads();
      }
      if (tid < 4) s_sum[tid] = sum;
      __syncthreads();
      if (tid == 0) ball_result(w, r, n, s_sum);
    }
    __syncthreads();
  }
  if (st) atomicOr(status, st);
}

// A representative's answer to every face it represents.
__global__ void k_spread(const uint32_t *near, uint32_t n, const double *g3, const uint8_t *gflag,
                         double *face3, uint8_t *faceflag) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t r = near[i];
  if (face3)
    for (int k = 0; k < 3; ++k) face3[3 * size_t(i) + k] = g3[3 * size_t(r) + k];
  if (faceflag) faceflag[i] = gflag[r];
}

__global__ void k_votes_to_frac(const uint8_t *good, uint32_t n, uint32_t votes, uint8_t *frac) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) frac[i] = uint32_t(good[i]) < votes;
}

// face_adjacency (adjacency.rs:43-51, 138-160): the 3 nf edge keys in
// slot-major order, (lo << 32) | hi, with their positions.
__global__ void k_edge_keys(const uint32_t *f, uint32_t nf, unsigned long long *key,
                            uint32_t *pos) {
  uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nf) return;
  const int slot[3][2] = {{0, 1}, {1, 2}, {2, 0}};
  for (int s = 0; s < 3; ++s) {
    uint32_t a = f[3 * size_t(t) + slot[s][0]], b = f[3 * size_t(t) + slot[s][1]];
    uint32_t lo = min(a, b), hi = max(a, b);
    size_t at = size_t(s) * nf + t;
    key[at] = (unsigned long long)lo << 32 | hi;
    pos[at] = uint32_t(at);
  }
}

// Every two consecutive equal keys of the stably sorted list are one face
// pair; entry w is (MISS, MISS) when keys w and w + 1 differ.
__global__ void k_face_pairs(const unsigned long long *key, const uint32_t *pos, uint32_t m,
                             uint32_t nf, uint32_t *fa, uint32_t *fb) {
  uint32_t w = blockIdx.x * blockDim.x + threadIdx.x;
  if (w + 1 >= m) return;
  bool pair = key[w] == key[w + 1];
  fa[w] = pair ? pos[w] % nf : MISS;
  fb[w] = pair ? pos[w + 1] % nf : MISS;
}

__device__ __forceinline__ uint32_t uf_find(uint32_t *parent, uint32_t x) {
  volatile uint32_t *p = parent;
  for (;;) {
    uint32_t up = p[x];
    if (up == x) return x;
    uint32_t upup = p[up];
    if (upup != up) p[x] = upup;  // path halving; only ever points to an ancestor
    x = upup;
  }
}

__global__ void k_uf_init(uint32_t *parent, uint32_t n) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) parent[i] = i;
}

// mask_components (components.rs:120-159): union of every pair whose two
// faces have mask == target, the larger root hooked under the smaller by
// compare-and-swap on a root, so no union is lost and each component's root is
// its lowest face.
__global__ void k_uf_union(const uint32_t *fa, const uint32_t *fb, uint32_t m, const uint8_t *mask,
                           uint8_t target, uint32_t *parent, uint32_t *status) {
  for (uint32_t w = blockIdx.x * blockDim.x + threadIdx.x; w < m; w += gridDim.x * blockDim.x) {
    uint32_t a = fa[w], b = fb[w];
    if (a == MISS || mask[a] != target || mask[b] != target) continue;
    for (int tries = 0;; ++tries) {
      if (tries == (1 << 20)) {
        atomicOr(status, ST_STACK);
        break;
      }
      uint32_t ra = uf_find(parent, a), rb = uf_find(parent, b);
      if (ra == rb) break;
      if (ra < rb) {
        uint32_t t = ra;
        ra = rb;
        rb = t;
      }
      if (atomicCAS(parent + ra, ra, rb) == ra) break;
    }
  }
}

// Each face of the set gets its root as a sort key (MISS outside the set).
__global__ void k_uf_roots(uint32_t *parent, const uint8_t *mask, uint8_t target, uint32_t n,
                           uint32_t *root, uint32_t *face) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  root[i] = mask[i] == target ? uf_find(parent, i) : MISS;
  face[i] = i;
}

// One thread per component: its area, summed in face order (the roots were
// sorted stably, so each run lists its faces ascending), as far as the sum takes
// to reach min_area: areas are not negative, so it stays there, and whether it
// does is all that is asked (the shell of a 66 144-face mesh took 1.9 ms to its
// end). Eight faces' areas are read at a time; read one by one, the 150 faces to
// the threshold were a chain of loads, 0.2 ms.
__global__ void k_component_areas(const uint32_t *root, const uint32_t *face, uint32_t n,
                                  const double *areas, double min_area, double *size) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n || root[i] == MISS || (i > 0 && root[i - 1] == root[i])) return;
  double s = 0.0;
  const uint32_t mine = root[i];
  for (uint32_t j = i; j < n; j += 8) {
    double a[8];
    bool in[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const uint32_t at = min(j + k, n - 1);
      in[k] = j + k < n && root[at] == mine;
      a[k] = areas[face[at]];
    }
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (in[k]) s += a[k];
    if (!in[7] || s >= min_area) break;
  }
  size[mine] = s;
}

// drop_small_components (components.rs:186-190).
__global__ void k_drop_small(uint8_t *mask, uint8_t target, uint32_t n, uint32_t *parent,
                             const double *size, double min_area) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n || mask[i] != target) return;
  if (size[uf_find(parent, i)] < min_area) mask[i] = !target;
}

// refine_boundary (segment.rs:438-474), one pass in two launches: the
// fracture faces touching the shell at the start of the pass, then the flips.
__global__ void k_grow_candidates(const uint32_t *fa, const uint32_t *fb, uint32_t m,
                                  const uint8_t *frac, uint8_t *cand) {
  uint32_t w = blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= m || fa[w] == MISS) return;
  uint32_t a = fa[w], b = fb[w];
  if (frac[a] != frac[b]) cand[frac[a] ? a : b] = 1;
}

__global__ void k_grow_flip(uint8_t *cand, uint8_t *frac, uint32_t n, const double *normals,
                            const double *ref, const uint8_t *has_ref, double cos_grow,
                            uint32_t *flipped) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n || !cand[i]) return;
  cand[i] = 0;
  const double *nn = normals + 3 * size_t(i), *r = ref + 3 * size_t(i);
  if (has_ref[i] && (nn[0] * r[0] + nn[1] * r[1]) + nn[2] * r[2] > cos_grow) {
    frac[i] = 0;
    *flipped = 1;
  }
}

// The shell's normal noise for the automatic growth angle: the clamped dot of
// each shell face's normal with its smoothed normal (the angle is taken on
// the host, with the same acos as the reference's).
__global__ void k_shell_dots(const uint8_t *frac, uint32_t n, const double *normals,
                             const double *ns, double *dots) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double *a = normals + 3 * size_t(i), *b = ns + 3 * size_t(i);
  double c = (a[0] * b[0] + a[1] * b[1]) + a[2] * b[2];
  dots[i] = frac[i] ? 2.0 : fmin(1.0, fmax(-1.0, c));
}

}  // namespace sherd
