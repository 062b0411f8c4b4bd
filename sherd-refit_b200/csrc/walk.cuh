// walk.cuh — closest-face queries by a warp whose lanes each hold a walk.
//
// mesh_distance run by 32 threads side by side takes as long as the longest of
// 32 walks, and at every leaf the others wait for one lane's faces: on the
// fracture samples of a collection three walks in four end at the root and the
// rest take 4 to 60 nodes. Here a lane whose walk has ended is given the next
// query (when WALK_REFILL of them are idle), and the faces of the leaves the
// lanes have come to are laid end to end and tested by all of them.
//
// The answers are mesh_distance's: every face within the padded bound is tested,
// whatever the order, and the smallest distance within the window is kept.
#pragma once

#include "traverse.cuh"

namespace sherd {

constexpr int WALK_REFILL = 4;  // idle lanes that make a warp refill

struct FaceWalk {
  const MeshView *m;
  F3 p;
  float window;    // distances above it do not count
  float best;      // the smallest so far within it, +inf before
  float bound2;    // the padded square of the bound boxes are held against
  int node, sp;
  uint32_t visits;
};

__device__ __forceinline__ void walk_bound(FaceWalk &w) {
  const float b = fminf(w.best, w.window);
  if (b == f_inf()) {
    w.bound2 = f_inf();
  } else {
    const float s = b + 4e-6f * b + w.m->pad;
    w.bound2 = s * s;
  }
}

// Starts the query of p against m within the window; false when it is answered
// already (w.best): nothing to find, or a mesh of one leaf.
template <bool ANY = false>
__device__ __forceinline__ bool walk_start(FaceWalk &w, const MeshView *m, F3 p, float window) {
  w.m = m;
  w.p = p;
  w.window = window;
  w.best = f_inf();
  w.node = w.sp = 0;
  w.visits = 0;
  if (m->nf == 0 || !(ANY ? window >= 0.0f : window > 0.0f)) return false;
  walk_bound(w);
  const float pc[3] = {p.x, p.y, p.z};
  // The vertex box, from which every face is at least as far as its own box.
  if (box_dist2(m->lo, m->hi, pc) > w.bound2) return false;
  if (!m->root_leaf) return true;
  for (uint32_t s = 0; s < m->root_leaf; ++s) {
    F3 a, b, c;
    uint32_t id;
    tri_at(*m, s, a, b, c, id);
    const float d = tri_distance(p, a, b, c);
    if (d <= window && d < w.best) w.best = d;
  }
  return false;
}

// A warp's shared words for its leaves.
struct WalkSlots {
  unsigned key[32];
};

// The faces [first, first + count) of each lane's leaf (count 0: none) tested
// against its point by all lanes, and its walk's best brought up to date.
__device__ __forceinline__ void walk_leaves(FaceWalk &w, uint32_t first, uint32_t count,
                                            WalkSlots &sh) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  uint32_t incl = count;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(FULL, incl, o);
    if (lane >= o) incl += y;
  }
  const uint32_t off = incl - count, total = __shfl_sync(FULL, incl, 31);
  sh.key[lane] = f2key(w.best);
  __syncwarp();
  const unsigned long long tri = reinterpret_cast<unsigned long long>(count ? w.m->tri : nullptr);
  for (uint32_t base = 0; base < total; base += 32) {
    const uint32_t e = base + lane;
    int j = 0;  // the last lane whose faces start at or before e
#pragma unroll
    for (int step = 16; step; step >>= 1)
      if (__shfl_sync(FULL, off, j + step) <= e) j += step;
    const F3 q = {__shfl_sync(FULL, w.p.x, j), __shfl_sync(FULL, w.p.y, j), __shfl_sync(FULL, w.p.z, j)};
    const float window = __shfl_sync(FULL, w.window, j);
    const uint32_t fj = __shfl_sync(FULL, first, j), oj = __shfl_sync(FULL, off, j);
    const float4 *t = reinterpret_cast<const float4 *>(__shfl_sync(FULL, tri, j)) + 3 * size_t(fj + (e - oj));
    if (e < total) {
      const float4 a = __ldg(t), b = __ldg(t + 1), c = __ldg(t + 2);
      const float d = tri_distance(q, {a.x, a.y, a.z}, {b.x, b.y, b.z}, {c.x, c.y, c.z});
      if (d <= window) atomicMin(&sh.key[j], f2key(d));
    }
  }
  __syncwarp();
  if (count && key2f(sh.key[lane]) < w.best) {
    w.best = key2f(sh.key[lane]);
    walk_bound(w);
  }
  __syncwarp();
}

// One node of every lane's walk (`active`: it has one); false where it has ended.
// ANY: a walk ends with the first face it finds.
template <bool ANY>
__device__ __forceinline__ bool walk_step(FaceWalk &w, bool active, int *stack_n, float *stack_k,
                                          WalkSlots &sh, uint32_t &st) {
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
    const bool go0 = in0 && !n.cnt[0], go1 = in1 && !n.cnt[1];
    // The leaves of a node are one run of slots (the left one's end where the
    // right one's begin).
    const bool leaf0 = in0 && n.cnt[0], leaf1 = in1 && n.cnt[1];
    first = leaf0 ? n.ref[0] : n.ref[1];
    faces = (leaf0 ? n.cnt[0] : 0) + (leaf1 ? n.cnt[1] : 0);
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
  if (__any_sync(0xffffffffu, faces != 0)) walk_leaves(w, first, faces, sh);
  if (!active || (ANY && w.best != f_inf())) return false;
  if (next < 0) {
    while (w.sp > 0) {
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

// The queries [0, n) of a block (or of one warp), handed out from *counter:
// `start(i, w)` starts query i and says whether it has to walk, `done(i, w)`
// takes its answer (w.best). Every lane of the warp calls it.
template <class Start, class Done>
__device__ __forceinline__ void face_walks(unsigned *counter, uint32_t n, WalkSlots &sh,
                                           Start &&start, Done &&done, uint32_t &st) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  int stack_n[STACK];
  float stack_k[STACK];
  FaceWalk w = {};
  uint32_t i = 0;
  bool active = false, more = true;
  for (;;) {
    unsigned idle = __ballot_sync(FULL, !active);
    while (more && __popc(idle) >= WALK_REFILL) {
      unsigned base = 0;
      if (lane == 0) base = atomicAdd(counter, unsigned(__popc(idle)));
      base = __shfl_sync(FULL, base, 0);
      more = base + __popc(idle) < n;
      if (!active) {
        i = base + __popc(idle & ((1u << lane) - 1u));
        if (i < n) {
          active = start(i, w);
          if (!active) done(i, w);
        }
      }
      idle = __ballot_sync(FULL, !active);
    }
    if (idle == FULL) return;
    const bool was = active;
    active = walk_step<false>(w, active, stack_n, stack_k, sh, st);
    if (was && !active) done(i, w);
  }
}

// One query a lane (`need`: it has one), the leaves' faces shared: the depth
// walks of k_pen_inside, 32 points of one or two units at a time, in which a
// lane's own loop over its leaf's faces had the others wait (the kernel 73 -> 63 ms
// on 28,224 items, 16 -> 13.5 on 1,792).
// Without refilling: the smallest distance
// from p to m within the window, or with ANY any such distance; +inf when there
// is none.
template <bool ANY>
__device__ __noinline__ float warp_walks(const MeshView *m, F3 p, float window, bool need,
                                         WalkSlots &sh, uint32_t &st) {
  int stack_n[STACK];
  float stack_k[STACK];
  FaceWalk w;
  w.best = f_inf();
  bool active = need && walk_start<ANY>(w, m, p, window);
  while (__any_sync(0xffffffffu, active))
    active = walk_step<ANY>(w, active, stack_n, stack_k, sh, st);
  return w.best;
}

}  // namespace sherd
