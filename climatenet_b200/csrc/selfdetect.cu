// selfdetect.cu — self-collision detection on the GPU (compiled with
// --fmad=false: every decision below must round like the reference).
//
//  1. LBVH over the mesh's triangles (Morton codes of the centroids, radix
//     sort, Karras hierarchy, bottom-up box refit).  Node boxes are exact
//     unions of the triangles' own bounding boxes, so a traversal with the
//     closed query box [x - 1.1 tol, x + 1.1 tol] finds exactly the candidate
//     set of getMeshPotentialTriangleCollision (geometry_util.cpp:284-327).
//  2. Per candidate: closest point with the reference's early exit and the
//     |c - x|^2 < tol^2 filter (checkMeshAllCollision geometry_util.cpp:229-262).
//     Hits that the pairing would skip without side effect (vertex in the
//     triangle, a zero barycentric coordinate; geometry_util.cpp:127-135) are
//     dropped here.
//  3. Hits are sorted by (vertex, triangle): the canonical candidate order.
//  4. Greedy node-node pairing in that order (geometry_util.cpp:94-219): a
//     vertex waits for the earlier ones its outcome depends on (k_pair).
//  5. Breadth-first Gauss-Seidel levels of the self-contact graph
//     (SFE:161-293) in one CTA, from the closed-form equivalent of the
//     reference's three BFS passes: edge level = min(dist(a), dist(b)) with
//     dist the BFS distance from the component's seeds (obstacle-contact
//     vertices; else its lowest-index degree-1 vertex; else its lowest-index
//     vertex).
#include <cuda_runtime.h>

#include <cub/cub.cuh>
#include <cuda/atomic>
#include <algorithm>
#include <cstring>
#include <stdexcept>
#include <string>
#include <vector>

#include "device.cuh"
#include "geometry.cuh"
#include "handle.hpp"
#include "kernels.hpp"
#include "lbvh.cuh"

namespace pdfb {
namespace {

constexpr int kRegCap = 16;   // pairing partners remembered per vertex
constexpr int kHitSlots = 32; // step path: candidate triangles kept per vertex
constexpr int kRebuildEvery = 8;  // step path: hierarchy rebuilt every k steps, refit in between

// Error bits of the handle's device error word set by the step path (read at
// the end of pdf_step): a device-side wait gave up, more partners or self
// contacts than the buffers hold, more hits than kHitSlots per vertex or than
// the hit buffer, BVH stack.
constexpr int kErrWait = 1, kErrSelfContacts = 4, kErrSelfHits = 8, kErrSelfStack = 16;
constexpr int kPairSpins = 1 << 22;  // polls before a wait of the pairing gives up: far above any legitimate wait

struct SelfWS {
  int max_nt = 0, max_nv = 0, hit_cap = 0;
  unsigned long long *mkey = nullptr, *mkey2 = nullptr;
  int *mval = nullptr, *mval2 = nullptr;             // sorted leaf -> triangle
  int *left = nullptr, *right = nullptr, *parent = nullptr, *leaf_parent = nullptr;
  int* visits = nullptr;
  unsigned long long* bbox = nullptr;                // 6 ordered-bit min/max
  int* n_hits = nullptr;  // two words: the count, and err
  unsigned long long *hkey = nullptr, *hkey2 = nullptr;
  int *hval = nullptr, *hval2 = nullptr;
  double* hbary = nullptr;
  int *reg = nullptr, *reg_n = nullptr, *touched = nullptr, *n_touched = nullptr, *err = nullptr;
  // pairing: per vertex the epoch it was last finished in, per hit the chosen
  // triangle corner (3: none), the paired hits, one ticket per mesh
  unsigned int* pair_done = nullptr;
  unsigned int pair_epoch = 0;
  int *paired = nullptr, *pair_hit = nullptr, *pair_base = nullptr, *pair_ticket = nullptr;
  int n_tickets = 0;
  // BFS scratch (slot space)
  int *deg = nullptr, *uf = nullptr, *dist = nullptr, *seed = nullptr, *cobst = nullptr, *cdeg1 = nullptr,
      *cmin = nullptr, *elev = nullptr, *lcount = nullptr;
  void* cub_tmp = nullptr;
  size_t cub_bytes = 0;
  // step path: one persistent hierarchy per mesh (regions at the mesh's
  // triangle offset, all meshes' triangles in total), per-vertex hit slots
  // and counts (shared by the meshes, consumed within the step)
  WNode* wnodes = nullptr;
  int *s_mval = nullptr, *s_left = nullptr, *s_right = nullptr, *s_parent = nullptr, *s_leaf_parent = nullptr,
      *s_visits = nullptr;
  int *hcount = nullptr, *hoff = nullptr, *slot_tri = nullptr, *n_total = nullptr;
  std::vector<int> since_build;  // per mesh: steps since its hierarchy was built (0 = never)
};

#define CKS(x)                                                                                    \
  do {                                                                                            \
    cudaError_t e_ = (x);                                                                         \
    if (e_ != cudaSuccess) throw std::runtime_error(std::string(#x) + ": " + cudaGetErrorString(e_)); \
  } while (0)

template <typename T>
T* salloc(size_t n) {
  T* p = nullptr;
  CKS(cudaMalloc((void**)&p, std::max<size_t>(1, n) * sizeof(T)));
  return p;
}

// Traversal: kWalkLanes lanes walk the hierarchy for one vertex.  Both children of a
// node are tested at their parent (one node record), the overlapping internal
// children go to the group's stack in shared memory, from which the lanes take
// up to kWalkLanes nodes at a time; overlapping leaf children are candidates.  The set
// found does not depend on the order.
//
// A walk is a chain of node loads (some 60 to 100 of them with one lane a
// vertex) and bound by their latency until the chip is full of walks; then the
// lanes that find no node cost more than the shorter chains save.  Measured (ncu):
// 14k vertices, kPairsOnly, 37 us (4 lanes 68, 16 lanes 44, one lane and an atomic
// a pair 197); 49k vertices, kStep, 99 us (4 lanes 116, 16 lanes 109, one lane
// 146); 131k and 250k vertices: one lane 217 and 256 us, two lanes 397 at 131k.
// So the step's meshes above kWalkVertices keep one lane (k_traverse_slots).  A
// stack that grows past kWalkWide is walked depth first, one node at a time, which
// bounds it by the tree's depth.
//
// Mode kStep: candidates that do not contain the vertex go to the vertex's
// kHitSlots slots, their number to hcount.  Mode kPairsOnly: every candidate
// (v, t) goes to hkey, a vertex's together and in triangle order unless it has
// more than some 50 (then kWalkUnsorted is set in *err).  Mode kHits: candidates
// that survive the closest-point filter and can pair go to hkey / hval / hbary.
constexpr int kTraverseThreads = 128, kWalkLanes = 8, kWalkWide = 32, kWalkDepth = 64, kWalkBuf = 64;
constexpr int kWalkVertices = 65536;
constexpr int kWalkOverflow = 2, kWalkUnsorted = 4;  // bits of *err (kPairsOnly, kHits)
enum WalkMode { kStep, kPairsOnly, kHits };
constexpr int kWalkStack = kWalkWide + 2 * kWalkLanes + kWalkDepth;
template <int kMode>
__global__ void __launch_bounds__(kTraverseThreads)
    k_traverse(int nv, int nt, const double* __restrict__ q, const int* __restrict__ tris, int v0, double tol,
               const WNode* __restrict__ nodes, int* __restrict__ hcount, int* __restrict__ slot_tri, int* n_hits,
               int cap, unsigned long long* hkey, int* hval, double* hbary, int* err) {
  constexpr int G = kWalkLanes, kGroups = kTraverseThreads / G, kStack = kWalkStack, kBuf = kWalkBuf;
  __shared__ int stacks[kGroups * kStack];
  __shared__ int bufs[kMode == kStep ? 1 : kGroups * kBuf];
  const int lane = threadIdx.x & 31, gl = lane % G, group = threadIdx.x / G;
  const unsigned int mask = ((1u << G) - 1u) << (lane - gl), below = mask & ((1u << lane) - 1u);
  const int v = blockIdx.x * kGroups + group;
  if (v >= nv) return;
  int* st = stacks + group * kStack;
  int* buf = bufs + (kMode == kStep ? 0 : group * kBuf);
  const double t = 1.1 * tol;
  const double3 x = ld3(q, v0 + v);
  const int gv = v0 + v;
  int* slots = slot_tri + (int64_t)v * kHitSlots;
  int count = 0, flushes = 0;
  auto own = [&](int tri) {
    return __ldg(tris + 3 * tri) == gv || __ldg(tris + 3 * tri + 1) == gv || __ldg(tris + 3 * tri + 2) == gv;
  };
  // the buffered candidates out (kPairsOnly, kHits)
  auto flush = [&]() {
    __syncwarp(mask);
    if (kMode == kPairsOnly && count > 0) {
      int base = 0;
      if (gl == 0) {
        base = atomicAdd(n_hits, count);
        if (++flushes > 1) atomicOr(err, kWalkUnsorted);
      }
      base = __shfl_sync(mask, base, lane - gl);
      for (int i = gl; i < count; i += G) {
        const int tri = buf[i];
        int rank = 0;
        for (int j = 0; j < count; ++j) rank += buf[j] < tri;
        if (base + rank < cap) hkey[base + rank] = ((unsigned long long)v << 32) | (unsigned int)tri;
      }
    } else if (kMode == kHits) {
      for (int i = gl; i < count; i += G) {
        const int tri = buf[i];
        double3 cp, w;
        closest_point(x, ld3(q, tris[3 * tri]), ld3(q, tris[3 * tri + 1]), ld3(q, tris[3 * tri + 2]), tol, &cp, &w);
        const double3 dd = cp - x;
        if (!(dot3(dd, dd) < tol * tol)) continue;
        if (w.x == 0 || w.y == 0 || w.z == 0) continue;
        const int k = atomicAdd(n_hits, 1);
        if (k < cap) {
          hkey[k] = ((unsigned long long)v << 32) | (unsigned int)tri;
          hval[k] = k;
          st3(hbary, k, w);
        }
      }
    }
    __syncwarp(mask);
    count = 0;
  };
  // a lane's candidate (hit false: none) into the group's list
  auto add = [&](bool hit, int tri) {
    if (kMode != kPairsOnly && hit) hit = !own(tri);
    const unsigned int m = __ballot_sync(mask, hit);
    const int at = count + __popc(m & below);
    if (hit) {
      if (kMode == kStep) {
        if (at < kHitSlots) slots[at] = tri;
      } else {
        buf[at] = tri;
      }
    }
    count += __popc(m);
  };
  if (nt == 1) {
    double3 tl, th;
    tri_box(ld3(q, tris[0]), ld3(q, tris[1]), ld3(q, tris[2]), &tl, &th);
    add(gl == 0 && box_overlap(x, t, tl, th), 0);
  } else {
    int sp = 1;
    if (gl == 0) st[0] = 0;
    __syncwarp(mask);
    while (sp > 0) {
      const int take = sp > kWalkWide ? 1 : min(sp, G);
      const int node = gl < take ? st[sp - 1 - gl] : -1;
      sp -= take;
      __syncwarp(mask);
      bool o0 = false, o1 = false;
      int c0 = 0, c1 = 0;
      if (node >= 0) {
        // the 112-byte record in seven 16-byte loads
        const double2* r = reinterpret_cast<const double2*>(nodes + node);
        const double2 b01 = __ldg(r), b23 = __ldg(r + 1), b45 = __ldg(r + 2), b67 = __ldg(r + 3),
                      b89 = __ldg(r + 4), b1011 = __ldg(r + 5);
        const int4 chv = __ldg(reinterpret_cast<const int4*>(r + 6));
        c0 = chv.x;
        c1 = chv.y;
        o0 = box_overlap(x, t, make_double3(b01.x, b01.y, b23.x), make_double3(b23.y, b45.x, b45.y));
        o1 = box_overlap(x, t, make_double3(b67.x, b67.y, b89.x), make_double3(b89.y, b1011.x, b1011.y));
      }
      const bool p0 = o0 && c0 >= 0, p1 = o1 && c1 >= 0;
      const unsigned int m0 = __ballot_sync(mask, p0), m1 = __ballot_sync(mask, p1);
      const int n0 = __popc(m0), n1 = __popc(m1);
      if (sp + n0 + n1 > kStack) {
        if (gl == 0) atomicOr(err, kMode == kStep ? kErrSelfStack : kWalkOverflow);
        break;
      }
      if (p0) st[sp + __popc(m0 & below)] = c0;
      if (p1) st[sp + n0 + __popc(m1 & below)] = c1;
      sp += n0 + n1;
      const bool any_leaf = __any_sync(mask, (o0 && c0 < 0) || (o1 && c1 < 0));
      if (any_leaf) {
        if (kMode != kStep && count + 2 * G > kBuf) flush();
        add(o0 && c0 < 0, ~c0);
        add(o1 && c1 < 0, ~c1);
      }
      __syncwarp(mask);
    }
  }
  if (kMode != kStep) {
    flush();
  } else if (gl == 0) {
    if (count > kHitSlots) {
      atomicOr(err, kErrSelfHits);
      count = kHitSlots;
    }
    hcount[v] = count;
  }
}

// Step-path traversal of large meshes, one lane a vertex: both children are tested at their parent (one node
// record load), overlapping leaf children are handled on the spot, the walk
// continues into the first overlapping internal child and keeps the other on
// a per-thread stack in shared memory (column-major: no bank conflicts).  A
// candidate is a triangle whose box overlaps the vertex's query box and that
// does not contain the vertex; candidates go to the vertex's slots,
// unordered, and the closest-point filter runs in k_filter_candidates.
constexpr int kTraverseStack = 48;
__global__ void __launch_bounds__(kTraverseThreads)
    k_traverse_slots(int nv, int nt, const double* __restrict__ q, const int* __restrict__ tris, int v0, double tol,
                     const WNode* __restrict__ nodes, int* __restrict__ hcount, int* __restrict__ slot_tri,
                     int* err) {
  __shared__ int stack[kTraverseStack * kTraverseThreads];
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= nv) return;
  const double t = 1.1 * tol;
  const double3 x = ld3(q, v0 + v);
  int count = 0;
  int* slots = slot_tri + (int64_t)v * kHitSlots;
  const int gv = v0 + v;
  auto candidate = [&](int tri) {
    if (__ldg(tris + 3 * tri) == gv || __ldg(tris + 3 * tri + 1) == gv || __ldg(tris + 3 * tri + 2) == gv) return;
    if (count < kHitSlots) slots[count] = tri;
    ++count;
  };
  if (nt == 1) {
    double3 tl, th;
    tri_box(ld3(q, tris[0]), ld3(q, tris[1]), ld3(q, tris[2]), &tl, &th);
    if (box_overlap(x, t, tl, th)) candidate(0);
  } else {
    int* st = stack + threadIdx.x;
    int sp = 0;
    int node = 0;
    while (node >= 0) {
      // the 112-byte record in seven 16-byte loads
      const double2* r = reinterpret_cast<const double2*>(nodes + node);
      const double2 b01 = __ldg(r), b23 = __ldg(r + 1), b45 = __ldg(r + 2), b67 = __ldg(r + 3),
                    b89 = __ldg(r + 4), b1011 = __ldg(r + 5);
      const int4 chv = __ldg(reinterpret_cast<const int4*>(r + 6));
      const int c0 = chv.x, c1 = chv.y;
      const bool o0 = box_overlap(x, t, make_double3(b01.x, b01.y, b23.x), make_double3(b23.y, b45.x, b45.y));
      const bool o1 = box_overlap(x, t, make_double3(b67.x, b67.y, b89.x), make_double3(b89.y, b1011.x, b1011.y));
      if (o0 && c0 < 0) candidate(~c0);
      if (o1 && c1 < 0) candidate(~c1);
      const bool d0 = o0 && c0 >= 0, d1 = o1 && c1 >= 0;
      if (d0 && d1) {
        if (sp >= kTraverseStack) {
          atomicOr(err, kErrSelfStack);
          break;
        }
        st[sp++ * kTraverseThreads] = c1;
        node = c0;
      } else if (d0) {
        node = c0;
      } else if (d1) {
        node = c1;
      } else {
        node = sp > 0 ? st[--sp * kTraverseThreads] : -1;
      }
    }
  }
  if (count > kHitSlots) {
    atomicOr(err, kErrSelfHits);
    count = kHitSlots;
  }
  hcount[v] = count;
}

template <int kMode, typename... Args>
void launch_traverse(cudaStream_t st, int nv, Args... args) {
  constexpr int per = kTraverseThreads / kWalkLanes;
  k_traverse<kMode><<<(nv + per - 1) / per, kTraverseThreads, 0, st>>>(nv, args...);
}

// The closest-point filter and the pairing precondition of mode 1 below on
// each vertex's candidates; survivors stay in the vertex's slots (in place,
// order kept) and hcount becomes their number.
__global__ void k_filter_candidates(int nv, const double* __restrict__ q, const int* __restrict__ tris, int v0,
                                    double tol, int* __restrict__ hcount, int* __restrict__ slot_tri) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= nv) return;
  const int cnt = hcount[v];
  if (cnt == 0) return;
  int* slots = slot_tri + (int64_t)v * kHitSlots;
  const double3 x = ld3(q, v0 + v);
  const double tol_sq = tol * tol;
  int kept = 0;
  for (int k = 0; k < cnt; ++k) {
    const int tri = slots[k];
    double3 cp, w;
    closest_point(x, ld3(q, tris[3 * tri]), ld3(q, tris[3 * tri + 1]), ld3(q, tris[3 * tri + 2]), tol, &cp, &w);
    const double3 dd = cp - x;
    if (!(dot3(dd, dd) < tol_sq)) continue;
    if (w.x == 0 || w.y == 0 || w.z == 0) continue;
    slots[kept++] = tri;
  }
  hcount[v] = kept;
}

// Hits in canonical (vertex, triangle) order without a global sort: vertex v
// owns [hoff[v], hoff[v] + hcount[v]); its triangles are sorted in place and
// the barycentric coordinates recomputed (same arithmetic as the filter).
__global__ void k_compact_hits(int nv, const double* __restrict__ q, const int* __restrict__ tris, int v0, double tol,
                               const int* __restrict__ hcount, const int* __restrict__ hoff,
                               const int* __restrict__ slot_tri, int cap, unsigned long long* hkey, int* hval,
                               double* hbary, int* n_total, int* err) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= nv) return;
  const int cnt = hcount[v], o = hoff[v];
  if (v == nv - 1) {
    const int total = o + cnt;
    if (total > cap) atomicOr(err, kErrSelfHits);
    *n_total = min(total, cap);
  }
  if (cnt == 0) return;
  int tl[kHitSlots];
  for (int k = 0; k < cnt; ++k) {
    const int tv = slot_tri[(int64_t)v * kHitSlots + k];
    int j = k;
    while (j > 0 && tl[j - 1] > tv) {
      tl[j] = tl[j - 1];
      --j;
    }
    tl[j] = tv;
  }
  const double3 x = ld3(q, v0 + v);
  for (int k = 0; k < cnt; ++k) {
    const int h = o + k;
    if (h >= cap) return;
    const int tri = tl[k];
    double3 cp, w;
    closest_point(x, ld3(q, tris[3 * tri]), ld3(q, tris[3 * tri + 1]), ld3(q, tris[3 * tri + 2]), tol, &cp, &w);
    hkey[h] = ((unsigned long long)v << 32) | (unsigned int)tri;
    hval[h] = h;
    st3(hbary, h, w);
  }
}

// Greedy node-node pairing (checkMeshSelfCollisions, geometry_util.cpp:94-219):
// the reference takes the hits in canonical (vertex, triangle) order, and a
// hit's outcome depends on the pairings made so far of its vertex and of the
// vertex's 1-ring.  k_pair runs the vertices that have hits in parallel, each
// vertex's own hits in order, and makes a vertex wait for every earlier vertex
// it can interact with, so that the outcome is the serial one.
//
// A vertex v reads whether pairs (x, t) exist for x in {v} + ring(v) and t in
// its triangles, and adds pairs (v, t).  An earlier vertex u < v matters to v
// only if
//   u is in ring(v) or in a triangle of v  (it may add a pair that v reads), or
//   u is in the ring of a vertex of a triangle of v  (v may add a pair that u
//   reads: v must not be there before u has looked).
// Pairs added by all others are invisible to v's tests, in whichever order
// they arrive.  Vertices are claimed in ascending order (32 at a time by a
// warp), so the lowest unfinished one is always running and never waits: the
// waits end.  Each is bounded all the same.
//
// Bound by the chain of waits (a contact patch is walked like a wavefront, one
// vertex deep along its rows); each link is a few L2 round trips, so
// everything that does not depend on another vertex (triangles, barycentric
// coordinates, the list of vertices to wait for) is loaded before the wait.
// Three 128 x 128 layers with 7.3k self contacts: 0.27 ms, against 27.5 ms for
// one thread that takes the hits one after the other; two 256 x 256 layers with
// 11.5k contacts: 0.26 ms (ncu, both sides).
//
// reg[16 v ..]: partners of v, -1 where none is written yet; reg_n[v]: their
// number.  A slot is claimed by an atomic and written after it; an unrelated
// vertex's slot that is claimed but still -1 matches nothing.
constexpr int kPairThreads = 128;
constexpr int kPairDeps = 48;  // vertices to wait for that a thread lists at a time

__device__ __forceinline__ void st_release(unsigned int* p, unsigned int v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Bit k set: vertex tv[k] is a partner of x.
__device__ __forceinline__ int partner_mask(const int* reg, int x, int n, int4 first, const int (&tv)[3]) {
  auto m1 = [&](int p) { return (p == tv[0] ? 1 : 0) | (p == tv[1] ? 2 : 0) | (p == tv[2] ? 4 : 0); };
  if (n <= 0) return 0;
  int m = m1(first.x) | m1(first.y) | m1(first.z) | m1(first.w);
  for (int r = 4; r < min(n, kRegCap); r += 4) {
    const int4 p = __ldcg(reinterpret_cast<const int4*>(reg + (int64_t)x * kRegCap + r));
    m |= m1(p.x) | m1(p.y) | m1(p.z) | m1(p.w);
  }
  return m;
}

__global__ void __launch_bounds__(kPairThreads)
    k_pair(int nv, const int* __restrict__ hcount, const int* __restrict__ hoff, int cap,
           const unsigned long long* __restrict__ hkey, const int* __restrict__ hval, const double* __restrict__ hbary,
           const int* __restrict__ tris, int v0, const int* __restrict__ ring_ptr, const int* __restrict__ ring_idx,
           int* reg, int* reg_n, int* touched, int* n_touched, unsigned int* done, unsigned int epoch, int* ticket,
           int* __restrict__ paired, int* err_word, int max_spins) {
  const int lane = threadIdx.x & 31;
  for (;;) {
    int base = 0;
    if (lane == 0) base = atomicAdd(ticket, 32);
    base = __shfl_sync(0xffffffffu, base, 0);
    if (base >= nv) return;
    const int v = base + lane;
    // (hits beyond the buffer were dropped: a vertex may be left with none)
    bool open = v < nv && hcount[v] > 0;
    const int h0 = open ? hoff[v] : 0;
    const int h1 = open ? min(h0 + hcount[v], cap) : 0;
    if (!__any_sync(0xffffffffu, open)) continue;
    const int gv = v0 + v;
    int rs = 0, re = 0;
    int deps[kPairDeps];
    int nd = 0;
    bool ok = true, full = false;
    auto is_done = [&](int u) { return *reinterpret_cast<const volatile unsigned int*>(done + u) == epoch; };
    // the unfinished earlier vertices that matter to this one (the first kPairDeps of them)
    auto list = [&]() {
      nd = 0;
      full = false;
      auto need = [&](int u) {
        if (u >= gv || full || hcount[u - v0] == 0 || is_done(u)) return;
        for (int k = 0; k < nd; ++k)
          if (deps[k] == u) return;
        if (nd < kPairDeps)
          deps[nd++] = u;
        else
          full = true;
      };
      for (int s = rs; s < re; ++s) need(ring_idx[s]);
      for (int h = h0; h < h1; ++h) {
        const int tri = (int)(hkey[h] & 0xffffffffu);
        for (int k = 0; k < 3; ++k) {
          const int t = tris[3 * tri + k];
          need(t);
          for (int s = ring_ptr[t]; s < ring_ptr[t + 1]; ++s) need(ring_idx[s]);
        }
      }
    };
    if (open) {
      rs = ring_ptr[gv];
      re = ring_ptr[gv + 1];
      list();
    }
    // the first hit's data
    int tri = 0;
    double wv[3] = {0., 0., 0.};
    int tv[3] = {0, 0, 0};
    auto load_hit = [&](int h) {
      tri = (int)(hkey[h] & 0xffffffffu);
      const double3 w = ld3(hbary, hval[h]);
      wv[0] = w.x;
      wv[1] = w.y;
      wv[2] = w.z;
      for (int k = 0; k < 3; ++k) tv[k] = tris[3 * tri + k];
    };
    if (h0 < h1) load_hit(h0);
    // one pass of the loop polls every lane's list and runs the lanes whose
    // list is empty: lanes of a warp may wait for one another
    int polls = 0;
    while (__any_sync(0xffffffffu, open)) {
      if (open && ok && nd > 0) {
        // the last four listed are read together
        unsigned int d[4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
          d[k] = nd > k ? *reinterpret_cast<const volatile unsigned int*>(done + deps[nd - 1 - k]) : epoch;
        int n = 0;
        while (n < 4 && d[n] == epoch) ++n;
        nd = max(0, nd - n);
        if (n == 0) {
          if (++polls > max_spins) {
            atomicOr(err_word, kErrWait);
            ok = false;
          } else if ((polls & 255) == 255 && (*reinterpret_cast<volatile int*>(err_word) & kErrWait)) {
            ok = false;
          }
        }
        if (nd == 0 && full) list();
      }
      if (open && (!ok || nd == 0)) {
        open = false;
        asm volatile("fence.acq_rel.gpu;" ::: "memory");  // what the vertices waited for wrote
        for (int h = h0; h < h1; ++h) {
          if (h > h0) load_hit(h);
          // partners of the vertex and of its ring, eight rows in flight
          const int4* rows = reinterpret_cast<const int4*>(reg);
          const int4 own = __ldcg(rows + (int64_t)gv * (kRegCap / 4));
          const int own_n = __ldcg(reg_n + gv);
          int cand = 7;
          for (int s0 = rs; s0 < re; s0 += 8) {
            int x[8], n[8];
            int4 f[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) x[k] = s0 + k < re ? ring_idx[s0 + k] : -1;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              n[k] = x[k] >= 0 ? __ldcg(reg_n + x[k]) : 0;
              f[k] = x[k] >= 0 ? __ldcg(rows + (int64_t)x[k] * (kRegCap / 4)) : make_int4(-1, -1, -1, -1);
            }
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              // the first triangle slot among the partners (isTriangleVertexIndexIn)
              const int m = n[k] > 0 ? partner_mask(reg, x[k], n[k], f[k], tv) : 0;
              cand &= ~(m & -m);
            }
          }
          int best = 3;
          if (ok && partner_mask(reg, gv, own_n, own, tv) == 0) {  // else already paired with a vertex of this triangle
            double bb = 0;
            for (int k = 0; k < 3; ++k)
              if ((cand >> k & 1) && wv[k] > bb) {
                best = k;
                bb = wv[k];
              }
          }
          if (best < 3) {
            const int other = tv[best];
            const int ra = atomicAdd(reg_n + other, 1), rb = atomicAdd(reg_n + gv, 1);
            if (ra >= kRegCap || rb >= kRegCap) {
              atomicOr(err_word, kErrSelfContacts);
              best = 3;
            }
            if (ra < kRegCap) __stcg(reg + (int64_t)other * kRegCap + ra, best < 3 ? gv : -1);
            if (rb < kRegCap) __stcg(reg + (int64_t)gv * kRegCap + rb, best < 3 ? other : -1);
            if (ra == 0) touched[atomicAdd(n_touched, 1)] = other;
            if (rb == 0) touched[atomicAdd(n_touched, 1)] = gv;
          }
          paired[h] = best;
        }
        st_release(done + gv, epoch);
      }
      __syncwarp();
    }
  }
}

// The paired hits in canonical order: pair_hit[k] is the hit of the mesh's
// k-th self contact, *pair_base the number of contacts of the meshes before it
// and *n_self their number with it.  One CTA, eight hits a thread and round.
constexpr int kPairScanThreads = 1024, kPairScanItems = 8;
__global__ void __launch_bounds__(kPairScanThreads)
    k_pair_compact(int n_hits, const int* n_hits_dev, const int* __restrict__ paired, int* __restrict__ pair_hit,
                   int* pair_base, DContacts c, int* err_word) {
  __shared__ int wsum[33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (n_hits_dev) n_hits = *n_hits_dev;
  const int base = *c.n_self;
  int total = 0;
  for (int t0 = 0; t0 < n_hits; t0 += kPairScanThreads * kPairScanItems) {
    const int i0 = t0 + threadIdx.x * kPairScanItems;
    int mine = 0;
#pragma unroll
    for (int k = 0; k < kPairScanItems; ++k)
      if (i0 + k < n_hits && paired[i0 + k] < 3) mine |= 1 << k;
    const int cnt = __popc(mine);
    int incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    if (warp == 0) {
      const int wv = wsum[lane];
      int w = wv;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += t;
      }
      wsum[lane] = w - wv;
      if (lane == 31) wsum[32] = w;
    }
    __syncthreads();
    int k0 = total + wsum[warp] + incl - cnt;
#pragma unroll
    for (int k = 0; k < kPairScanItems; ++k)
      if (mine >> k & 1) {
        if (base + k0 < c.self_cap) pair_hit[k0] = i0 + k;
        ++k0;
      }
    total += wsum[32];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    if (base + total > c.self_cap) atomicOr(err_word, kErrSelfContacts);
    *pair_base = base;
    *c.n_self = min(base + total, c.self_cap);
  }
}

__device__ void write_basis_s(double* B, double3 n) {
  double3 t = cross3(n, make_double3(1., 0., 0.));
  if (sqrt(dot3(t, t)) < 1.e-15) t = cross3(n, make_double3(0., 1., 0.));
  t = normalized3(t);
  const double3 bt = normalized3(cross3(n, t));
  B[0] = n.x; B[1] = n.y; B[2] = n.z;
  B[3] = t.x; B[4] = t.y; B[5] = t.z;
  B[6] = bt.x; B[7] = bt.y; B[8] = bt.z;
}

// The contact records of the mesh's paired hits (frames where the caller keeps them).
__global__ void k_pair_records(const int* __restrict__ pair_hit, const int* __restrict__ pair_base,
                               const int* __restrict__ paired, const unsigned long long* __restrict__ hkey,
                               const int* __restrict__ hval, const double* __restrict__ hbary,
                               const double* __restrict__ q, const int* __restrict__ tris, int v0, double mu,
                               DContacts c) {
  const int base = *pair_base, S = *c.n_self;
  for (int s = base + blockIdx.x * blockDim.x + threadIdx.x; s < S; s += gridDim.x * blockDim.x) {
    const int h = pair_hit[s - base];
    const int gv = v0 + (int)(hkey[h] >> 32);
    const int tri = (int)(hkey[h] & 0xffffffffu);
    const int ta = tris[3 * tri], tb = tris[3 * tri + 1], tc = tris[3 * tri + 2];
    const int best = paired[h];
    const double3 cpt = tri_point(ld3(q, ta), ld3(q, tb), ld3(q, tc), ld3(hbary, hval[h]));
    const double3 nrm = normalized3(ld3(q, gv) - cpt);
    c.s_vertex[s] = gv;
    c.s_partner[s] = best == 0 ? ta : (best == 1 ? tb : tc);
    c.s_face[3 * s] = ta;
    c.s_face[3 * s + 1] = tb;
    c.s_face[3 * s + 2] = tc;
    st3(c.s_normal, s, nrm);
    c.s_mu[s] = mu;
    if (c.s_basis) write_basis_s(c.s_basis + 9 * (int64_t)s, nrm);
  }
}

// Hits sorted by (vertex, triangle): each vertex's range.
__global__ void k_hit_ranges(int n, const unsigned long long* __restrict__ hkey, int* hcount, int* hoff) {
  const int h = blockIdx.x * blockDim.x + threadIdx.x;
  if (h >= n) return;
  const int v = (int)(hkey[h] >> 32);
  if (h == 0 || (int)(hkey[h - 1] >> 32) != v) hoff[v] = h;
  atomicAdd(hcount + v, 1);
}

// The registers of the last step's paired vertices emptied, the tickets rewound.
__global__ void k_reset_registered(int* reg, int* reg_n, int* touched, int* n_touched, int* tickets, int n_tickets) {
  const int n = *n_touched;
  const int t0 = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
  for (int i = t0; i < n; i += step) {
    const int v = touched[i];
    reg_n[v] = 0;
    int4* row = reinterpret_cast<int4*>(reg + (int64_t)v * kRegCap);
#pragma unroll
    for (int k = 0; k < kRegCap / 4; ++k) row[k] = make_int4(-1, -1, -1, -1);
  }
  for (int i = t0; i < n_tickets; i += step) tickets[i] = 0;
}

__device__ int uf_find(int* uf, int x) {
  while (true) {
    const int p = uf[x];
    if (p == x) return x;
    const int gp = uf[p];
    if (gp != p) atomicCAS(uf + x, p, gp);
    x = p;
  }
}

// Breadth-first levels (one CTA).  Slot space: every contact vertex has a slot.
constexpr int kLevelWarps = 32, kLevelTable = 128;
__global__ void k_levels(DContacts c, int* deg, int* uf, int* dist, int* seed, int* cobst, int* cdeg1, int* cmin,
                         int* elev, int* lcount, int cap_levels) {
  __shared__ int changed;
  __shared__ int maxlvl;
  const int S = *c.n_self, C = *c.n_contacts;
  const int V = min(*c.n_slots, c.slot_cap);
  const int tid = threadIdx.x, nth = blockDim.x;
  const int INF = 0x3fffffff;
  if (S == 0) {
    if (tid == 0) {
      *c.n_levels = 0;
      c.level_ptr[0] = 0;
    }
    return;
  }
  for (int s = tid; s < V; s += nth) {
    deg[s] = 0;
    uf[s] = s;
    dist[s] = INF;
    seed[s] = 0;
    cobst[s] = 0;
    cdeg1[s] = INF;
    cmin[s] = INF;
  }
  __syncthreads();
  for (int e = tid; e < S; e += nth) {
    atomicAdd(deg + c.s_slota[e], 1);
    atomicAdd(deg + c.s_slotb[e], 1);
  }
  for (int k = tid; k < C; k += nth) seed[c.c_slot[k]] = 1;
  __syncthreads();
  // connected components: hook the larger root under the smaller until stable
  do {
    __syncthreads();
    if (tid == 0) changed = 0;
    __syncthreads();
    for (int e = tid; e < S; e += nth) {
      const int ra = uf_find(uf, c.s_slota[e]), rb = uf_find(uf, c.s_slotb[e]);
      if (ra != rb) {
        atomicMin(uf + max(ra, rb), min(ra, rb));
        changed = 1;
      }
    }
    __syncthreads();
  } while (changed);
  for (int s = tid; s < V; s += nth) uf[s] = uf_find(uf, s);
  __syncthreads();
  for (int s = tid; s < V; s += nth) {
    const int r = uf[s];
    const int vx = c.slot_vertex[s];
    if (seed[s]) atomicOr(cobst + r, 1);
    if (deg[s] == 1) atomicMin(cdeg1 + r, vx);
    if (deg[s] >= 1) atomicMin(cmin + r, vx);
  }
  __syncthreads();
  for (int s = tid; s < V; s += nth) {
    const int r = uf[s];
    const int vx = c.slot_vertex[s];
    bool src;
    if (cobst[r])
      src = seed[s] != 0;
    else
      src = vx == (cdeg1[r] != INF ? cdeg1[r] : cmin[r]);
    dist[s] = src ? 0 : INF;
  }
  __syncthreads();
  int d = 0;
  do {
    __syncthreads();
    if (tid == 0) changed = 0;
    __syncthreads();
    for (int e = tid; e < S; e += nth) {
      const int a = c.s_slota[e], b = c.s_slotb[e];
      if (dist[a] == d && dist[b] == INF) {
        dist[b] = d + 1;
        changed = 1;
      }
      if (dist[b] == d && dist[a] == INF) {
        dist[a] = d + 1;
        changed = 1;
      }
    }
    __syncthreads();
    ++d;
  } while (changed);
  if (tid == 0) maxlvl = 0;
  __syncthreads();
  for (int e = tid; e < S; e += nth) elev[e] = min(dist[c.s_slota[e]], dist[c.s_slotb[e]]);
  // the reference opens one level per breadth-first frontier, including the
  // last frontier that finds no new edge: levels = max reached distance + 1
  for (int s = tid; s < V; s += nth)
    if (dist[s] < INF) atomicMax(&maxlvl, dist[s]);
  __syncthreads();
  const int nl = min(maxlvl + 1, cap_levels);
  // level_order: the contacts of each level in contact order.  A warp takes a
  // run of consecutive contacts; with the runs' counts per level added up, it
  // knows where its own go, and hands out places 32 contacts at a time (lanes
  // of one level in lane order).  One thread that places them one after the
  // other needs 60 ns each: 0.42 ms of this kernel's 0.51 ms at 7.3k contacts (now 0.09 ms).
  const int lane = tid & 31, warp = tid >> 5;
  auto place = [&](int e0, int e1, int* next) {
    for (int e = e0 + lane; e - lane < e1; e += 32) {
      const int l = e < e1 ? min(elev[e], nl - 1) : -1;
      const unsigned int same = __match_any_sync(0xffffffffu, l);
      int at = 0;
      const int leader = __ffs(same) - 1;
      if (lane == leader && l >= 0) {
        at = next[l];
        next[l] = at + __popc(same);
      }
      at = __shfl_sync(0xffffffffu, at, leader);
      if (l >= 0) c.level_order[at + __popc(same & ((1u << lane) - 1u))] = e;
      __syncwarp();
    }
  };
  if (nl <= kLevelTable) {
    __shared__ int table[kLevelWarps][kLevelTable];
    const int per = (S + kLevelWarps - 1) / kLevelWarps;
    const int e0 = min(S, warp * per), e1 = min(S, e0 + per);
    for (int k = tid; k < kLevelWarps * kLevelTable; k += nth) (&table[0][0])[k] = 0;
    __syncthreads();
    for (int e = e0 + lane; e < e1; e += 32) atomicAdd(&table[warp][min(elev[e], nl - 1)], 1);
    __syncthreads();
    if (warp == 0) {
      int acc = 0;  // contacts of the levels before the 32 of this round
      for (int l0 = 0; l0 < nl; l0 += 32) {
        const int l = l0 + lane;
        int n = 0;
        if (l < nl)
          for (int w = 0; w < kLevelWarps; ++w) {
            const int t = table[w][l];
            table[w][l] = n;
            n += t;
          }
        int incl = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int t = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += t;
        }
        const int start = acc + incl - n;
        if (l < nl) {
          c.level_ptr[l] = start;
          for (int w = 0; w < kLevelWarps; ++w) table[w][l] += start;
        }
        acc += __shfl_sync(0xffffffffu, incl, 31);
      }
      if (lane == 0) {
        c.level_ptr[nl] = acc;
        *c.n_levels = nl;
      }
    }
    __syncthreads();
    place(e0, e1, table[warp]);
    return;
  }
  // more levels than the table holds (long chains of contacts): one warp
  for (int l = tid; l < nl; l += nth) lcount[l] = 0;
  __syncthreads();
  for (int e = tid; e < S; e += nth) atomicAdd(lcount + min(elev[e], nl - 1), 1);
  __syncthreads();
  if (tid == 0) {
    int acc = 0;
    for (int l = 0; l < nl; ++l) {
      c.level_ptr[l] = acc;
      acc += lcount[l];
      lcount[l] = c.level_ptr[l];
    }
    c.level_ptr[nl] = acc;
    *c.n_levels = nl;
  }
  __syncthreads();
  if (warp == 0) place(0, S, lcount);
}

void ws_alloc(SelfWS& w, int nv, int nt, int hit_cap, int slot_cap) {
  w.max_nv = nv;
  w.max_nt = nt;
  w.hit_cap = hit_cap;
  w.mkey = salloc<unsigned long long>(nt);
  w.mkey2 = salloc<unsigned long long>(nt);
  w.mval = salloc<int>(nt);
  w.mval2 = salloc<int>(nt);
  w.left = salloc<int>(nt);
  w.right = salloc<int>(nt);
  w.parent = salloc<int>(nt);
  w.leaf_parent = salloc<int>(nt);
  w.visits = salloc<int>(nt);
  w.bbox = salloc<unsigned long long>(6);
  w.n_hits = salloc<int>(2);
  w.err = w.n_hits + 1;
  w.hkey = salloc<unsigned long long>(hit_cap);
  w.hkey2 = salloc<unsigned long long>(hit_cap);
  w.hval = salloc<int>(hit_cap);
  w.hval2 = salloc<int>(hit_cap);
  w.hbary = salloc<double>(3 * (size_t)hit_cap);
  w.hcount = salloc<int>(nv);
  w.hoff = salloc<int>(nv);
  w.slot_tri = salloc<int>((size_t)nv * kHitSlots);
  w.n_total = salloc<int>(1);
  size_t b1 = 0, b2 = 0, b3 = 0;
  CKS(cub::DeviceScan::ExclusiveSum(nullptr, b3, w.hcount, w.hoff, nv));
  CKS(cub::DeviceRadixSort::SortPairs(nullptr, b1, w.mkey, w.mkey2, w.mval, w.mval2, nt));
  CKS(cub::DeviceRadixSort::SortPairs(nullptr, b2, w.hkey, w.hkey2, w.hval, w.hval2, hit_cap));
  w.cub_bytes = std::max(std::max(b1, b2), b3);
  w.cub_tmp = salloc<char>(w.cub_bytes);
  (void)slot_cap;
}

void ws_free(SelfWS& w) {
  void* ptrs[] = {w.mkey, w.mkey2, w.mval, w.mval2, w.left, w.right, w.parent, w.leaf_parent,
                  w.visits, w.bbox, w.n_hits, w.hkey, w.hkey2, w.hval, w.hval2, w.hbary,
                  w.reg, w.reg_n, w.touched, w.n_touched, w.deg, w.uf, w.dist, w.seed, w.cobst, w.cdeg1,
                  w.cmin, w.elev, w.lcount, w.cub_tmp, w.wnodes, w.hcount, w.hoff, w.slot_tri, w.n_total,
                  w.s_mval, w.s_left, w.s_right, w.s_parent, w.s_leaf_parent, w.s_visits,
                  w.pair_done, w.paired, w.pair_hit, w.pair_base, w.pair_ticket};
  for (void* p : ptrs)
    if (p) cudaFree(p);
  w = SelfWS{};
}

// Bits that hold the values 0 .. n - 1.
int bits_for(int n) {
  int b = 1;
  while (b < 31 && (1 << b) < n) ++b;
  return b;
}

// Builds the LBVH over triangles [t0, t0+nt) (scene-global vertex indices
// with vertices [v0, v0+nv)) and traverses it from every vertex of the range.
// Returns the number of emitted records (may exceed the capacity); up to it they
// are in hkey2 (kHits: with hval2 their places in hbary) sorted by (vertex, triangle).
template <int kMode>
int detect_mesh(SelfWS& w, const double* q, const int* tris_global, int v0, int nv, int nt, double tol,
                cudaStream_t st) {
  const int tb = 256;
  size_t bytes = w.cub_bytes;
  if (nt > 1) {
    const unsigned long long init[6] = {~0ULL, ~0ULL, ~0ULL, 0ULL, 0ULL, 0ULL};
    CKS(cudaMemcpyAsync(w.bbox, init, sizeof(init), cudaMemcpyHostToDevice, st));
    k_bbox<<<std::min(1024, (nv + tb - 1) / tb), tb, 0, st>>>(nv, q + 3 * (size_t)v0, w.bbox);
    k_tri_keys<<<(nt + tb - 1) / tb, tb, 0, st>>>(nt, q, tris_global, v0, w.bbox, nullptr, nullptr, w.mkey, w.mval);
    // the keys come in triangle order and the sort is stable: the Morton bits
    // give the order of the whole key
    CKS(cub::DeviceRadixSort::SortPairs(w.cub_tmp, bytes, w.mkey, w.mkey2, w.mval, w.mval2, nt, 32, 62, st));
    k_build<<<(nt - 1 + tb - 1) / tb, tb, 0, st>>>(nt, w.mkey2, w.left, w.right, w.parent, w.leaf_parent);
    CKS(cudaMemsetAsync(w.visits, 0, sizeof(int) * nt, st));
    k_refit_wide<<<(nt + tb - 1) / tb, tb, 0, st>>>(nt, w.mval2, q, tris_global, w.left, w.parent, w.leaf_parent,
                                                    w.wnodes, w.visits);
  }
  // the count and the error bits lie side by side: one clear, one read
  CKS(cudaMemsetAsync(w.n_hits, 0, 2 * sizeof(int), st));
  launch_traverse<kMode>(st, nv, nt, q, tris_global, v0, tol, w.wnodes, (int*)nullptr, (int*)nullptr, w.n_hits,
                         w.hit_cap, w.hkey, w.hval, w.hbary, w.err);
  int res[2] = {0, 0};
  CKS(cudaMemcpyAsync(res, w.n_hits, sizeof(res), cudaMemcpyDeviceToHost, st));
  CKS(cudaStreamSynchronize(st));
  const int nh = res[0], err = res[1];
  if (err & kWalkOverflow)
    throw std::overflow_error("BVH traversal stack overflow (a vertex's walk needs more than the stack holds)");
  if (nh > 0 && nh <= w.hit_cap) {
    const int tbits = bits_for(nt), vbits = bits_for(nv);
    if (kMode == kHits) {
      CKS(cub::DeviceRadixSort::SortPairs(w.cub_tmp, bytes, w.hkey, w.hkey2, w.hval, w.hval2, nh, 0, tbits, st));
      std::swap(w.hkey, w.hkey2);
      std::swap(w.hval, w.hval2);
      CKS(cub::DeviceRadixSort::SortPairs(w.cub_tmp, bytes, w.hkey, w.hkey2, w.hval, w.hval2, nh, 32, 32 + vbits, st));
    } else {
      if (err & kWalkUnsorted) {
        CKS(cub::DeviceRadixSort::SortKeys(w.cub_tmp, bytes, w.hkey, w.hkey2, nh, 0, tbits, st));
        std::swap(w.hkey, w.hkey2);
      }
      CKS(cub::DeviceRadixSort::SortKeys(w.cub_tmp, bytes, w.hkey, w.hkey2, nh, 32, 32 + vbits, st));
    }
  }
  return nh;
}

// Step path of detect_mesh: same candidate semantics, no host round trip.
// The hits of mesh [v0, v0+nv) end in hkey2 / hval2 / hbary in canonical
// order with their count in *w.n_total; errors go to err_word.
void detect_mesh_step(SelfWS& w, const double* q, const int* tris_global, int v0, int nv, int nt, int t0,
                      bool rebuild, double tol, cudaStream_t st, int* err_word) {
  const int tb = 256;
  int* mval = w.s_mval + t0;
  int* left = w.s_left + t0;
  int* parent = w.s_parent + t0;
  int* leaf_parent = w.s_leaf_parent + t0;
  WNode* nodes = w.wnodes + t0;
  if (rebuild) {
    const unsigned long long init[6] = {~0ULL, ~0ULL, ~0ULL, 0ULL, 0ULL, 0ULL};
    CKS(cudaMemcpyAsync(w.bbox, init, sizeof(init), cudaMemcpyHostToDevice, st));
    k_bbox<<<std::min(1024, (nv + tb - 1) / tb), tb, 0, st>>>(nv, q + 3 * (size_t)v0, w.bbox);
    k_tri_keys<<<(nt + tb - 1) / tb, tb, 0, st>>>(nt, q, tris_global, v0, w.bbox, nullptr, nullptr, w.mkey, w.mval);
    // key = morton << 32 | triangle and the sort is stable on triangles in
    // ascending order: the 30 Morton bits give the full key order
    size_t bytes = w.cub_bytes;
    CKS(cub::DeviceRadixSort::SortPairs(w.cub_tmp, bytes, w.mkey, w.mkey2, w.mval, mval, nt, 32, 62, st));
    if (nt > 1)
      k_build<<<(nt - 1 + tb - 1) / tb, tb, 0, st>>>(nt, w.mkey2, left, w.s_right + t0, parent, leaf_parent);
  }
  if (nt > 1) {
    CKS(cudaMemsetAsync(w.s_visits + t0, 0, sizeof(int) * nt, st));
    k_refit_wide<<<(nt + tb - 1) / tb, tb, 0, st>>>(nt, mval, q, tris_global, left, parent, leaf_parent, nodes,
                                                    w.s_visits + t0);
  }
  if (nv <= kWalkVertices)
    launch_traverse<kStep>(st, nv, nt, q, tris_global, v0, tol, nodes, w.hcount, w.slot_tri, (int*)nullptr, 0,
                           (unsigned long long*)nullptr, (int*)nullptr, (double*)nullptr, err_word);
  else
    k_traverse_slots<<<(nv + kTraverseThreads - 1) / kTraverseThreads, kTraverseThreads, 0, st>>>(
        nv, nt, q, tris_global, v0, tol, nodes, w.hcount, w.slot_tri, err_word);
  k_filter_candidates<<<(nv + tb - 1) / tb, tb, 0, st>>>(nv, q, tris_global, v0, tol, w.hcount, w.slot_tri);
  size_t bytes = w.cub_bytes;
  CKS(cub::DeviceScan::ExclusiveSum(w.cub_tmp, bytes, w.hcount, w.hoff, nv, st));
  k_compact_hits<<<(nv + tb - 1) / tb, tb, 0, st>>>(nv, q, tris_global, v0, tol, w.hcount, w.hoff, w.slot_tri,
                                                    w.hit_cap, w.hkey2, w.hval2, w.hbary, w.n_total, err_word);
}

// Pairs the hits of mesh [v0, v0 + nv), in hkey2 / hval2 / hbary with their
// ranges in hcount / hoff, and appends its self contacts.  n_hits_dev: their
// number on the device (else n_hits).
void pair_mesh(SelfWS& w, const double* q, const int* tris, int v0, int nv, int mesh, const int* ring_ptr,
               const int* ring_idx, double mu, int n_hits, const int* n_hits_dev, const DContacts& c, int* err_word,
               cudaStream_t st) {
  const int warps = (nv + 31) / 32, wpc = kPairThreads / 32;
  // more CTAs than fit are no harm (tickets), 16 a SM keep every warp of a 300k-vertex mesh resident
  k_pair<<<std::min((warps + wpc - 1) / wpc, 16 * 148), kPairThreads, 0, st>>>(
      nv, w.hcount, w.hoff, w.hit_cap, w.hkey2, w.hval2, w.hbary, tris, v0, ring_ptr, ring_idx, w.reg, w.reg_n,
      w.touched, w.n_touched, w.pair_done, w.pair_epoch, w.pair_ticket + mesh, w.paired, err_word, kPairSpins);
  k_pair_compact<<<1, kPairScanThreads, 0, st>>>(n_hits, n_hits_dev, w.paired, w.pair_hit, w.pair_base, c, err_word);
  k_pair_records<<<148, 128, 0, st>>>(w.pair_hit, w.pair_base, w.paired, w.hkey2, w.hval2, w.hbary, q, tris, v0, mu, c);
}

// pairing / level scratch sized by the scene
void ws_alloc_pairing(SelfWS& w, int N, int slot_cap, int cap_levels, int n_meshes, int self_cap) {
  w.reg = salloc<int>((size_t)N * kRegCap);
  CKS(cudaMemset(w.reg, 0xff, sizeof(int) * kRegCap * (size_t)N));
  w.pair_done = salloc<unsigned int>(N);
  CKS(cudaMemset(w.pair_done, 0, sizeof(unsigned int) * N));
  w.paired = salloc<int>(w.hit_cap);
  w.pair_hit = salloc<int>(self_cap);
  w.pair_base = salloc<int>(1);
  w.n_tickets = n_meshes;
  w.pair_ticket = salloc<int>(n_meshes);
  CKS(cudaMemset(w.pair_ticket, 0, sizeof(int) * n_meshes));
  w.reg_n = salloc<int>(N);
  CKS(cudaMemset(w.reg_n, 0, sizeof(int) * N));
  w.touched = salloc<int>(N);
  w.n_touched = salloc<int>(1);
  CKS(cudaMemset(w.n_touched, 0, sizeof(int)));
  w.deg = salloc<int>(slot_cap);
  w.uf = salloc<int>(slot_cap);
  w.dist = salloc<int>(slot_cap);
  w.seed = salloc<int>(slot_cap);
  w.cobst = salloc<int>(slot_cap);
  w.cdeg1 = salloc<int>(slot_cap);
  w.cmin = salloc<int>(slot_cap);
  w.elev = salloc<int>(cap_levels);
  w.lcount = salloc<int>(cap_levels + 1);
}

}  // namespace

int self_detect_init(pdf_handle* h) {
  try {
    SelfWS* w = new SelfWS();
    int max_nt = 1, max_nv = 1;
    for (const auto& md : h->model.meshes) {
      max_nt = std::max(max_nt, md.n_triangles);
      max_nv = std::max(max_nv, md.n_vertices);
    }
    ws_alloc(*w, max_nv, max_nt, std::max(1024, 8 * max_nv), h->model.N);
    ws_alloc_pairing(*w, h->model.N, h->model.N, h->cap_self, (int)h->model.meshes.size(), h->cap_self);
    const size_t T = std::max<size_t>(1, h->model.tris.size() / 3);
    w->wnodes = salloc<WNode>(T);
    w->s_mval = salloc<int>(T);
    w->s_left = salloc<int>(T);
    w->s_right = salloc<int>(T);
    w->s_parent = salloc<int>(T);
    w->s_leaf_parent = salloc<int>(T);
    w->s_visits = salloc<int>(T);
    w->since_build.assign(h->model.meshes.size(), 0);
    h->d.self_ws = w;
  } catch (const std::exception& e) {
    h->err = e.what();
    return PDF_CUDA_ERROR;
  }
  return PDF_OK;
}

void self_detect_free(pdf_handle* h) {
  if (!h->d.self_ws) return;
  SelfWS* w = (SelfWS*)h->d.self_ws;
  ws_free(*w);
  delete w;
  h->d.self_ws = nullptr;
}

int self_detect_step(pdf_handle* h) {
  SelfWS& w = *(SelfWS*)h->d.self_ws;
  cudaStream_t st = h->stream;
  DContacts& c = h->d.c;
  // PhysicScene::getSelfCollisionsInfo(tol^2) -> checkMeshSelfCollisions(mesh, sqrt(tol^2))
  const double tol2 = h->prm.self_collision_tolerance * h->prm.self_collision_tolerance;
  const double tol = std::sqrt(tol2);
  CKS(cudaMemsetAsync(c.n_self, 0, sizeof(int), st));
  k_reset_registered<<<64, 256, 0, st>>>(w.reg, w.reg_n, w.touched, w.n_touched, w.pair_ticket, w.n_tickets);
  if (++w.pair_epoch == 0) {  // wrapped: no vertex may look finished
    CKS(cudaMemsetAsync(w.pair_done, 0, sizeof(unsigned int) * h->model.N, st));
    w.pair_epoch = 1;
  }
  CKS(cudaMemsetAsync(w.n_touched, 0, sizeof(int), st));
  // no host round trip: counts stay on the device, errors go to the handle's
  // error word (read at the end of pdf_step)
  for (size_t mi = 0; mi < h->model.meshes.size(); ++mi) {
    const auto& md = h->model.meshes[mi];
    const int* mtris = h->d.tris + 3 * (size_t)md.triangle_offset;
    // the hierarchy only steers the search: its boxes are refit exactly every
    // step, so rebuilding it every step or every k steps finds the same set
    int& since = w.since_build[mi];
    const bool rebuild = since == 0 || since >= kRebuildEvery;
    since = rebuild ? 1 : since + 1;
    detect_mesh_step(w, h->d.q, mtris, md.vertex_offset, md.n_vertices, md.n_triangles, md.triangle_offset, rebuild,
                     tol, st, h->d.sync.err);
    const double mu = h->model.friction[(size_t)md.material * h->model.n_materials + md.material];
    pair_mesh(w, h->d.q, mtris, md.vertex_offset, md.n_vertices, (int)mi, h->d.ring_ptr, h->d.ring_idx, mu, 0,
              w.n_total, c, h->d.sync.err, st);
  }
  return PDF_OK;
}

void self_levels_step(pdf_handle* h) {
  SelfWS& w = *(SelfWS*)h->d.self_ws;
  k_levels<<<1, 32 * kLevelWarps, 0, h->stream>>>(h->d.c, w.deg, w.uf, w.dist, w.seed, w.cobst, w.cdeg1, w.cmin, w.elev,
                                      w.lcount, h->cap_self);
}

int standalone_candidates(const double* pos, int nv, const int* tris, int nt, double tol, int* pairs, int cap, int* n,
                          int device, std::string& err) {
  if (!pos || nv <= 0 || nt <= 0 || !tris) {
    err = "invalid mesh";
    return PDF_INVALID_ARG;
  }
  CKS(cudaSetDevice(device));
  SelfWS w;
  double* dq = salloc<double>(3 * (size_t)nv);
  int* dt = salloc<int>(3 * (size_t)nt);
  int status = PDF_OK;
  try {
    CKS(cudaMemcpy(dq, pos, 3 * sizeof(double) * nv, cudaMemcpyHostToDevice));
    CKS(cudaMemcpy(dt, tris, 3 * sizeof(int) * nt, cudaMemcpyHostToDevice));
    int hit_cap = std::max(1024, cap);
    ws_alloc(w, nv, nt, hit_cap, nv);
    w.wnodes = salloc<WNode>(nt);
    int nh = detect_mesh<kPairsOnly>(w, dq, dt, 0, nv, nt, tol, 0);
    if (n) *n = nh;
    if (nh > hit_cap || nh > cap) {
      err = "candidate buffer too small";
      status = PDF_CAPACITY_EXCEEDED;
    } else if (pairs && nh > 0) {
      std::vector<unsigned long long> keys(nh);
      CKS(cudaMemcpy(keys.data(), w.hkey2, nh * sizeof(unsigned long long), cudaMemcpyDeviceToHost));
      for (int k = 0; k < nh; ++k) {
        pairs[2 * k] = (int)(keys[k] >> 32);
        pairs[2 * k + 1] = (int)(keys[k] & 0xffffffffu);
      }
    }
  } catch (...) {
    ws_free(w);
    cudaFree(dq);
    cudaFree(dt);
    throw;
  }
  ws_free(w);
  cudaFree(dq);
  cudaFree(dt);
  return status;
}

int standalone_self(const double* pos, int nv, const int* tris, int nt, double tol, pdf_contact* out, int cap, int* n,
                    int device, std::string& err) {
  if (!pos || nv <= 0 || nt <= 0 || !tris) {
    err = "invalid mesh";
    return PDF_INVALID_ARG;
  }
  // a one-mesh scene: rings from the triangles
  std::vector<std::vector<int>> nb(nv);
  for (int t = 0; t < nt; ++t)
    for (int k = 0; k < 3; ++k) {
      int a = tris[3 * t + k], b = tris[3 * t + (k + 1) % 3];
      if (a < 0 || a >= nv || b < 0 || b >= nv) {
        err = "triangle index out of range";
        return PDF_INVALID_ARG;
      }
      nb[a].push_back(b);
      nb[b].push_back(a);
    }
  std::vector<int> rp(nv + 1, 0), ri;
  for (int v = 0; v < nv; ++v) {
    std::sort(nb[v].begin(), nb[v].end());
    nb[v].erase(std::unique(nb[v].begin(), nb[v].end()), nb[v].end());
    rp[v + 1] = rp[v] + (int)nb[v].size();
    ri.insert(ri.end(), nb[v].begin(), nb[v].end());
  }
  CKS(cudaSetDevice(device));
  SelfWS w;
  std::vector<void*> mem;
  auto track = [&](void* p) {
    mem.push_back(p);
    return p;
  };
  int status = PDF_OK;
  try {
    double* dq = (double*)track(salloc<double>(3 * (size_t)nv));
    int* dt = (int*)track(salloc<int>(3 * (size_t)nt));
    int* drp = (int*)track(salloc<int>(nv + 1));
    int* dri = (int*)track(salloc<int>(ri.size()));
    CKS(cudaMemcpy(dq, pos, 3 * sizeof(double) * nv, cudaMemcpyHostToDevice));
    CKS(cudaMemcpy(dt, tris, 3 * sizeof(int) * nt, cudaMemcpyHostToDevice));
    CKS(cudaMemcpy(drp, rp.data(), sizeof(int) * (nv + 1), cudaMemcpyHostToDevice));
    if (!ri.empty()) CKS(cudaMemcpy(dri, ri.data(), sizeof(int) * ri.size(), cudaMemcpyHostToDevice));
    const int scap = std::max(1, 2 * nv);
    DContacts c{};
    c.cap = 1;
    c.n_self = (int*)track(salloc<int>(1));
    c.s_vertex = (int*)track(salloc<int>(scap));
    c.s_partner = (int*)track(salloc<int>(scap));
    c.s_face = (int*)track(salloc<int>(3 * (size_t)scap));
    c.s_normal = (double*)track(salloc<double>(3 * (size_t)scap));
    c.s_mu = (double*)track(salloc<double>(scap));
    c.self_cap = scap;
    CKS(cudaMemset(c.n_self, 0, sizeof(int)));
    ws_alloc(w, nv, nt, std::max(1024, 4 * nv), nv);
    w.wnodes = salloc<WNode>(nt);
    ws_alloc_pairing(w, nv, 1, 1, 1, scap);
    int nh = detect_mesh<kHits>(w, dq, dt, 0, nv, nt, tol, 0);
    if (nh > w.hit_cap) {
      err = "hit buffer too small";
      status = PDF_CAPACITY_EXCEEDED;
    } else {
      if (nh > 0) {
        CKS(cudaMemset(w.hcount, 0, sizeof(int) * nv));
        CKS(cudaMemset(w.hoff, 0, sizeof(int) * nv));
        k_hit_ranges<<<(nh + 255) / 256, 256>>>(nh, w.hkey2, w.hcount, w.hoff);
        w.pair_epoch = 1;
        pair_mesh(w, dq, dt, 0, nv, 0, drp, dri, 0., nh, nullptr, c, w.err, 0);
      }
      int S = 0, e2 = 0;
      CKS(cudaMemcpy(&S, c.n_self, sizeof(int), cudaMemcpyDeviceToHost));
      CKS(cudaMemcpy(&e2, w.err, sizeof(int), cudaMemcpyDeviceToHost));
      if (e2 & kErrWait) throw std::runtime_error("a wait of the pairing gave up");
      if (e2) {
        S = 0;
        err = "pairing capacity exceeded";
        status = PDF_CAPACITY_EXCEEDED;
      }
      if (n) *n = S;
      if (out && status == PDF_OK) {
        const int m = std::min(S, cap);
        std::vector<int> vx(m), pa(m), fa(3 * m);
        std::vector<double> nr(3 * m);
        if (m > 0) {
          CKS(cudaMemcpy(vx.data(), c.s_vertex, m * sizeof(int), cudaMemcpyDeviceToHost));
          CKS(cudaMemcpy(pa.data(), c.s_partner, m * sizeof(int), cudaMemcpyDeviceToHost));
          CKS(cudaMemcpy(fa.data(), c.s_face, 3 * m * sizeof(int), cudaMemcpyDeviceToHost));
          CKS(cudaMemcpy(nr.data(), c.s_normal, 3 * m * sizeof(double), cudaMemcpyDeviceToHost));
        }
        for (int k = 0; k < m; ++k) {
          pdf_contact& o = out[k];
          std::memset(&o, 0, sizeof(o));
          o.vertex = vx[k];
          o.partner = pa[k];
          for (int j = 0; j < 3; ++j) {
            o.face[j] = fa[3 * k + j];
            o.normal[j] = nr[3 * k + j];
          }
        }
        if (S > cap) {
          err = "output buffer too small";
          status = PDF_CAPACITY_EXCEEDED;
        }
      }
    }
  } catch (...) {
    ws_free(w);
    for (void* p : mem) cudaFree(p);
    throw;
  }
  ws_free(w);
  for (void* p : mem) cudaFree(p);
  return status;
}

// ---------------------------------------------------------------------------
// Allocation-free candidate detection (pdf_detect_candidates_noalloc).
//
// Some callers cannot allocate device memory at the point where they need
// the candidate pairs: code running inside another framework's memory pool
// that must not grow the process footprint, real-time loops with a fixed
// memory budget that forbid cudaMalloc/cudaFree after start-up, and hosts whose
// allocator is not the CUDA runtime's.  For them the whole workspace of the
// detection (LBVH boxes and nodes, Morton keys, candidate keys, radix-sort
// temporary storage) lives in one file-scope device array of fixed size.
// Every GPU that loads this library holds that array until the process exits.
constexpr int kNoAllocMaxTriangles = 65536;
constexpr int kNoAllocMaxPairs = 262144;
constexpr size_t kNoAllocSortBytes = size_t(8) << 20;
constexpr size_t align256(size_t x) { return (x + 255) & ~size_t(255); }
// byte layout of the array (each block 256-byte aligned)
constexpr size_t kNodeBytes = align256(sizeof(WNode) * kNoAllocMaxTriangles);  // wnodes
constexpr size_t kTriKeyBytes = align256(sizeof(unsigned long long) * kNoAllocMaxTriangles);  // mkey, mkey2
constexpr size_t kTriIntBytes = align256(sizeof(int) * kNoAllocMaxTriangles);  // mval, mval2, left, right, parent, leaf_parent, visits
constexpr size_t kPairKeyBytes = align256(sizeof(unsigned long long) * kNoAllocMaxPairs);  // hkey, hkey2
constexpr size_t kSmallBytes = 256 * 2;                                                     // bbox, n_hits and err
constexpr size_t kNoAllocScratchBytes = kNodeBytes + 2 * kTriKeyBytes + 7 * kTriIntBytes + 2 * kPairKeyBytes +
                                        kSmallBytes + kNoAllocSortBytes;

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

__global__ void k_keys_to_pairs(int n, const unsigned long long* __restrict__ keys, int* __restrict__ pairs) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  pairs[2 * k] = (int)(keys[k] >> 32);
  pairs[2 * k + 1] = (int)(keys[k] & 0xffffffffu);
}

int noalloc_candidates(const double* positions, int nv, const int* triangles, int nt, double tol, int* pairs,
                       int cap, int* n_out, cudaStream_t st, std::string& err) {
  if (!positions || !triangles || nv <= 0 || nt <= 0 || cap < 0 || !n_out) {
    err = "invalid arguments";
    return PDF_INVALID_ARG;
  }
  if (nt > kNoAllocMaxTriangles) {
    err = "pdf_detect_candidates_noalloc handles at most " + std::to_string(kNoAllocMaxTriangles) +
          " triangles (got " + std::to_string(nt) + ")";
    return PDF_CAPACITY_EXCEEDED;
  }
  // Set-up, repeated on every call with the caller's device current: the
  // array's device address on this device (the name is only a host-side
  // stand-in; cudaGetSymbolAddress allocates nothing) and the check that the
  // radix sort's workspace fits the reserved block.  Looking the address up on
  // every call keeps it valid after a cudaDeviceReset and needs no lock when
  // several host threads call.
  void* p = nullptr;
  cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
  if (e != cudaSuccess || !p) {
    err = std::string("cudaGetSymbolAddress(g_noalloc_scratch): ") + cudaGetErrorString(e);
    return PDF_CUDA_ERROR;
  }
  size_t b1 = 0, b2 = 0;
  CKS(cub::DeviceRadixSort::SortPairs(nullptr, b1, (unsigned long long*)nullptr, (unsigned long long*)nullptr,
                                      (int*)nullptr, (int*)nullptr, kNoAllocMaxTriangles));
  CKS(cub::DeviceRadixSort::SortPairs(nullptr, b2, (unsigned long long*)nullptr, (unsigned long long*)nullptr,
                                      (int*)nullptr, (int*)nullptr, kNoAllocMaxPairs));
  if (std::max(b1, b2) > kNoAllocSortBytes) {
    err = "radix-sort workspace larger than the reserved scratch";
    return PDF_CAPACITY_EXCEEDED;
  }
  unsigned char* base = (unsigned char*)p;
  size_t off = 0;
  auto take = [&](size_t bytes) {
    unsigned char* q = base + off;
    off += bytes;
    return q;
  };
  SelfWS w;
  w.max_nt = nt;
  w.max_nv = nv;
  w.hit_cap = kNoAllocMaxPairs;
  w.wnodes = (WNode*)take(kNodeBytes);
  w.mkey = (unsigned long long*)take(kTriKeyBytes);
  w.mkey2 = (unsigned long long*)take(kTriKeyBytes);
  w.mval = (int*)take(kTriIntBytes);
  w.mval2 = (int*)take(kTriIntBytes);
  w.left = (int*)take(kTriIntBytes);
  w.right = (int*)take(kTriIntBytes);
  w.parent = (int*)take(kTriIntBytes);
  w.leaf_parent = (int*)take(kTriIntBytes);
  w.visits = (int*)take(kTriIntBytes);
  w.hkey = (unsigned long long*)take(kPairKeyBytes);
  w.hkey2 = (unsigned long long*)take(kPairKeyBytes);
  w.bbox = (unsigned long long*)take(256);
  w.n_hits = (int*)take(256);
  w.err = w.n_hits + 1;
  w.cub_tmp = take(kNoAllocSortBytes);
  w.cub_bytes = kNoAllocSortBytes;
  const int nh = detect_mesh<kPairsOnly>(w, positions, triangles, 0, nv, nt, tol, st);
  *n_out = nh;
  if (nh > kNoAllocMaxPairs || nh > cap) {
    err = "candidate pairs exceed the output capacity or the scratch limit (" + std::to_string(kNoAllocMaxPairs) + ")";
    return PDF_CAPACITY_EXCEEDED;
  }
  if (nh > 0) k_keys_to_pairs<<<(nh + 255) / 256, 256, 0, st>>>(nh, w.hkey2, pairs);
  CKS(cudaGetLastError());
  CKS(cudaStreamSynchronize(st));
  return PDF_OK;
}

}  // namespace pdfb

extern "C" int pdf_detect_candidates_noalloc(const double* positions, int32_t n_vertices, const int32_t* triangles,
                                             int32_t n_triangles, double tolerance, int32_t* pairs, int32_t cap,
                                             int32_t* n, void* cuda_stream) {
  std::string err;
  int st;
  try {
    st = pdfb::noalloc_candidates(positions, n_vertices, triangles, n_triangles, tolerance, pairs, cap, n,
                                  (cudaStream_t)cuda_stream, err);
  } catch (const std::overflow_error& e) {
    err = e.what();
    st = PDF_CAPACITY_EXCEEDED;
  } catch (const std::exception& e) {
    err = e.what();
    st = PDF_CUDA_ERROR;
  }
  if (st != PDF_OK) pdfb::set_global_error(err);
  return st;
}
