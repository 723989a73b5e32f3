// lgpu_traverse.cuh — the instance-level traversals used by the wavefront
// kernels, over one stack for instance-BVH and mesh-BVH nodes.
//
// trace_tlas runs one ray to its end; an entered mesh is delimited on the
// stack by a marker.  The persistent kernels run the same search as a state
// machine (TraceState) whose node, leaf and object steps the lanes of a warp
// take together.  Both find the closest hit that the nested traversal in
// lgpu_intersect.cuh finds, with its rule for ties between objects, but in
// other trees, with wider box tests (kTravSlack) and in an order that ignores
// the three low bits of a distance: at an exactly equal distance another face
// of a mesh can be reported, and a triangle that a ray grazes can be found
// that the reference's boxes reject.  Rays whose answer depends on the
// reference's object order among several meshes get the reference's own loop
// (wf_trace_fallback).
//
// The stack keeps its first kSmemStack entries in shared memory, laid out
// entry-major (entry k of thread t at k*blockDim.x + t) so a warp's pushes
// and pops hit distinct banks; deeper entries go to a per-thread local
// array.
#pragma once

#include "lgpu_intersect.cuh"

namespace lgpu {

// The instance-BVH traversal tests boxes with a relative slack: a child is
// kept while its rounded entry distance is at most (1 + 2^-16) times its
// rounded exit (the closest hit so far included), and a popped entry is
// dropped only beyond (1 + 2^-16) times the closest hit.  A box's rounded
// entry can lie a few ulps beyond a triangle it contains (its vertex on the
// box's face), and without the slack such a triangle can be culled when a
// neighbouring one was hit first (one ray of 1.14 million in the benchmark
// scene traced with the surface-area-heuristic trees).  The slack only adds
// node tests; the reference-order traversal keeps the exact test.
constexpr float kTravSlack = 1.f + 1.f / 65536.f;

// 10 entries: the persistent kernels push at most two per node and seldom
// need more, and the shared memory this leaves is L1 for the nodes (8 and 16
// were 1 % slower on the benchmark frame)
constexpr int kSmemStack = 10;
constexpr int kLocalStack = kStackCap + kTlasStackCap + 4 - kSmemStack;
constexpr uint32_t kMarker = 0xFFFFFFFEu;

struct SplitStack {
  StackEntry* sm;  // this thread's column in shared memory
  uint32_t stride;
  StackEntry* lm;  // local overflow
  int sp;
  // kTravLocalStack once an entry beyond the shared part was used, and
  // kTravOverflow (merged into the thread's TravStats::flags when its work is
  // counted)
  uint32_t flags;
  // this thread's column of the world-ray save area (9 floats, stride 128;
  // persistent kernels only)
  float* ws = nullptr;
  __device__ __forceinline__ StackEntry& at(int k) {
    if (k < kSmemStack) return sm[k * stride];
    flags |= kTravLocalStack;
    return lm[k - kSmemStack];
  }
  // push and pop branch to a shared or a local access: through at()'s
  // reference the compiler emits generic loads and stores, which cost
  // registers (spills) and issue slots (traversal -6 % measured)
  __device__ __forceinline__ void push(StackEntry e) { put(sp++, e); }
  __device__ __forceinline__ void put(int k, StackEntry e) {
    if (k < kSmemStack) {
      sm[k * stride] = e;
    } else {
      flags |= kTravLocalStack;
      lm[k - kSmemStack] = e;
    }
  }
  __device__ __forceinline__ StackEntry pop() {
    --sp;
    if (sp < kSmemStack) return sm[sp * stride];
    return lm[sp - kSmemStack];
  }
};

constexpr int kSplitCap = kSmemStack + kLocalStack;
// Objects of the largest scenes in which wf_trace_fallback may keep the
// reference's object loop on the stack: its groups and a mesh's entries fit
// together.
constexpr uint32_t kMaxLoopObjects = 1024;
static_assert(kMaxLoopObjects / 32 + kStackCap <= kSplitCap, "object groups and a mesh's entries");
// push_children (lgpu_intersect.cuh) writing through a SplitStack.  With
// `sorted` false (any-hit queries, whose boolean answer does not depend on
// the visiting order) the hit children are pushed in child order.
template <bool ROWS>
__device__ __forceinline__ bool push_children_split(const WideNode& nd, const Ray& r, float t_max,
                                                    SplitStack& st, bool sorted) {
  float t[8];
  uint32_t ref[8];
  // ROWS: the row-wise test (the persistent kernels, which have the
  // registers for it); otherwise the per-child test (both give the same t)
  if (ROWS) {
    node_boxes_t(nd, r, t_max, t, kTravSlack);
#pragma unroll
    for (int c = 0; c < 8; c++) {
      ref[c] = nd.child[c];
      if (ref[c] == kEmptyChild) t[c] = 0.f;
    }
  } else {
    bool const nx = r.inv.x < 0.f, ny = r.inv.y < 0.f, nz = r.inv.z < 0.f;
#pragma unroll
    for (int c = 0; c < 8; c++) {
      ref[c] = nd.child[c];
      t[c] = (ref[c] != kEmptyChild) ? child_box_t(nd, c, r, nx, ny, nz, t_max, kTravSlack) : 0.f;
    }
  }
  int hits = 0;
#pragma unroll
  for (int c = 0; c < 8; c++) hits += (t[c] != 0.f) ? 1 : 0;
  if (st.sp + hits > kSplitCap) return false;
  if (!sorted) {
    if (st.sp + hits <= kSmemStack) {
      // as below: shared-memory stores only
      StackEntry* p = st.sm + st.sp * st.stride;
#pragma unroll
      for (int c = 0; c < 8; c++)
        if (t[c] != 0.f) {
          *p = StackEntry{ref[c], t[c]};
          p += st.stride;
        }
      st.sp += hits;
      return true;
    }
#pragma unroll
    for (int c = 0; c < 8; c++)
      if (t[c] != 0.f) st.push(StackEntry{ref[c], t[c]});
    return true;
  }
  // Far to near by a sorting network on 32-bit keys: a hit's distance bits
  // with their 3 low bits replaced by 7 - child (equal distances keep child
  // order; a miss's key, 7 - child alone, is below every hit's).  19
  // compare-exchanges of integer max/min cost fewer instructions than the
  // pairwise ranks of push_children (measured: closest-hit traversal
  // -1.4 %), and the hits are then pushed in sequence with their child
  // references read again from the node (an L1 hit) instead of kept in
  // registers.  The order can differ from the exact far-to-near order only
  // between children whose entry distances lie within 8 ulps, which changes
  // no closest distance (ties only; the reference-order traversal keeps
  // push_children's exact order).  The stored distance is the key's, at
  // most 7 ulps below the box's, so an entry is never culled early.
  uint32_t key[8];
#pragma unroll
  for (int c = 0; c < 8; c++) key[c] = (t[c] != 0.f ? (__float_as_uint(t[c]) & ~7u) : 0u) | uint32_t(7 - c);
  constexpr int kNet[19][2] = {{0, 1}, {2, 3}, {4, 5}, {6, 7}, {0, 2}, {1, 3}, {4, 6}, {5, 7}, {1, 2}, {5, 6},
                               {0, 4}, {3, 7}, {1, 5}, {2, 6}, {1, 4}, {3, 6}, {2, 4}, {3, 5}, {3, 4}};
#pragma unroll
  for (int k = 0; k < 19; k++) {
    uint32_t const a = key[kNet[k][0]], b = key[kNet[k][1]];
    key[kNet[k][0]] = max(a, b);
    key[kNet[k][1]] = min(a, b);
  }
  if (st.sp + hits <= kSmemStack) {
    // every hit lands in the shared part of the stack: no per-entry choice of memory
    StackEntry* const p = st.sm + st.sp * st.stride;
#pragma unroll
    for (int j = 0; j < 8; j++)
      if (j < hits) p[j * st.stride] = StackEntry{nd.child[7 - (key[j] & 7u)], __uint_as_float(key[j] & ~7u)};
    st.sp += hits;
    return true;
  }
#pragma unroll
  for (int j = 0; j < 8; j++)
    if (j < hits) st.at(st.sp + j) = StackEntry{nd.child[7 - (key[j] & 7u)], __uint_as_float(key[j] & ~7u)};
  st.sp += hits;
  return true;
}

// Instance-BVH traversal with the same semantics as scene_hit's instance
// path (ties to the higher object index, inside-bounds meshes tested in full
// and flagged in the hit).  Returns whether a hit was accepted.
template <bool ANY>
__device__ __forceinline__ bool trace_tlas(const DevScene& S, const Ray& w, HitRec& h, uint32_t skip,
                                           SplitStack& st, TravStats& ts) {
  h.inside = false;
  if (S.n_objects == 0) return false;
  float const t0 = segment_box_entry(S.tlas_bounds, w, h.z);
  if (t0 == kFltMax) return false;
  st.sp = 0;
  st.push(StackEntry{S.tlas_root, t0});
  bool in_mesh = false, lowered = false, cur_inside = false, hit_any = false;
  Ray l = w;
  f3 mr = f3{0.f, 0.f, 0.f};
  uint32_t cur = 0;
  float zs = 0.f, cur_exit = 0.f;
  while (st.sp > 0) {
    StackEntry const e = st.pop();
    if (e.ref == kMarker) {
      in_mesh = false;
      if (lowered && h.obj != cur) h.z = zs;
      lowered = false;
      continue;
    }
    if (e.t > h.z * kTravSlack) continue;
    if (!(e.ref & kLeafBit)) {
      ts.nodes++;
      if (!push_children_split<ANY>(S.nodes[e.ref], in_mesh ? l : w, h.z, st, !ANY)) {
        ts.flags |= 1u;
        break;
      }
      continue;
    }
    uint32_t const cnt = ((e.ref >> 28) & 7u) + 1u;
    uint32_t const slot = e.ref & kSlotMask;
    if (in_mesh) {
      for (uint32_t k = 0; k < cnt; k++) {
        const TriSlot& T = S.tris[slot + k];
        ts.tris++;
        float t, b0, b1, b2;
        if (tri_test(T, l, mr, h.z, t, b0, b1, b2)) {
          h.z = t;
          h.obj = cur;
          h.face = __float_as_uint(T.v0[3]);
          h.b0 = b0;
          h.b1 = b1;
          h.b2 = b2;
          h.pl = ray_at(l, t);
          h.inside = cur_inside;
          h.exit = cur_exit;
          hit_any = true;
          if (ANY) return true;
        }
      }
      continue;
    }
    // instance leaf: the first object now, the rest of the leaf afterwards
    uint32_t const i = S.tlas_objects[slot];
    if (cnt > 1) {
      if (st.sp + 1 > kSplitCap) {
        ts.flags |= 1u;
        break;
      }
      st.push(StackEntry{kLeafBit | ((cnt - 2u) << 28) | (slot + 1u), e.t});
    }
    if (i == skip) continue;
    ts.insts++;
    const DevObject& ob = S.objects[i];
    bool const low = !ANY && h.obj != UINT32_MAX && i < h.obj;
    float const z_saved = h.z;
    if (low) h.z = prev_float(z_saved);
    Ray const li = to_local(ob, w);
    if (ob.type != LGPU_OBJ_TRIMESH) {
      float t;
      f3 x;
      bool hit;
      if (ob.type == LGPU_OBJ_SPHERE) {
        hit = sphere_test(li, h.z, t);
        if (hit) x = ray_at(li, t);
      } else {
        hit = plane_test(li, h.z, t, x);
      }
      if (hit) {
        h.z = t;
        h.obj = i;
        h.face = UINT32_MAX;
        h.pl = x;
        h.inside = false;
        hit_any = true;
        if (ANY) return true;
      } else if (low) {
        h.z = z_saved;
      }
      continue;
    }
    const DevMesh& m = S.meshes[ob.mesh];
    bool inside;
    float ex;
    float r0 = aabb_scalar(m.bounds, li, h.z, inside, ex);
    if (r0 != kFltMax && !ANY && inside) r0 = kBias;
    if (r0 == kFltMax || r0 > h.z) {
      if (low) h.z = z_saved;
      continue;
    }
    if (st.sp + 2 > kSplitCap) {
      ts.flags |= 1u;
      break;
    }
    l = li;
    mr = cross3(l.p, l.u);
    cur = i;
    cur_inside = inside;
    cur_exit = ex;
    zs = z_saved;
    lowered = low;
    in_mesh = true;
    st.push(StackEntry{kMarker, 0.f});
    st.push(StackEntry{m.trav_root, r0});
  }
  return hit_any;
}

// ---- resumable traversal of the persistent kernels ---------------------------------

// Two single-precision values in one 64-bit register pair: Blackwell's
// packed add and multiply round each half as the scalar operation does, so
// the planes of two boxes cost two issue slots instead of four.
__device__ __forceinline__ uint64_t pack2(float x) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float min3(float a, float b, float c) {
  float r;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// Entry distances of all 8 child boxes (node_boxes_t's values, two children
// per instruction), handed one by one to f(child, entry, hit).  SLACK: with
// kTravSlack; without it child_box_t's test.
template <bool SLACK, class F>
__device__ __forceinline__ void node_children(const WideNode& nd, const Ray& r, float t_max, F f) {
  bool const nx = r.inv.x < 0.f, ny = r.inv.y < 0.f, nz = r.inv.z < 0.f;
  const ulonglong2* const nrx = reinterpret_cast<const ulonglong2*>(nx ? nd.hix : nd.lox);
  const ulonglong2* const frx = reinterpret_cast<const ulonglong2*>(nx ? nd.lox : nd.hix);
  const ulonglong2* const nry = reinterpret_cast<const ulonglong2*>(ny ? nd.hiy : nd.loy);
  const ulonglong2* const fry = reinterpret_cast<const ulonglong2*>(ny ? nd.loy : nd.hiy);
  const ulonglong2* const nrz = reinterpret_cast<const ulonglong2*>(nz ? nd.hiz : nd.loz);
  const ulonglong2* const frz = reinterpret_cast<const ulonglong2*>(nz ? nd.loz : nd.hiz);
  uint64_t const px = pack2(-r.p.x), py = pack2(-r.p.y), pz = pack2(-r.p.z);
  uint64_t const ix = pack2(r.inv.x), iy = pack2(r.inv.y), iz = pack2(r.inv.z);
  uint64_t const slack = pack2(kTravSlack);
#pragma unroll
  for (int h = 0; h < 2; h++) {
    ulonglong2 const a = nrx[h], b = frx[h], c = nry[h], d = fry[h], e = nrz[h], g = frz[h];
#pragma unroll
    for (int k = 0; k < 2; k++) {
      float x0, x1, y0, y1, z0, z1;
      unpack2(mul2(add2(k ? a.y : a.x, px), ix), x0, x1);
      unpack2(mul2(add2(k ? c.y : c.x, py), iy), y0, y1);
      unpack2(mul2(add2(k ? e.y : e.x, pz), iz), z0, z1);
      float const n0 = fmaxf(max3(x0, y0, z0), kBias), n1 = fmaxf(max3(x1, y1, z1), kBias);
      unpack2(mul2(add2(k ? b.y : b.x, px), ix), x0, x1);
      unpack2(mul2(add2(k ? d.y : d.x, py), iy), y0, y1);
      unpack2(mul2(add2(k ? g.y : g.x, pz), iz), z0, z1);
      float f0 = fminf(min3(x0, y0, z0), t_max), f1 = fminf(min3(x1, y1, z1), t_max);
      if (SLACK) {
        uint64_t ff;
        asm("mov.b64 %0, {%1, %2};" : "=l"(ff) : "f"(f0), "f"(f1));
        unpack2(mul2(ff, slack), f0, f1);
      }
      f(4 * h + 2 * k, n0, n0 <= f0);
      f(4 * h + 2 * k + 1, n1, n1 <= f1);
    }
    // keeps the second half's loads after the first half's tests (fewer
    // live registers)
    asm volatile("" ::: "memory");
  }
}

// A stack entry is a child reference with its entry distance, or, with
// kGroupBit set, a node some of whose hit children were not visited yet:
// their mask in the 8 low bits of t, whose other bits are a lower bound of
// their entry distances.  In the object loop a group entry in world space is
// 32 objects from an index on, with the mask of those still to be tested in t.
constexpr uint32_t kGroupBit = 0x40000000u;  // node indices stay below it (kMaxSlots)
constexpr uint32_t kNoRef = kEmptyChild;

// What a lane of a persistent kernel does next, as the addend that counts
// the lanes of each kind in one warp sum (a byte per kind).
constexpr uint32_t kLanePop = 0u;             // takes the next stack entry
constexpr uint32_t kLaneNode = 1u;            // tests the children of node `ref`
constexpr uint32_t kLaneTri = 1u << 8;        // tests the triangles of mesh leaf `ref`
constexpr uint32_t kLaneObj = 1u << 16;       // tests the object of instance leaf `ref`
constexpr uint32_t kLaneDone = 1u << 24;      // its ray is finished
constexpr uint32_t kLaneIdle = (1u << 24) | (1u << 31);  // has no ray (bits 30 and 31 of the sum are not read)

// The three queries of the persistent kernels: closest hits and shadow rays
// through the instance BVH and the traversal trees, and the reference's loop
// over the objects in index order through its own trees, with its box tests
// (no slack) and its order of a node's children.
constexpr int kQueryClosest = 0, kQueryAny = 1, kQueryLoop = 2;

// trace_tlas as a resumable state machine: trace_begin sets up a ray, then
// trace_pop and one of trace_node, trace_leaf and trace_object advance it.
// The persistent trace kernels call these in a loop shared by the whole warp
// and give a lane a new ray once its ray is finished.
//
// The state is what has to survive between steps and no more: the closest
// hit's face, barycentrics and point go to the hit record when the hit is
// accepted, the ray's moment is computed per leaf, and what a query skips
// follows from its phase.  The closest-hit kernel so fits 80 registers (6
// blocks per SM) without spills; with the whole hit in registers it spilled
// 150 B there and ran best at 96 (benchmark frame: closest-hit 145 ms, with
// the short state 127 ms).
struct TraceState {
  // the ray of the current level: the world ray, or the mesh-local ray while
  // a mesh is entered, when the world ray waits in shared memory
  // (SplitStack::ws)
  Ray w;
  float z;         // closest hit so far (the bound of an any-hit query)
  uint32_t obj;    // its object, UINT32_MAX: none
  float exit;      // where the ray leaves its bounds if they contain the ray origin, else -1
  float cur_exit;  // the same for the entered mesh
  uint32_t cur;    // object of the entered mesh
  uint32_t n_inside;  // meshes met whose bounds contain the ray origin
  uint32_t kind;   // what the lane does next (kLane*)
  uint32_t ref;    // the node or leaf it does that with
  int base;        // stack height at which the entered mesh is done; -1 in world space
  bool lowered;    // z was lowered for the entered mesh (it loses ties)
  // closest hits: 1, closest hit; 2, any hit among the objects below wobj; 3,
  // closest hit without object wobj (shadow rays: any hit without object wobj)
  int phase;
  uint32_t wobj;
};

// The next step: node or leaf `ref`, or the stack's top if it is kNoRef.
__device__ __forceinline__ void trace_next(TraceState& t, uint32_t ref) {
  t.ref = ref;
  t.kind = (ref & kLeafBit) ? (t.base >= 0 ? kLaneTri : kLaneObj) : kLaneNode;
  if (ref == kNoRef) t.kind = kLanePop;
}

__device__ __forceinline__ void trace_begin(const DevScene& S, TraceState& t, SplitStack& st) {
  t.obj = UINT32_MAX;
  t.exit = -1.f;
  t.lowered = false;
  t.base = -1;
  t.n_inside = 0;
  st.sp = 0;
  t.kind = kLaneDone;
  // without objects there is no instance BVH: every ray misses
  if (S.n_objects != 0 && segment_box_entry(S.tlas_bounds, t.w, t.z) != kFltMax) trace_next(t, S.tlas_root);
}

// Takes the next entry from the stack, leaving the entered mesh when its
// entries are used up.  An entry beyond the closest hit is dropped (the lane
// pops again).  For a node, `todo` is the mask of the children to test.
template <int Q>
__device__ __forceinline__ void trace_pop(const DevScene& S, TraceState& t, SplitStack& st, uint32_t& todo) {
  if (st.sp <= t.base) {
    // the mesh is done: back to the world ray, and to the distance before it
    // was lowered unless the mesh was hit
    t.base = -1;
    if (Q == kQueryClosest && t.lowered && t.obj != t.cur) t.z = next_float(t.z);
    t.lowered = false;
    t.w.p = f3{st.ws[0], st.ws[128], st.ws[2 * 128]};
    t.w.u = f3{st.ws[3 * 128], st.ws[4 * 128], st.ws[5 * 128]};
    t.w.inv = f3{st.ws[6 * 128], st.ws[7 * 128], st.ws[8 * 128]};
  }
  if (st.sp == 0) {
    t.kind = kLaneDone;
    return;
  }
  StackEntry const e = st.pop();
  uint32_t ref = e.ref;
  if (Q == kQueryAny) {
    if (!(ref & kLeafBit) && (ref & kGroupBit)) {
      uint32_t const m = __float_as_uint(e.t);
      uint32_t const c = 31u - __clz(m);
      uint32_t const rest = m ^ (1u << c);
      if (rest) st.push(StackEntry{ref, __uint_as_float(rest)});
      ref = S.nodes[ref ^ kGroupBit].child[c];
    }
  } else if (Q == kQueryLoop) {
    if (t.base < 0) {
      uint32_t const m = __float_as_uint(e.t), rest = m & (m - 1u);
      if (rest) st.push(StackEntry{ref, __uint_as_float(rest)});
      ref = kLeafBit | ((ref ^ kGroupBit) + uint32_t(__ffs(m) - 1));
    } else if (e.t > t.z) {
      return;
    }
  } else {
    uint32_t bound = __float_as_uint(e.t);
    if (!(ref & kLeafBit) && (ref & kGroupBit)) {
      // without the mask, which would lift the bound by up to 252 units in
      // the last place, over the slack's 128 to 256
      todo = bound & 0xFFu;
      bound &= ~0xFFu;
      ref ^= kGroupBit;
    }
    if (__uint_as_float(bound) > t.z * kTravSlack) return;
  }
  trace_next(t, ref);
}

// Tests the children of node t.ref that are in `todo`.
//
// Closest-hit rays visit a node's hit children from near to far without
// sorting them: the nearest is the next step's (no stack access), the second
// is pushed with its distance, and the others wait as a group entry.  Once
// that is popped and its bound is not beyond the closest hit, the node's
// remaining children are tested again, against the closest hit by then.  Few
// nodes have a third hit child that is still wanted (4 % more node tests on
// the benchmark frame), and the order is that of a full sort by (distance
// without its 3 low bits, child): finding the two nearest of 8 takes 17
// min/max operations where a sorting network takes 38 and up to 8 pushes.
// Shadow rays visit them from the last to the first (their answer does not
// depend on the order, and distance order is slower), as one group.
// The object loop pushes them all, as push_children does, but the nearest.
template <int Q>
__device__ __forceinline__ void trace_node(const DevScene& S, TraceState& t, SplitStack& st, uint32_t todo) {
  uint32_t const ref = t.ref;
  uint32_t next = kNoRef;
  const WideNode& nd = S.nodes[ref];
  if (Q == kQueryLoop) {
    float tc[8];
    int hits = 0, rank[8];
    node_children<false>(nd, t.w, t.z, [&](int c, float entry, bool hit) {
      tc[c] = hit ? entry : 0.f;
      hits += hit ? 1 : 0;
    });
    if (st.sp + hits > kSplitCap) {
      st.flags |= kTravOverflow;
      t.kind = kLaneDone;
      return;
    }
    child_ranks(tc, rank);
#pragma unroll
    for (int c = 0; c < 8; c++)
      if (tc[c] != 0.f) {
        if (rank[c] == hits - 1) next = nd.child[c];
        else st.put(st.sp + rank[c], StackEntry{nd.child[c], tc[c]});
      }
    st.sp += hits > 0 ? hits - 1 : 0;
    trace_next(t, next);
    return;
  }
  if (st.sp + 2 > kSplitCap) {
    st.flags |= kTravOverflow;
    t.kind = kLaneDone;
    return;
  }
  uint32_t m = 0;
  if (Q == kQueryAny) {
    node_children<true>(nd, t.w, t.z, [&](int c, float, bool hit) {
      if (hit) m |= 1u << c;
    });
    if (m) {
      uint32_t const c = 31u - __clz(m);
      uint32_t const rest = m ^ (1u << c);
      if (rest) st.push(StackEntry{ref | kGroupBit, __uint_as_float(rest)});
      next = nd.child[c];
    }
    trace_next(t, next);
    return;
  }
  uint32_t key[8];
  node_children<true>(nd, t.w, t.z, [&](int c, float tc, bool hit) {
    key[c] = hit ? ((__float_as_uint(tc) & ~7u) | uint32_t(7 - c)) : 0xFFFFFFFFu;
    if (hit) m |= 1u << c;
  });
  if (todo != 0xFFu) {
    m &= todo;
#pragma unroll
    for (int c = 0; c < 8; c++)
      if (!((todo >> c) & 1u)) key[c] = 0xFFFFFFFFu;
  }
  // the two smallest keys
  uint32_t lo[4], hi[4];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    lo[k] = min(key[2 * k], key[2 * k + 1]);
    hi[k] = max(key[2 * k], key[2 * k + 1]);
  }
#pragma unroll
  for (int n = 2; n > 0; n >>= 1)
#pragma unroll
    for (int k = 0; k < n; k++) {
      uint32_t const a = max(lo[k], lo[k + n]);
      lo[k] = min(lo[k], lo[k + n]);
      hi[k] = __vimin3_u32(a, hi[k], hi[k + n]);
    }
  if (m) {
    uint32_t const c1 = 7u - (lo[0] & 7u);
    next = nd.child[c1];
    m ^= 1u << c1;
    if (m) {
      uint32_t const c2 = 7u - (hi[0] & 7u);
      uint32_t const ref2 = nd.child[c2];
      m ^= 1u << c2;
      if (m) st.push(StackEntry{ref | kGroupBit, __uint_as_float((hi[0] & ~0xFFu) | m)});
      st.push(StackEntry{ref2, __uint_as_float(hi[0] & ~7u)});
    }
  }
  trace_next(t, next);
}

// Tests the triangles of mesh leaf t.ref.  accept(face, b0, b1, b2, point,
// distance) records a closer hit.
template <int Q, class A>
__device__ __forceinline__ void trace_leaf(const DevScene& S, TraceState& t, uint32_t& tris, A accept) {
  bool const any = Q == kQueryAny || (Q == kQueryClosest && t.phase == 2);
  uint32_t const cnt = ((t.ref >> 28) & 7u) + 1u;
  uint32_t const slot = t.ref & kSlotMask;
  t.kind = kLanePop;
  f3 const mr = cross3(t.w.p, t.w.u);
  for (uint32_t k = 0; k < cnt; k++) {
    const TriSlot& T = S.tris[slot + k];
    tris++;
    float tt, b0, b1, b2;
    if (tri_test(T, t.w, mr, t.z, tt, b0, b1, b2)) {
      t.obj = t.cur;
      if (any) {
        t.kind = kLaneDone;
        return;
      }
      t.z = tt;
      t.exit = t.cur_exit;
      accept(__float_as_uint(T.v0[3]), b0, b1, b2, ray_at(t.w, tt), tt);
    }
  }
}

// Tests the object of instance leaf t.ref (the rest of the leaf waits on the
// stack): a sphere or plane in full, a mesh by its bounds, after which the
// next step enters its tree.
template <int Q, class A>
__device__ __forceinline__ void trace_object(const DevScene& S, TraceState& t, SplitStack& st, uint32_t& insts,
                                             A accept) {
  bool const any = Q == kQueryAny || (Q == kQueryClosest && t.phase == 2);
  uint32_t const cnt = ((t.ref >> 28) & 7u) + 1u;
  uint32_t const slot = t.ref & kSlotMask;
  t.kind = kLanePop;
  uint32_t const i = Q == kQueryLoop ? slot : S.tlas_objects[slot];
  if (Q != kQueryLoop && cnt > 1) {
    if (st.sp + 1 > kSplitCap) {
      st.flags |= kTravOverflow;
      t.kind = kLaneDone;
      return;
    }
    st.push(StackEntry{kLeafBit | ((cnt - 2u) << 28) | (slot + 1u), 0.f});
  }
  if (Q == kQueryAny && i == t.wobj) return;
  if (Q == kQueryClosest && ((t.phase == 2 && i >= t.wobj) || (t.phase == 3 && i == t.wobj))) return;
  insts++;
  const DevObject& ob = S.objects[i];
  bool const low = Q == kQueryClosest && !any && t.obj != UINT32_MAX && i < t.obj;
  // a lower-index object loses ties: it has to be hit below the next float
  float const z = low ? prev_float(t.z) : t.z;
  Ray const li = to_local(ob, t.w);
  if (ob.type != LGPU_OBJ_TRIMESH) {
    float tt;
    f3 x;
    bool hit;
    if (ob.type == LGPU_OBJ_SPHERE) {
      hit = sphere_test(li, z, tt);
      if (hit) x = ray_at(li, tt);
    } else {
      hit = plane_test(li, z, tt, x);
    }
    if (hit) {
      t.obj = i;
      if (any) {
        t.kind = kLaneDone;
        return;
      }
      t.z = tt;
      t.exit = -1.f;
      accept(UINT32_MAX, 0.f, 0.f, 0.f, x, tt);
    }
    return;
  }
  const DevMesh& m = S.meshes[ob.mesh];
  bool inside;
  float ex;
  float r0 = aabb_scalar(m.bounds, li, z, inside, ex);
  // shadow rays and the reference's loop enter a mesh from inside at its exit
  // distance
  if (Q == kQueryClosest && r0 != kFltMax && inside) {
    t.n_inside++;
    r0 = kBias;
  }
  if (r0 == kFltMax || r0 > z) return;
  st.ws[0] = t.w.p.x;
  st.ws[128] = t.w.p.y;
  st.ws[2 * 128] = t.w.p.z;
  st.ws[3 * 128] = t.w.u.x;
  st.ws[4 * 128] = t.w.u.y;
  st.ws[5 * 128] = t.w.u.z;
  st.ws[6 * 128] = t.w.inv.x;
  st.ws[7 * 128] = t.w.inv.y;
  st.ws[8 * 128] = t.w.inv.z;
  t.w = li;
  t.z = z;
  t.cur = i;
  t.cur_exit = inside ? ex : -1.f;
  t.lowered = low;
  t.base = st.sp;
  trace_next(t, Q == kQueryLoop ? m.root : m.trav_root);
}

// intersect::scene for the wavefront kernels: the instance BVH through
// trace_tlas, the reference's linear object loop (nested traversal, local
// stack) for reference order, tiny scenes and the order-dependent case.
template <bool ANY>
__device__ __forceinline__ bool scene_trace(const DevScene& S, const Ray& w, HitRec& h, uint32_t skip,
                                            bool reference_order, SplitStack& st, StackEntry* lstack,
                                            StackEntry* ltstack, TravStats& ts) {
  if (reference_order || S.n_objects <= 4)
    return scene_hit<ANY>(S, w, h, skip, true, lstack, ltstack, ts);
  HitRec const h0 = h;
  bool hit = trace_tlas<ANY>(S, w, h, skip, st, ts);
  if (!ANY && hit && h.inside && h.exit > h.z) {
    h = h0;
    hit = scene_hit<false>(S, w, h, skip, true, lstack, ltstack, ts);
  }
  return hit;
}

}  // namespace lgpu
