// Device code of the renderer: the device scene image, the exact scene
// evaluators (leaf BVH, union_round trees, generic leaves), the persistent
// depth march, the Whitted trace, the FP16 brick cache, the batched launch and
// the adjoint march.  Compiled by nvcc into the library and, with FT_JIT
// defined, by NVRTC at run time together with a scene's hook programs lowered
// to CUDA (ft_scene_jit); it therefore includes no host headers.
#pragma once

#ifndef FT_JIT
#include <cuda_fp16.h>
#endif

#include "ft_device.cuh"
#include "ft_layout.h"

using ftd::DevNode;
using ftd::F3;
using ftd::f3;
using ftd::Info;

namespace {

#ifdef FT_JIT
// (the run-time compiler has no constant-expression infinity builtin)
#define kInf (__int_as_float(0x7f800000))
#else
constexpr float kInf = __builtin_huge_valf();
#endif

struct DevLeaf {
  float bmin[3], bmax[3];
  int32_t kind, node, first, count;
};
struct DevBvhNode {
  float bmin[3], bmax[3];
  int32_t lhs, rhs, leaf, pad;
};
// Candidate grid: cell c of the box from gmin lists (DevScene::cells, cell
// first + c) the primitives that can be the nearest or lie within the blend
// radius at some point of it.  dims[0] == 0: none.
struct alignas(16) DevGrid {
  float gmin[3];
  float inv_cell;
  int32_t dims[3];
  int32_t first;
};
// Distance up to which a cell lists every primitive: a little above the blend
// radius, so that a hit (whose own distance is at most epsilon) finds all the
// primitives with a weight in its normal and material in its cell's list.
__host__ __device__ inline float ur_list_reach(float r) { return 1.05f * r + 1.0e-3f; }
struct DevUrTree {
  float r;
  int32_t n_prims, prim_first, bvh_root, inner_root, depth, fallback_first, fallback_count;
  int32_t far_first, far_end;  // far-walk nodes
  DevGrid fine, outer;
};
struct DevUrBvh {
  float bmin[3], bmax[3];
  int32_t left, right, prim_begin, prim_count;
};
struct DevUrInner {
  int32_t child[2];
  int32_t lo, hi;
};

// Scenes whose distance has a short form, taken by the march loops without
// the general leaf walk; its data are kernel parameters, read from the constant
// bank.
//   kFastTree   one union_round tree (`tree`, box 1), alone or beside one
//               primitive whose distance is at least its box's (entry[0],
//               box 0; an extruded polygon's is not);
//   kFastPair   two primitives (entry and boxes 0, 1: the BVH root's children);
//   kFastUnion  primitives only: the first n_always compact records at every
//               point, the others through the candidate grids and far walk of
//               `tree`, box 1 around them;
//   kFastLeaves one or two leaves of any other kinds (leaf and boxes 0, 1; one
//               leaf is leaf[1], with leaf[0] -1), entry[k] where leaf k is a
//               primitive.
enum FastKind : int32_t { kFastLeaves = -1, kFastNone = 0, kFastTree = 1, kFastPair = 2, kFastUnion = 3 };
struct alignas(16) DevFast {
  int32_t kind;
  int32_t n_always;
  int32_t tree_lhs;   // kFastTree: the tree is the BVH root's left child
  int32_t all;        // kFastUnion: every primitive is in the first n_always
  uint32_t entry[2];  // compact entries, kNoPrim for none
  int32_t leaf[2];    // kFastLeaves
  float4 rec[3];      // the compact record of entry[0], or of the first always-evaluated primitive
  float bmin[2][3], bmax[2][3];
  DevUrTree tree;
};
constexpr uint32_t kNoPrim = 0xffffffffu;
constexpr uint32_t kInsideCell = 0xffffffffu;  // entry count of a cell inside one primitive

struct DevScene {
  DevFast fast;
  const DevNode* __restrict__ nodes;
  const DevLeaf* __restrict__ leaves;
  const int4* __restrict__ leaf_info;  // per leaf: kind, node, first (hooked: record, -1 none), count
  const float4* __restrict__ hooked;   // records of hooked leaves (kHookedWords each)
  const DevBvhNode* __restrict__ bvh;
  const float4* __restrict__ bvh_pairs;  // per inner node of bvh: { lmin, lhs } { lmax, - } { rmin, rhs } { rmax, - }
  const uint32_t* __restrict__ gops;
  const DevUrTree* __restrict__ urtrees;
  const DevUrBvh* __restrict__ ur_bvh;
  const int32_t* __restrict__ ur_bvh_prims;
  const int32_t* __restrict__ ur_prims;
  const DevUrInner* __restrict__ ur_inner;
  const float4* __restrict__ cprims;   // compact primitives (three words each, compact_distance)
  const uint4* __restrict__ ur_paths;  // per tree primitive: sides taken from the root (low, high word), depth
  const uint2* __restrict__ cells;     // per grid cell: first entry, entries
  const float4* __restrict__ far_nodes;     // two words per node (ftgpu::FarNode)
  const uint32_t* __restrict__ far_entries;  // compact entries of the far walks' leaves
  const uint2* __restrict__ entries;   // lower bound of the distance from the cell (ascending), compact index | rare
  const ft_program* __restrict__ programs;
  const ft_instr* __restrict__ instrs;
  const ft_material* __restrict__ materials;
  const ft_light* __restrict__ lights;
  const int32_t* __restrict__ node_op_begin;
  const int32_t* __restrict__ node_op_end;
  const int32_t* __restrict__ ur_inner_blend;
  const int32_t* __restrict__ obj_node;     // per object id: the node carrying its transform, -1 none
  int32_t n_obj_node;
  int32_t n_materials, n_lights, env_program;
  int32_t bvh_root;
  int32_t bvh_ref;  // the root as a pair reference: an index into bvh_pairs, or ~leaf
  float smin[3], smax[3];
};

#ifdef FT_JIT
// The scene's hook programs lowered to CUDA (generated by ft_scene_jit and
// defined after this header in the same translation unit).
__device__ F3 ft_jit_program(int index, const F3* args);
#endif

// Hook program `index` of the scene: native code in a run-time compiled
// module, the register interpreter otherwise.
__device__ __forceinline__ F3 scene_program(const DevScene& S, int index, const F3* args,
                                            unsigned long long* instr_count) {
#ifdef FT_JIT
  return ft_jit_program(index, args);
#else
  return ftd::run_program(S.programs[index], S.instrs, args, instr_count);
#endif
}

struct RayParams {
  float origin[3], fwd[3], right[3], up[3];
  float tan_fov, aspect;
  uint32_t width, height, aa, grid, max_steps;
  float max_dist, eps, step_scale;
  uint32_t tiles_x;
  uint32_t tile_w, tile_h;  // pixels per work tile (rays of a tile are consecutive work items)
  uint32_t refill;          // idle lanes that make a warp of the persistent march refill
  uint32_t jitter;          // 1: jittered AA offsets (XorShift64 per pixel sample), 0: the sqrt(aa) grid
  uint32_t jitter_seed;     // xor-ed into each pixel sample's seed
  uint64_t n_items;
};

// XorShift64 (R:4735-4761): the jittered sub-pixel offsets of the progressive
// renderer, seeded per pixel sample by seed_pixel_sample (R:4763-4774).
struct XorShift64 {
  unsigned long long state;
  __device__ explicit XorShift64(unsigned long long seed) : state(seed == 0ull ? 0x9E3779B97F4A7C15ull : seed) {}
  __device__ unsigned long long next_u64() {
    unsigned long long x = state;
    x ^= x << 13;
    x ^= x >> 7;
    x ^= x << 17;
    state = x;
    return x;
  }
  __device__ float next_f32() {
    const uint32_t v = static_cast<uint32_t>(next_u64() >> 40);
    return static_cast<float>(v) / static_cast<float>(1u << 24);
  }
};

__device__ __forceinline__ unsigned long long seed_pixel_sample(uint32_t x, uint32_t y, uint32_t width, uint32_t s) {
  const unsigned long long base = (static_cast<unsigned long long>(y) * width + x) * 0x9E3779B97F4A7C15ull +
                                  0xBF58476D1CE4E5B9ull;
  return base ^ (static_cast<unsigned long long>(s) * 0x94D049BB133111EBull) ^ 0xD6E8FEB86659FD93ull;
}

// NDC of primary sample s of pixel (px, py) before the aspect scale: the
// sqrt(aa) x sqrt(aa) grid of pixel_sample_offsets (R:4838-4854) in the NDC
// map of render_depth_tile (R:3951-3955), or the jittered offsets of the
// progressive renderer (R:4008-4013).
__device__ __forceinline__ void sample_ndc(const RayParams& P, uint32_t px, uint32_t py, uint32_t s, float* nx,
                                           float* ny) {
  if (P.jitter) {
    XorShift64 rng(seed_pixel_sample(px, py, P.width, s) ^ static_cast<unsigned long long>(P.jitter_seed));
    const float jx = rng.next_f32() - 0.5f;
    const float jy = rng.next_f32() - 0.5f;
    *nx = ((static_cast<float>(px) + 0.5f + jx) / static_cast<float>(P.width)) * 2.0f - 1.0f;
    *ny = 1.0f - ((static_cast<float>(py) + 0.5f + jy) / static_cast<float>(P.height)) * 2.0f;
    return;
  }
  const float sx = (static_cast<float>(s % P.grid) + 0.5f) / static_cast<float>(P.grid);
  const float sy = (static_cast<float>(s / P.grid) + 0.5f) / static_cast<float>(P.grid);
  *nx = ((static_cast<float>(px) + sx) / static_cast<float>(P.width)) * 2.0f - 1.0f;
  *ny = 1.0f - ((static_cast<float>(py) + sy) / static_cast<float>(P.height)) * 2.0f;
}


// Per-thread work counters (only compiled into the statistics variant).
struct Counters {
  unsigned long long evals, prims, boxes, hook_instrs, steps, far_steps, fetches, blends, cands;
};
constexpr int kNumCounters = 9;

// Warp sum of every counter into stats[0 .. kNumCounters) (all 32 lanes call it).
__device__ __forceinline__ void flush_stats(const Counters& c, unsigned long long* stats) {
  unsigned long long v[kNumCounters] = {c.evals, c.prims, c.boxes, c.hook_instrs, c.steps,
                                        c.far_steps, c.fetches, c.blends, c.cands};
#pragma unroll
  for (int j = 0; j < kNumCounters; ++j) {
    unsigned long long x = v[j];
    for (int off = 16; off > 0; off >>= 1) x += __shfl_down_sync(0xffffffffu, x, off);
    if ((threadIdx.x & 31u) == 0u && x) atomicAdd(&stats[j], x);
  }
}

template <bool kStats>
struct Ctx {
  Counters c;
  __device__ void eval() {
    if (kStats) ++c.evals;
  }
  __device__ void prim() {
    if (kStats) ++c.prims;
  }
  __device__ void box(unsigned n = 1) {
    if (kStats) c.boxes += n;
  }
  __device__ void step() {
    if (kStats) ++c.steps;
  }
  __device__ void far_step() {
    if (kStats) ++c.far_steps;
  }
  __device__ void fetch() {
    if (kStats) ++c.fetches;
  }
  // union_round combines of a restricted fold, candidate-list entries tested
  __device__ void blend(unsigned n = 1) {
    if (kStats) c.blends += n;
  }
  __device__ void cand() {
    if (kStats) ++c.cands;
  }
  __device__ unsigned long long* hooks() { return kStats ? &c.hook_instrs : nullptr; }
};

__device__ __forceinline__ float node_lb(F3 p, const float* mn, const float* mx) { return ftd::aabb_lb(p, mn, mx); }

// Object and material id of an evaluation's surface.
__device__ __forceinline__ uint2 surface_ids(const DevScene& S, int32_t ref) {
  if (ref == ftd::kNoRef) return make_uint2(0u, 0u);
  const int node = ref >= 0 ? ref : __float_as_int(__ldg(S.cprims + 3 * static_cast<size_t>(~ref) + 2).z);
  return make_uint2(S.nodes[node].object_id, S.nodes[node].material_id);
}

// A primitive of a kind without a compact record, out of line.
__device__ __noinline__ float rare_distance(const DevNode& n, F3 p) { return ftd::prim_distance(n, p); }

// eval_custom_sdf_distance (R:6139-6180) of a Custom node (a user `sdf`
// definition): the point in its frame, through domain(p) when present, into
// distance(p), then distance_post(d, p) when present.  The device node keeps
// the distance program in `program`, domain in `ival`, distance_post in `b`.
template <bool kStats>
__device__ __noinline__ float custom_distance(const DevScene& S, const DevNode& n, F3 p, Ctx<kStats>& cx) {
  cx.prim();
  F3 q = ftd::to_local(p, n);
  if (n.ival >= 0) q = scene_program(S, n.ival, &q, cx.hooks());
  float d = scene_program(S, n.program, &q, cx.hooks()).x;
  if (n.b >= 0) {
    F3 args[2] = {f3(d, d, d), q};
    d = scene_program(S, n.b, args, cx.hooks()).x;
  }
  return d;
}

// Generic leaf: postfix program over the leaf's node tree (exact).
template <bool kStats>
__device__ __noinline__ Info eval_generic(const DevScene& S, int first, int count, F3 p, Ctx<kStats>& cx) {
  Info vs[ftgpu::kMaxGenericValueStack];
  F3 ps[ftgpu::kMaxGenericPointStack];
  int vsp = 0, psp = 0;
  ps[0] = p;
  for (int k = 0; k < count; ++k) {
    uint32_t w = S.gops[first + k];
    uint32_t op = w >> ftgpu::kGOpShift;
    const DevNode& n = S.nodes[w & ftgpu::kGNodeMask];
    switch (op) {
      case ftgpu::kGPrim:
        cx.prim();
        vs[vsp++] = Info{ftd::prim_distance(n, ps[psp]), static_cast<int32_t>(w & ftgpu::kGNodeMask)};
        break;
      case ftgpu::kGDomainPush: {
        F3 q = ftd::to_local(ps[psp], n);
        ps[psp + 1] = scene_program(S, n.program, &q, cx.hooks());
        ++psp;
        break;
      }
      case ftgpu::kGLocalPush:
        ps[psp + 1] = ftd::to_local(ps[psp], n);
        ++psp;
        break;
      case ftgpu::kGPostPop: {
        float d = vs[vsp - 1].d;
        F3 args[2] = {f3(d, d, d), ps[psp]};
        vs[vsp - 1].d = scene_program(S, n.program, args, cx.hooks()).x;
        --psp;
        break;
      }
      case ftgpu::kGNoisePop:
        vs[vsp - 1].d = ftd::apply_noise(ps[psp], vs[vsp - 1].d, n.ival, n.f[0], n.f[1]);
        --psp;
        break;
      case ftgpu::kGPop: --psp; break;
      case ftgpu::kGBinary: {
        Info r = vs[--vsp];
        Info l = vs[--vsp];
        vs[vsp++] = ftd::combine(n.kind, n.f[0], n.f[1], l, r);
        break;
      }
      case ftgpu::kGSlice: {
        F3 q = ps[psp];
        float coord = n.ival == 0 ? q.x : (n.ival == 1 ? q.y : q.z);
        float slab = ftd::rmax(n.f[0] - coord, coord - n.f[1]);
        vs[vsp - 1].d = ftd::rmax(vs[vsp - 1].d, slab);
        break;
      }
      case ftgpu::kGSmooth: vs[vsp - 1].d -= n.f[0] * 0.1f; break;
      case ftgpu::kGCustom: vs[vsp++] = Info{custom_distance(S, n, ps[psp], cx), static_cast<int32_t>(w & ftgpu::kGNodeMask)}; break;
    }
  }
  return vs[0];
}

// union_round tree of primitives with a single radius r.
//
// For every primitive with exact distance >= r each union_round it feeds is
// in its min(a, b) regime (op_union_round, R:6024-6029), so the tree value
// only depends on the set N of primitives closer than r:
//   * N empty: the value is the minimum primitive distance, exactly;
//   * otherwise: evaluate the tree restricted to subtrees containing an
//     N-primitive, treating every other subtree as +inf, which reproduces
//     op_union_round(a, b, r) bit for bit for any b >= r.
// N is gathered through a BVH over the tree's primitives with pruning bound
// max(r, min(best so far, cutoff)); primitive AABBs bound their distances from
// below, so no primitive that can change the result is skipped.
//
// The restricted fold runs along root paths: a primitive's path gives the
// side taken at each depth, so the lowest common ancestor of two primitives is
// where their paths first differ, and no node is loaded on the way.

// Primitive `idx` of the compact array at p.
template <bool kSphereYX = false, bool kStats>
__device__ __forceinline__ float compact_at(const DevScene& S, uint32_t entry, F3 p, Ctx<kStats>& cx) {
  cx.prim();
  const float4* w = S.cprims + 3 * static_cast<size_t>(entry & ~ftd::kRareFlag);
  const float4 c = __ldg(w + 2);
  if (entry & ftd::kRareFlag) return rare_distance(S.nodes[__float_as_int(c.z)], p);
  return ftd::compact_distance<kSphereYX>(__ldg(w), __ldg(w + 1), c.x, c.y, p);
}

// Value one level up of a subtree whose sibling holds no near primitive: the
// other child is +inf (exact for any far subtree, see above), on either side.
__device__ __forceinline__ float ur_lift(float v, float r) { return ftd::op_union_round(v, kInf, r); }

// `levels` lifts.  Once a lift returns its input unchanged, every further one
// does too, so the walk ends.
template <bool kStats>
__device__ __forceinline__ float ur_lifts(float v, int levels, float r, Ctx<kStats>& cx) {
  for (int k = 0; k < levels; ++k) {
    const float lifted = ur_lift(v, r);
    cx.blend();
    if (lifted == v) break;
    v = lifted;
  }
  return v;
}

// Depth at which two root paths part.
__device__ __forceinline__ int ur_lca(uint4 a, uint4 b) {
  const uint32_t lo = a.x ^ b.x, hi = a.y ^ b.y;
  return lo ? __ffs(static_cast<int>(lo)) - 1 : 31 + __ffs(static_cast<int>(hi));
}

// op_union_round of two subtrees, the ids of the smaller child (combine).
__device__ __forceinline__ Info ur_join(Info l, Info r, float radius) {
  return Info{ftd::op_union_round(l.d, r.d, radius), l.d <= r.d ? l.ref : r.ref};
}

// The fold for three or more near primitives, out of line: sorted by in-order
// position they are joined deepest common ancestor first, holding the subtrees
// whose right part is still open on a stack.
template <bool kStats>
__device__ __noinline__ Info ur_fold_many(const DevScene& S, float r, int* idx, float* dist, int nn,
                                          Ctx<kStats>& cx) {
  for (int i = 1; i < nn; ++i) {
    const int ki = idx[i];
    const float kd = dist[i];
    int j = i - 1;
    for (; j >= 0 && idx[j] > ki; --j) {
      idx[j + 1] = idx[j];
      dist[j + 1] = dist[j];
    }
    idx[j + 1] = ki;
    dist[j + 1] = kd;
  }
  Info open[ftgpu::kUrNear];
  int at[ftgpu::kUrNear];  // depth of the ancestor that joins open[k] with what follows
  int sp = 0;
  uint4 path = __ldg(S.ur_paths + idx[0]);
  Info cur{0.0f, ftd::kNoRef};
  for (int i = 0; i < nn; ++i) {
    cur = Info{dist[i], ~idx[i]};
    int dep = static_cast<int>(path.z), l = -1;
    if (i + 1 < nn) {
      const uint4 nxt = __ldg(S.ur_paths + idx[i + 1]);
      l = ur_lca(path, nxt);
      path = nxt;
    }
    while (sp > 0 && at[sp - 1] > l) {
      --sp;
      cur.d = ur_lifts(cur.d, dep - at[sp] - 1, r, cx);
      cur = ur_join(open[sp], cur, r);
      cx.blend();
      dep = at[sp];
    }
    cur.d = ur_lifts(cur.d, dep - l - 1, r, cx);
    if (l >= 0) {
      open[sp] = cur;
      at[sp++] = l;
    }
  }
  return cur;
}

// The fold for one or two near primitives, in registers.
template <bool kStats>
__device__ __forceinline__ Info ur_fold_small(const DevScene& S, float r, int i0, float d0, int i1, float d1, int nn,
                                              Ctx<kStats>& cx) {
  const uint4 a = __ldg(S.ur_paths + i0);
  if (nn == 1) return Info{ur_lifts(d0, static_cast<int>(a.z), r, cx), ~i0};
  const uint4 b = __ldg(S.ur_paths + i1);
  const int l = ur_lca(a, b);
  const Info v0{ur_lifts(d0, static_cast<int>(a.z) - l - 1, r, cx), ~i0};
  const Info v1{ur_lifts(d1, static_cast<int>(b.z) - l - 1, r, cx), ~i1};
  Info v = i0 < i1 ? ur_join(v0, v1, r) : ur_join(v1, v0, r);  // the smaller position is in the left subtree
  cx.blend();
  v.d = ur_lifts(v.d, l, r, cx);
  return v;
}

// The near set of a union_round tree at a point: the nearest primitive, and
// those closer than r: the first two in registers, further ones, rare, in the
// caller's arrays (idx, dist; they are handed to the out-of-line fold, which
// would otherwise put the whole set into local memory).
struct UrNear {
  Info best{kInf, ftd::kNoRef};
  int i0 = 0, i1 = 0, nn = 0;
  float d0 = 0.0f, d1 = 0.0f;
  __device__ __forceinline__ void add(int i, float d, float r, int* idx, float* dist) {
    if (d < best.d) best = Info{d, ~i};
    if (d < r) {
      if (nn == 0) {
        i0 = i;
        d0 = d;
      } else if (nn == 1) {
        i1 = i;
        d1 = d;
      } else if (nn < ftgpu::kUrNear) {
        idx[nn] = i;
        dist[nn] = d;
      }
      ++nn;
    }
  }
  // limit below which a primitive still matters
  __device__ __forceinline__ float limit(float r, float cutoff) const { return ftd::rmax(r, fminf(best.d, cutoff)); }
};

// Tree value from its near set.
template <bool kStats>
__device__ __forceinline__ Info ur_value(const DevScene& S, const DevUrTree& t, const UrNear& n, int* idx,
                                         float* dist, F3 p, Ctx<kStats>& cx) {
  if (n.nn == 0) return n.best;
  if (n.nn <= 2) return ur_fold_small(S, t.r, n.i0, n.d0, n.i1, n.d1, n.nn, cx);
  if (n.nn > ftgpu::kUrNear) return eval_generic(S, t.fallback_first, t.fallback_count, p, cx);
  idx[0] = n.i0;
  dist[0] = n.d0;
  idx[1] = n.i1;
  dist[1] = n.d1;
  return ur_fold_many(S, t.r, idx, dist, n.nn, cx);
}

// Nearest primitive below best.d from a point outside the candidate grids,
// where every primitive is outside its box: the nodes in depth-first order, a
// subtree skipped when its box is farther than the best so far.  Out of
// line: it is rare beside the grids' cell walks, whose code stays in the march
// loops.  A node is two 16-byte loads and there is no stack: the leaf-BVH walk
// it replaces for these points spent over a thousand cycles on a node (14
// scalar loads and a stack in local memory), and rays that pass over a scene
// set the time of a small frame.  `tie`: whether the distance found occurred
// twice.
template <bool kSphereYX, bool kStats>
__device__ __noinline__ Info far_nearest(const DevScene& S, const DevUrTree& t, F3 p, Info best, bool* tie,
                                         Ctx<kStats>& cx) {
  bool same = false;
  for (int k = t.far_first; k < t.far_end;) {
    const float4 a = __ldg(S.far_nodes + 2 * static_cast<size_t>(k));
    const float4 b = __ldg(S.far_nodes + 2 * static_cast<size_t>(k) + 1);
    const float mn[3] = {a.x, a.y, a.z}, mx[3] = {b.x, b.y, b.z};
    cx.box();
    if (ftd::aabb_lb2(p, mn, mx) > 1.000001f * best.d * best.d) {  // (not an equally near one, whatever the rounding)
      k = __float_as_int(a.w);
      continue;
    }
    const int prims = __float_as_int(b.w);
    if (prims >= 0) {
      for (int e = prims >> 3, end = e + (prims & 7); e < end; ++e) {
        const uint32_t entry = __ldg(S.far_entries + e);
        const float d = compact_at<kSphereYX>(S, entry, p, cx);
        same = d == best.d || (same && !(d < best.d));
        if (d < best.d) best = Info{d, ~static_cast<int32_t>(entry & ~ftd::kRareFlag)};
      }
    }
    ++k;
  }
  *tie = same;
  return best;
}

// The BVH walk of a tree without candidate grids, out of line.
template <bool kStats>
__device__ __noinline__ Info eval_urtree_far(const DevScene& S, const DevUrTree& t, F3 p, float cutoff,
                                             Ctx<kStats>& cx) {
  UrNear n;
  int near_idx[ftgpu::kUrNear];
  float near_dist[ftgpu::kUrNear];
  int stack[48];
  int sp = 0;
  stack[sp++] = t.bvh_root;
  for (int walk = 0; sp > 0 && walk < ftgpu::kMaxWalk; ++walk) {  // a tree walk pops each node once
    const DevUrBvh& bn = S.ur_bvh[stack[--sp]];
    cx.box();
    if (node_lb(p, bn.bmin, bn.bmax) >= n.limit(t.r, cutoff)) continue;
    if (bn.prim_count > 0) {
      for (int k = 0; k < bn.prim_count; ++k) {
        const int idx = t.prim_first + S.ur_bvh_prims[bn.prim_begin + k];
        const DevNode& pn = S.nodes[S.ur_prims[idx]];
        cx.box();
        if (node_lb(p, pn.bmin, pn.bmax) >= n.limit(t.r, cutoff)) continue;
        const uint32_t rare = __float_as_uint(__ldg(S.cprims + 3 * static_cast<size_t>(idx) + 2).w) & ftd::kRareFlag;
        n.add(idx, compact_at(S, static_cast<uint32_t>(idx) | rare, p, cx), t.r, near_idx, near_dist);
      }
      continue;
    }
    const DevUrBvh& L = S.ur_bvh[bn.left];
    const DevUrBvh& R = S.ur_bvh[bn.right];
    float ll = node_lb(p, L.bmin, L.bmax), rl = node_lb(p, R.bmin, R.bmax);
    if (sp + 2 > 48) return eval_generic(S, t.fallback_first, t.fallback_count, p, cx);
    if (ll <= rl) {
      stack[sp++] = bn.right;
      stack[sp++] = bn.left;
    } else {
      stack[sp++] = bn.left;
      stack[sp++] = bn.right;
    }
  }
  return ur_value(S, t, n, near_idx, near_dist, p, cx);
}

// Cell of p in a grid; false outside it.
__device__ __forceinline__ bool grid_cell(const DevGrid& g, F3 p, int* cell) {
  const float gx = (p.x - g.gmin[0]) * g.inv_cell, gy = (p.y - g.gmin[1]) * g.inv_cell,
              gz = (p.z - g.gmin[2]) * g.inv_cell;
  if (!(gx >= 0.0f && gy >= 0.0f && gz >= 0.0f && gx < (float)g.dims[0] && gy < (float)g.dims[1] &&
        gz < (float)g.dims[2]))
    return false;
  const int ix = min((int)gx, g.dims[0] - 1), iy = min((int)gy, g.dims[1] - 1), iz = min((int)gz, g.dims[2] - 1);
  *cell = g.first + ix + g.dims[0] * (iy + g.dims[1] * iz);
  return true;
}

// A walk is bound by the latency of its three dependent loads (cell, entry,
// primitive) and the branches between them, so each is one vector load of a
// compact record and the distance has no branch.  With the scene's header in
// the constant bank, the 512-primitive field's depth frame (1920x1080, 2x2)
// takes 10.6 ms, against 29.8 ms with scalar loads from 128-byte nodes, a box
// test per candidate and parent-link folds.
//
// The tree's value at p, exact where it is below `cutoff`: the candidates of
// p's cell in the fine grid, or outside it in the coarser outer grid around it
// (its cells list the primitives that can be the nearest there), else the
// nearest primitive (outside the grids all are more than r away).  A cell's list is sorted by a lower bound of its points'
// distances, so the first entry at or above the running limit ends it.
template <bool kStats>
__device__ __forceinline__ Info eval_urtree(const DevScene& S, const DevUrTree& t, F3 p, float cutoff,
                                            Ctx<kStats>& cx) {
  int cell = 0;
  if (!grid_cell(t.fine, p, &cell) && !grid_cell(t.outer, p, &cell)) {
    bool tie;
    return t.fine.dims[0] > 0 ? far_nearest<false>(S, t, p, Info{cutoff, ftd::kNoRef}, &tie, cx)
                              : eval_urtree_far(S, t, p, cutoff, cx);
  }
  const uint2 range = __ldg(S.cells + cell);
  const float r = t.r;
  UrNear n;
  int near_idx[ftgpu::kUrNear];
  float near_dist[ftgpu::kUrNear];
  for (uint32_t k = range.x, end = range.x + range.y; k < end; ++k) {
    const uint2 e = __ldg(S.entries + k);
    cx.cand();
    if (__uint_as_float(e.x) >= n.limit(r, cutoff)) break;
    n.add(static_cast<int>(e.y & ~ftd::kRareFlag), compact_at(S, e.y, p, cx), r, near_idx, near_dist);
  }
  return ur_value(S, t, n, near_idx, near_dist, p, cx);
}

// A leaf [distance_post] [domain] primitive, the common form of a hooked
// object, in registers: the steps of its postfix program (eval_generic keeps
// its operands in local memory).
template <bool kStats>
__device__ __noinline__ Info eval_hooked(const DevScene& S, int node, F3 p, Ctx<kStats>& cx) {
  const DevNode* n = &S.nodes[node];
  const DevNode* post = nullptr;
  F3 pp = p;
  if (n->kind == FT_NODE_DISTANCE_POST) {
    post = n;
    pp = ftd::to_local(p, *n);
    node = n->a;
    n = &S.nodes[node];
  }
  F3 q = pp;
  if (n->kind == FT_NODE_DOMAIN) {
    F3 local = ftd::to_local(pp, *n);
    q = scene_program(S, n->program, &local, cx.hooks());
    node = n->a;
    n = &S.nodes[node];
  }
  cx.prim();
  float d = ftd::prim_distance(*n, q);
  if (post) {
    F3 args[2] = {f3(d, d, d), pp};
    d = scene_program(S, post->program, args, cx.hooks()).x;
  }
  return Info{d, node};
}

// The leaves of the leaf BVH in the order of bvh_distance_info (R:743-786):
// nearest child first, a node left out when its box bound exceeds the best
// distance at that time.  next() descends to the next leaf and returns, so
// the lanes of a warp reach their leaves' evaluations together instead of
// half of them waiting on box tests.  A node's two child boxes are four
// 16-byte loads; the nearer child stays in registers.
template <bool kStats>
struct LeafWalk {
  static constexpr int kStack = 48;  // (the median-split build is about log2(leaves) deep)
  F3 p;
  int ref, sp = 0;
  float lb;
  bool have = true;
  int stack[kStack];
  float bound[kStack];
  __device__ __forceinline__ LeafWalk(const DevScene& S, F3 q, Ctx<kStats>& cx) : p(q), ref(S.bvh_ref) {
    lb = node_lb(q, S.smin, S.smax);
    cx.box();
  }
  // Next leaf whose bound is not above `best`, -1 at the end; its bound is lb.
  __device__ __forceinline__ int next(const DevScene& S, float best, Ctx<kStats>& cx) {
    for (int walk = 0; walk < ftgpu::kMaxWalk; ++walk) {  // a tree walk visits each node once
      if (!have) {
        if (sp == 0) return -1;
        --sp;
        ref = stack[sp];
        lb = bound[sp];
      }
      have = false;
      if (lb > best) continue;
      if (ref < 0) return ~ref;
      const float4* w = S.bvh_pairs + 4 * static_cast<size_t>(ref);
      const float4 a = __ldg(w), b = __ldg(w + 1), c = __ldg(w + 2), e = __ldg(w + 3);
      const float lmn[3] = {a.x, a.y, a.z}, lmx[3] = {b.x, b.y, b.z}, rmn[3] = {c.x, c.y, c.z}, rmx[3] = {e.x, e.y, e.z};
      const float ll = node_lb(p, lmn, lmx), rl = node_lb(p, rmn, rmx);
      cx.box(2);
      if (sp == kStack) return -1;  // deeper than the build makes it
      const bool lfirst = ll <= rl;
      stack[sp] = __float_as_int(lfirst ? c.w : a.w);
      bound[sp] = lfirst ? rl : ll;
      ++sp;
      ref = __float_as_int(lfirst ? a.w : c.w);
      lb = lfirst ? ll : rl;
      have = true;
    }
    return -1;
  }
};

// The general leaf walk's tree evaluation, out of line (the short scene form
// inlines its own).
template <bool kStats>
__device__ __noinline__ Info eval_urtree_leaf(const DevScene& S, const DevUrTree& t, F3 p, float cutoff,
                                              Ctx<kStats>& cx) {
  return eval_urtree(S, t, p, cutoff, cx);
}

// The same from the leaf's record (modifiers without rotation over a compact
// primitive): { post centre, post program } { domain centre, domain program }
// and the primitive's three words, program -1 for a modifier it has not.  The
// lanes of a warp are at different leaves, so a load is a transaction per lane
// whatever its width: five of 16 bytes replace some thirty of 4 (512 compiled
// shells, 640x360: 54.4 -> 48.2 ms).
constexpr int kHookedWords = 6;
template <bool kStats>
__device__ __noinline__ Info eval_hooked_record(const DevScene& S, int record, F3 p, Ctx<kStats>& cx) {
  const float4* w = S.hooked + kHookedWords * static_cast<size_t>(record);
  const float4 post = __ldg(w), dom = __ldg(w + 1), a = __ldg(w + 2), b = __ldg(w + 3), c = __ldg(w + 4);
  const int post_program = __float_as_int(post.w), dom_program = __float_as_int(dom.w);
  F3 pp = p;
  if (post_program >= 0) pp = f3(p.x - post.x, p.y - post.y, p.z - post.z);
  F3 q = pp;
  if (dom_program >= 0) {
    F3 local = f3(pp.x - dom.x, pp.y - dom.y, pp.z - dom.z);
    q = scene_program(S, dom_program, &local, cx.hooks());
  }
  cx.prim();
  float d = ftd::compact_distance<true>(a, b, c.x, c.y, q);
  if (post_program >= 0) {
    F3 args[2] = {f3(d, d, d), pp};
    d = scene_program(S, post_program, args, cx.hooks()).x;
  }
  return Info{d, __float_as_int(c.z)};
}

// A leaf other than a primitive.
template <bool kStats>
__device__ __forceinline__ Info eval_composite(const DevScene& S, int leaf, int4 info, F3 p, float cutoff,
                                               Ctx<kStats>& cx) {
  if (info.x == ftgpu::kLeafHooked)
    return info.z >= 0 ? eval_hooked_record(S, info.z, p, cx) : eval_hooked(S, info.y, p, cx);
  if (info.x == ftgpu::kLeafUrTree) return eval_urtree_leaf(S, S.urtrees[info.z], p, cutoff, cx);
  if (S.nodes[info.y].kind == FT_NODE_CUSTOM) {
    // accel_leaf_distance_info (R:635-657): a Custom leaf farther from its box
    // than a tenth of the box diagonal (clamped to [0.05, 0.5]) is that box
    // bound, not its program
    const DevLeaf& lf = S.leaves[leaf];
    cx.box();
    float lb = node_lb(p, lf.bmin, lf.bmax);
    float ex = lf.bmax[0] - lf.bmin[0], ey = lf.bmax[1] - lf.bmin[1], ez = lf.bmax[2] - lf.bmin[2];
    float far = ftd::rclamp(sqrtf(ex * ex + ey * ey + ez * ez) * 0.1f, 0.05f, 0.5f);
    if (lb > far) return Info{lb, info.y};
  }
  return eval_generic(S, info.z, info.w, p, cx);
}

template <bool kStats>
__device__ __forceinline__ Info eval_leaf(const DevScene& S, int leaf, F3 p, float cutoff, Ctx<kStats>& cx) {
  const int4 info = __ldg(S.leaf_info + leaf);  // kind, node, first, count
  if (info.x == ftgpu::kLeafPrim) {
    const DevNode& n = S.nodes[info.y];
    cx.prim();
    return Info{ftd::prim_distance(n, p), info.y};
  }
  return eval_composite(S, leaf, info, p, cutoff, cx);
}

// Accelerator::distance_info over the leaf BVH (bvh_distance_info,
// R:743-786): nearest-first, a node is skipped when its box bound exceeds the
// best distance so far, a later leaf replaces the result only when strictly
// closer.
template <bool kStats>
__device__ __noinline__ Info scene_distance_bvh(const DevScene& S, F3 p, Ctx<kStats>& cx) {
  Info cur{kInf, ftd::kNoRef};
  LeafWalk<kStats> walk(S, p, cx);
  for (int leaf; (leaf = walk.next(S, cur.d, cx)) >= 0;) {
    const Info in = eval_leaf(S, leaf, p, cur.d, cx);
    if (in.d < cur.d) cur = in;
  }
  return cur;
}

// The primitive of DevFast::rec (a ground, usually), from the constant bank.
template <bool kSphereYX, bool kStats>
__device__ __forceinline__ float fast_prim(const DevScene& S, F3 p, Ctx<kStats>& cx) {
  cx.prim();
  const float4* w = S.fast.rec;
  if (__float_as_uint(w[2].w) & ftd::kRareFlag) return rare_distance(S.nodes[__float_as_int(w[2].z)], p);
  return ftd::compact_distance<kSphereYX>(w[0], w[1], w[2].x, w[2].y, p);
}

__device__ __forceinline__ int32_t compact_ref(uint32_t entry) { return ~static_cast<int32_t>(entry & ~ftd::kRareFlag); }

// kFastTree with a primitive leaf: the two-leaf walk above (nearer box first,
// the other leaf when its box bound is not above the distance found) with the
// primitive evaluated first in either order, so that its distance bounds the
// tree's walk.  t2 and p2 are the squared box bounds of the tree and the
// primitive.  Where the tree comes first it is exact below the cutoff, and at
// or above it the primitive's distance wins as it would there (a walk outside
// the grids that finds nothing below the cutoff returns it without a surface);
// a negative primitive distance (a point inside it) does not cut the walk.
template <bool kStats>
__device__ __forceinline__ Info tree_and_prim(const DevScene& S, F3 p, float t2, float p2, Ctx<kStats>& cx) {
  const DevFast& F = S.fast;
  const bool tree_first = F.tree_lhs ? t2 <= p2 : t2 < p2;
  const Info prim{fast_prim<false>(S, p, cx), compact_ref(F.entry[0])};
  if (!tree_first && !(sqrtf(t2) <= prim.d)) return prim;
  const Info tree = eval_urtree(S, F.tree, p, tree_first && prim.d < 0.0f ? kInf : prim.d, cx);
  if (!tree_first) return tree.d < prim.d ? tree : prim;
  return tree.ref == ftd::kNoRef || (prim.d < tree.d && sqrtf(p2) <= tree.d) ? prim : tree;
}

// kFastPair: the two-leaf walk of two primitives.
template <bool kStats>
__device__ __forceinline__ Info pair_distance(const DevScene& S, F3 p, float l2, float r2, Ctx<kStats>& cx) {
  const DevFast& F = S.fast;
  const bool lfirst = l2 <= r2;
  const uint32_t e0 = lfirst ? F.entry[0] : F.entry[1], e1 = lfirst ? F.entry[1] : F.entry[0];
  const Info a{compact_at<true>(S, e0, p, cx), compact_ref(e0)};
  if (!(sqrtf(lfirst ? r2 : l2) <= a.d)) return a;
  const Info b{compact_at<true>(S, e1, p, cx), compact_ref(e1)};
  return b.d < a.d ? b : a;
}

// kFastLeaves: the nearer leaf, then the other when its box bound is not above
// the distance found (the strictly-closer replace of bvh_distance_info); l and
// r are the box bounds.  One evaluation site for both leaves.
template <bool kStats>
__device__ __forceinline__ Info leaves_distance(const DevScene& S, F3 p, float l, float r, Ctx<kStats>& cx) {
  const DevFast& F = S.fast;
  bool left = F.leaf[0] >= 0 && l <= r;
  const float second_lb = left ? r : l;
  Info cur{kInf, ftd::kNoRef};
#pragma unroll 1
  for (int k = 0; k < 2; ++k) {
    const uint32_t e = left ? F.entry[0] : F.entry[1];
    const int leaf = left ? F.leaf[0] : F.leaf[1];
    const Info in = e != kNoPrim ? Info{compact_at<true>(S, e, p, cx), compact_ref(e)}
                                 : eval_composite(S, leaf, __ldg(S.leaf_info + leaf), p, k == 0 ? kInf : cur.d, cx);
    if (k == 0 || in.d < cur.d) cur = in;
    if (F.leaf[0] < 0 || !(second_lb <= cur.d)) break;
    left = !left;
  }
  return cur;
}

// kFastUnion: the nearest of the always-evaluated primitives (all of a small
// scene; else the few whose box dwarfs the rest, a ground) and of the
// candidates of p's cell, in ascending order of their lower bounds, up to the
// first that cannot be nearer.
//
// The leaf-BVH walk (bvh_distance_info) gives the same nearest distance with
// two exceptions that depend on its order: inside the solids it keeps the
// first negative distance found (every other box bound is at least 0), and of
// equal distances the first.  So a point with two negative distances, or with
// a tie for the nearest, takes that walk, and one in a cell inside a solid.  A
// point outside both grids takes the far walk unless the box of the listed
// primitives is no nearer than the distance found.
template <bool kStats>
__device__ __forceinline__ Info union_distance(const DevScene& S, F3 p, Ctx<kStats>& cx) {
  const DevFast& F = S.fast;
  Info best{kInf, ftd::kNoRef};
  int negative = 0;
  bool tie = false;
  auto add = [&](float d, int i) {
    tie = d == best.d || (tie && !(d < best.d));
    if (d < best.d) best = Info{d, ~i};
    negative += d < 0.0f;
  };
  if (F.n_always > 0) add(fast_prim<true>(S, p, cx), 0);
#pragma unroll 1
  for (int i = 1; i < F.n_always; ++i) {  // the same record for every lane
    const float4* w = S.cprims + 3 * i;
    const float4 a = __ldg(w), b = __ldg(w + 1), c = __ldg(w + 2);
    cx.prim();
    add(__float_as_uint(c.w) & ftd::kRareFlag ? rare_distance(S.nodes[__float_as_int(c.z)], p)
                                              : ftd::compact_distance<true>(a, b, c.x, c.y, p),
        i);
  }
  bool walk = false;  // take the leaf-BVH walk
  if (!F.all) {
    int cell = 0;
    if (grid_cell(F.tree.fine, p, &cell) || grid_cell(F.tree.outer, p, &cell)) {
      const uint2 range = __ldg(S.cells + cell);
      walk = range.y == kInsideCell;
      for (uint32_t k = range.x, end = walk ? k : range.x + range.y; k < end; ++k) {
        const uint2 e = __ldg(S.entries + k);
        cx.cand();
        if (__uint_as_float(e.x) >= fmaxf(best.d, 1.17549435e-38f)) break;
        add(compact_at<true>(S, e.y, p, cx), static_cast<int>(e.y & ~ftd::kRareFlag));
      }
    } else {
      cx.box();
      if (sqrtf(ftd::aabb_lb2(p, F.bmin[1], F.bmax[1])) < best.d) {
        bool same;
        const Info far = far_nearest<true>(S, F.tree, p, best, &same, cx);
        tie = same || (tie && far.ref == best.ref);
        best = far;
      }
    }
  }
  if (walk || tie || negative > 1) return scene_distance_bvh(S, p, cx);
  return best;
}

// Scenes without a form of their own: one or two leaves, or the leaf walk.
template <bool kStats>
__device__ __forceinline__ Info general_distance(const DevScene& S, F3 p, Ctx<kStats>& cx) {
  const DevFast& F = S.fast;
  if (F.kind == kFastNone) return scene_distance_bvh(S, p, cx);
  if (F.leaf[0] < 0) return leaves_distance(S, p, 0.0f, 0.0f, cx);
  cx.box(2);
  return leaves_distance(S, p, node_lb(p, F.bmin[0], F.bmax[0]), node_lb(p, F.bmin[1], F.bmax[1]), cx);
}
template <bool kStats>
__device__ __noinline__ Info scene_distance_general(const DevScene& S, F3 p, Ctx<kStats>& cx) {
  return general_distance(S, p, cx);
}

// What a march kernel is compiled for: scenes with a short form, scenes without
// one (general), or any (mixed batches, statistics, paths: there the general
// distance is a call).  In one kernel, the general distance inline made the
// field's depth frame 4 % and a preview 4 to 6 % slower; behind a call, itself
// calling the composite leaf's evaluator, a ground beside one boolean took 10
// to 17 % longer than with its own kernel.
enum Form : int { kFormAny = 0, kFormGeneral = 1, kFormShort = 2 };

// The scene distance at p (Accelerator::distance_info).
template <int kForm = kFormAny, bool kStats>
__device__ __forceinline__ Info scene_distance_inl(const DevScene& S, F3 p, Ctx<kStats>& cx) {
  cx.eval();
  const DevFast& F = S.fast;
  if (kForm == kFormGeneral) return general_distance(S, p, cx);
  if (F.kind == kFastUnion) return union_distance(S, p, cx);
  if (kForm == kFormAny && F.kind <= kFastNone) return scene_distance_general(S, p, cx);
  if (F.entry[0] == kNoPrim) return eval_urtree(S, F.tree, p, kInf, cx);
  cx.box(2);
  const float l2 = ftd::aabb_lb2(p, F.bmin[0], F.bmax[0]), r2 = ftd::aabb_lb2(p, F.bmin[1], F.bmax[1]);
  return F.kind == kFastTree ? tree_and_prim(S, p, r2, l2, cx) : pair_distance(S, p, l2, r2, cx);
}

template <int kForm = kFormAny, bool kStats>
__device__ __noinline__ Info scene_distance(const DevScene& S, F3 p, Ctx<kStats>& cx) {
  return scene_distance_inl<kForm>(S, p, cx);
}

template <int kForm = kFormAny, bool kStats>
__device__ __forceinline__ float scene_d(const DevScene& S, F3 p, Ctx<kStats>& cx) {
  return scene_distance<kForm>(S, p, cx).d;
}

// The same leaf-BVH walk reporting the winning hard-union leaf: the leaf whose
// subtree the reference's Union walks descend into when resolving a hit's
// normal and material (R:4471-4478, R:6995-7002).
template <bool kStats>
__device__ __noinline__ Info scene_distance_leaf(const DevScene& S, F3 p, int* leaf, Ctx<kStats>& cx) {
  cx.eval();
  Info cur{kInf, ftd::kNoRef};
  int nearest = 0;
  const unsigned long long boxes = cx.c.boxes;
  LeafWalk<kStats> walk(S, p, cx);
  for (int li; (li = walk.next(S, cur.d, cx)) >= 0;) {
    const Info in = eval_leaf(S, li, p, cur.d, cx);
    if (in.d < cur.d) {
      cur = in;
      nearest = li;
    }
  }
  cx.c.boxes = boxes;  // (not counted as culls)
  *leaf = nearest;
  return cur;
}

// ray_aabb_intersection (R:4141-4173)
__device__ bool ray_aabb(F3 o, F3 d, const float* mn, const float* mx, float* t0o, float* t1o) {
  float tmin = -kInf, tmax = kInf;
  float os[3] = {o.x, o.y, o.z}, ds[3] = {d.x, d.y, d.z};
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    if (fabsf(ds[k]) <= 1.0e-8f) {
      if (os[k] < mn[k] || os[k] > mx[k]) return false;
      continue;
    }
    float inv = 1.0f / ds[k];
    float t0 = (mn[k] - os[k]) * inv, t1 = (mx[k] - os[k]) * inv;
    if (t0 > t1) {
      float tt = t0;
      t0 = t1;
      t1 = tt;
    }
    tmin = fmaxf(tmin, t0);
    tmax = fminf(tmax, t1);
    if (tmax < tmin) return false;
  }
  *t0o = tmin;
  *t1o = tmax;
  return true;
}

struct HitOut {
  float t;
  uint32_t mat;
  bool hit;
  F3 normal;
};

template <int kForm, bool kStats>
__device__ HitOut march(const DevScene& S, const RayParams& P, F3 o, F3 d, bool want_normal, Ctx<kStats>& cx) {
  HitOut h{0.0f, 0u, false, f3(0.0f, 0.0f, 0.0f)};
  float t0, t1;
  if (!ray_aabb(o, d, S.smin, S.smax, &t0, &t1)) return h;
  float max_t = fminf(P.max_dist, t1);
  float traveled = fmaxf(0.0f, fmaxf(t0, 0.0f));
  float prev = traveled;
  const float eps = P.eps;
  const float scale = ftd::rclamp(P.step_scale, 0.05f, 1.0f);
  const float min_step = fmaxf(eps * 0.5f, 1.0e-5f);
  for (uint32_t s = 0; s < P.max_steps; ++s) {
    if (traveled > max_t) return h;
    cx.step();
    Info info = scene_distance<kForm>(S, o + d * traveled, cx);
    if (fabsf(info.d) < eps) {
      float lo = prev, hi = traveled;
      for (int k = 0; k < 10; ++k) {
        float mid = 0.5f * (lo + hi);
        float dm = fabsf(scene_d<kForm>(S, o + d * mid, cx));
        if (dm < eps) hi = mid;
        else lo = mid;
      }
      F3 pos = o + d * hi;
      if (want_normal) {
        // estimate_normal (R:4202-4215)
        float e = fmaxf(eps * 4.0f, 1.0e-5f);
        float dx = scene_d<kForm>(S, f3(pos.x + e, pos.y, pos.z), cx) - scene_d<kForm>(S, f3(pos.x - e, pos.y, pos.z), cx);
        float dy = scene_d<kForm>(S, f3(pos.x, pos.y + e, pos.z), cx) - scene_d<kForm>(S, f3(pos.x, pos.y - e, pos.z), cx);
        float dz = scene_d<kForm>(S, f3(pos.x, pos.y, pos.z + e), cx) - scene_d<kForm>(S, f3(pos.x, pos.y, pos.z - e), cx);
        F3 nn = f3(dx, dy, dz);
        h.normal = ftd::len3(nn) > 1.0e-8f ? ftd::normalize3(nn) : f3(0.0f, 1.0f, 0.0f);
      }
      Info fin = scene_distance<kForm>(S, pos, cx);
      h.t = hi;
      h.mat = surface_ids(S, fin.ref).y;
      h.hit = true;
      return h;
    }
    prev = traveled;
    traveled += fmaxf(fabsf(info.d) * scale, min_step);
  }
  return h;
}

// Pixel and sample of work item i.  32-bit divisions where the frame allows: a
// 64-bit one is a call of some hundred instructions, in the refill that a warp
// of the persistent marches runs for a few lanes at a time.
__device__ __forceinline__ void item_coords(const RayParams& P, uint64_t i, uint32_t* px, uint32_t* py, uint32_t* s) {
  const uint32_t per_tile = P.tile_w * P.tile_h * P.aa;
  uint32_t k, tx, ty;
  if (P.n_items <= 0xffffffffull) {
    const uint32_t i32 = static_cast<uint32_t>(i), tile = i32 / per_tile;
    k = i32 - tile * per_tile;
    ty = tile / P.tiles_x;
    tx = tile - ty * P.tiles_x;
  } else {
    const uint64_t tile = i / per_tile;
    k = static_cast<uint32_t>(i - tile * per_tile);
    tx = static_cast<uint32_t>(tile % P.tiles_x);
    ty = static_cast<uint32_t>(tile / P.tiles_x);
  }
  *s = k % P.aa;
  const uint32_t j = k / P.aa;
  *px = tx * P.tile_w + j % P.tile_w;
  *py = ty * P.tile_h + j / P.tile_w;
}

#include "ft_bricks.cuh"

// Many renders in one launch: per-item scene, parameters and brick cache, and
// the prefix sums that map a global work item to (item, local work item) and
// an item's outputs into the concatenated output arrays.
struct BatchView {
  const DevScene* scenes;
  const RayParams* params;
  const DevBricks* bricks;
  const uint64_t* ray_first;  // n_items + 1 entries
  const uint64_t* out_first;  // first output sample of each item
  uint32_t n_items;
  uint64_t n_rays;
};

// Item holding global work item `g` (ray_first is sorted; ray_first[0] = 0).
__device__ __forceinline__ uint32_t batch_item(const BatchView& V, uint64_t g) {
  uint32_t lo = 0, hi = V.n_items;  // ray_first[lo] <= g < ray_first[hi]
  while (hi - lo > 1) {
    uint32_t mid = (lo + hi) >> 1;
    if (__ldg(&V.ray_first[mid]) <= g) lo = mid;
    else hi = mid;
  }
  return lo;
}

template <bool kStats, int kForm>
__global__ void __launch_bounds__(128) march_depth_kernel(const __grid_constant__ DevScene S,
                                                          const __grid_constant__ RayParams P, float* __restrict__ t_out,
                                                          uint8_t* __restrict__ mask_out,
                                                          uint32_t* __restrict__ mat_out,
                                                          float* __restrict__ normal_out,
                                                          unsigned long long* __restrict__ stats) {
  uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  Ctx<kStats> cx;
  cx.c = Counters{};
  bool active = i < P.n_items;
  uint32_t px = 0, py = 0, s = 0;
  if (active) {
    item_coords(P, i, &px, &py, &s);
    active = px < P.width && py < P.height;
  }
  if (active) {
    float ndc_x, ndc_y;
    sample_ndc(P, px, py, s, &ndc_x, &ndc_y);
    ndc_x *= P.aspect;
    F3 fwd = f3(P.fwd[0], P.fwd[1], P.fwd[2]), rt = f3(P.right[0], P.right[1], P.right[2]);
    F3 up = f3(P.up[0], P.up[1], P.up[2]);
    F3 dir = ftd::normalize3(fwd + rt * (ndc_x * P.tan_fov) + up * (ndc_y * P.tan_fov));
    dir = ftd::normalize3(dir);
    F3 o = f3(P.origin[0], P.origin[1], P.origin[2]);
    HitOut h = march<kForm>(S, P, o, dir, normal_out != nullptr, cx);
    size_t idx = (static_cast<size_t>(py) * P.width + px) * P.aa + s;
    t_out[idx] = h.hit ? h.t : 0.0f;
    mask_out[idx] = h.hit ? 1 : 0;
    if (mat_out) mat_out[idx] = h.hit ? h.mat : 0u;
    if (normal_out) {
      normal_out[3 * idx] = h.normal.x;
      normal_out[3 * idx + 1] = h.normal.y;
      normal_out[3 * idx + 2] = h.normal.z;
    }
  }
  if (kStats) flush_stats(cx.c, stats);
}

// Primary ray of work item i (pixel_sample_offsets R:4838-4854, NDC map of
// render_depth_tile R:3951-3955, generate_ray render_api.rs:132-144 and the
// second normalisation of the tile loop).
template <bool kYFirst = false>
__device__ __forceinline__ bool item_ray(const RayParams& P, uint64_t i, F3* dir, size_t* out_idx) {
  uint32_t px, py, s;
  item_coords(P, i, &px, &py, &s);
  if (px >= P.width || py >= P.height) return false;
  float ndc_x, ndc_y;
  sample_ndc(P, px, py, s, &ndc_x, &ndc_y);
  ndc_x *= P.aspect;
  F3 fwd = f3(P.fwd[0], P.fwd[1], P.fwd[2]), rt = f3(P.right[0], P.right[1], P.right[2]);
  F3 up = f3(P.up[0], P.up[1], P.up[2]);
  F3 d = ftd::normalize3_fma<false>(fwd + rt * (ndc_x * P.tan_fov) + up * (ndc_y * P.tan_fov));
  *dir = ftd::normalize3_fma<kYFirst>(d);
  *out_idx = (static_cast<size_t>(py) * P.width + px) * P.aa + s;
  return true;
}

// Persistent march with per-lane state machines.
//
// Every loop iteration performs exactly one scene distance evaluation per
// live lane, whatever the lane is doing: a march step (R:4100-4137), one of
// the ten bisection steps (refine_hit_distance, R:4180-4200), one of the six
// estimate_normal taps (R:4202-4215) or the final material lookup.  Lanes
// whose ray finished pick up the next work item from a global counter once
// `refill` lanes of the warp are idle (24 by default: see kWfRefill), so
// divergent march lengths do not leave lanes idle for the rest of the warp's
// life.  The sequence of evaluation points of
// each ray is exactly the reference's.
//
// With kBricks (the FP16 precision form) a ray starts in the far-field phase:
// up to far_batch steps per iteration on the brick lower bound b (one texture
// fetch each), stepping by b - band/2 so the exact distance stays above band/2,
// until b < band or the ray leaves the brick region (each far-field step counts
// as one step against max_steps).  It then continues from that point with the
// plain method's exact FP32 march (same step rule), and goes back to the far
// field whenever an exact step finds
// |d| > band_exit.  A hit found by the exact march takes the plain method's
// ten bisections between its last two samples (the reference's depth); a
// hit reached by the counted descent onto the ground plane, whose bracket
// ends at the plane crossing rather than at a sample, finds the eps-shell
// crossing by secant steps on the exact distance (each verified by an exact
// evaluation).  The normal is the plain method's.
enum Phase : int { kMarch = 0, kRefine = 1, kNormal = 2, kFinal = 3, kFar = 4, kSecant = 5 };
constexpr unsigned long long kMarchWallNs = 20ull * 1000000000ull;  // per warp

//
// With kBatch the launch serves many renders: each lane carries the index of
// the item its ray belongs to and reads that item's scene, parameters and
// brick cache from the batch tables (otherwise they are the kernel's own
// parameters); outputs are the concatenated arrays of all items.
//
// Five resident blocks per SM (96 registers): a small frame is bound by the
// latency of its longest rays' evaluations and a 256x256 preview takes 0.42 ms
// of march against 0.46 with six or eight blocks; the 512-primitive field at
// 1920x1080 takes 12.7, 12.7 and 11.8 ms (refilling at 8 idle lanes).
template <bool kStats, bool kBricks, bool kBatch, int kForm = kFormAny>
__global__ void __launch_bounds__(128, 5) march_depth_persistent(
    const __grid_constant__ DevScene S0, const __grid_constant__ RayParams P0, const __grid_constant__ DevBricks B0,
    const __grid_constant__ BatchView V,
                                                              float* __restrict__ t_out,
                                                              uint8_t* __restrict__ mask_out,
                                                              uint32_t* __restrict__ mat_out,
                                                              float* __restrict__ normal_out,
                                                              unsigned long long* __restrict__ stats,
                                                              unsigned long long* __restrict__ next_item) {
#ifdef FT_JIT
  constexpr bool kRayYFirst = true;
#else
  constexpr bool kRayYFirst = kBricks;
#endif
  const unsigned lane = threadIdx.x & 31u;
  const bool want_normal = normal_out != nullptr;
  const uint64_t n_work = kBatch ? V.n_rays : P0.n_items;
  const unsigned refill = kBatch ? V.params[0].refill : P0.refill;
  Ctx<kStats> cx;
  cx.c = Counters{};

  bool live = false;
  bool queue_done = false;
  size_t idx = 0;
  uint32_t item_of_lane = 0;
  // Self-checks: a ray takes at most max_steps + 17 iterations (one step per
  // march or far-field iteration, then bisection or secant, normal taps and
  // the final lookup), and a warp runs for at most kMarchWallNs.  A lane past
  // either limit records it in next_item[1] (bit per phase; bit 8: time) and
  // gives up, so a fault in the march ends the launch instead of hanging it.
  uint32_t ray_iters = 0;
  uint32_t loop_iters = 0;
  const unsigned long long t_start = __shfl_sync(0xffffffffu, lane == 0 ? ftd::global_ns() : 0ull, 0);
  // per-ray constants (per item with kBatch)
  F3 o = f3(P0.origin[0], P0.origin[1], P0.origin[2]);
  float eps = P0.eps;
  float scale = ftd::rclamp(P0.step_scale, 0.05f, 1.0f);
  float min_step = fmaxf(eps * 0.5f, 1.0e-5f);
  float ne = fmaxf(eps * 4.0f, 1.0e-5f);
  F3 d = f3(0.0f, 0.0f, 0.0f), pos = f3(0.0f, 0.0f, 0.0f);
  float traveled = 0.0f, prev = 0.0f, max_t = 0.0f, lo = 0.0f, hi = 0.0f;
  float nx = 0.0f, ny = 0.0f, nz = 0.0f;  // estimate_normal differences
  uint32_t steps = 0;
  int phase = kMarch, k = 0;
  // precision form: secant bracket values of the counted descent, material
  // of the accepted hit point
  float dlo = 0.0f, dhi = 0.0f;
  uint32_t hit_mat = 0u;
  bool mat_known = false;
  auto write_miss = [&]() {
    live = false;
    t_out[idx] = 0.0f;
    mask_out[idx] = 0;
    if (mat_out) mat_out[idx] = 0u;
    if (normal_out) {
      normal_out[3 * idx] = 0.0f;
      normal_out[3 * idx + 1] = 0.0f;
      normal_out[3 * idx + 2] = 0.0f;
    }
  };
  auto write_hit = [&](uint32_t mat) {
    live = false;
    t_out[idx] = hi;
    mask_out[idx] = 1;
    if (mat_out) mat_out[idx] = mat;
    if (normal_out) {
      F3 nn = f3(nx, ny, nz);
      F3 nr = ftd::len3(nn) > 1.0e-8f ? ftd::normalize3(nn) : f3(0.0f, 1.0f, 0.0f);
      normal_out[3 * idx] = nr.x;
      normal_out[3 * idx + 1] = nr.y;
      normal_out[3 * idx + 2] = nr.z;
    }
  };

  for (;;) {
    if ((++loop_iters & 1023u) == 0u) {
      unsigned long long now = lane == 0 ? ftd::global_ns() : 0ull;
      now = __shfl_sync(0xffffffffu, now, 0);
      if (now - t_start > kMarchWallNs) {
        if (lane == 0) atomicOr(&next_item[1], 1ull << 8);
        break;
      }
    }
    // Refill idle lanes when enough of the warp is idle (or all of it).
    unsigned idle = __ballot_sync(0xffffffffu, !live);
    if (!queue_done && (__popc(idle) >= refill || idle == 0xffffffffu)) {
      unsigned n = __popc(idle);
      unsigned long long base = 0;
      if (lane == 0) base = atomicAdd(next_item, static_cast<unsigned long long>(n));
      base = __shfl_sync(0xffffffffu, base, 0);
      if (base >= n_work) queue_done = true;
      if (!live) {
        unsigned rank = __popc(idle & ((1u << lane) - 1u));
        uint64_t item = base + rank;
        bool got = false;
        if (item < n_work) {
          if (kBatch) {
            item_of_lane = batch_item(V, item);
            const RayParams& Pi = V.params[item_of_lane];
            got = item_ray<kRayYFirst>(Pi, item - V.ray_first[item_of_lane], &d, &idx);
            idx += V.out_first[item_of_lane];
            o = f3(Pi.origin[0], Pi.origin[1], Pi.origin[2]);
            eps = Pi.eps;
            scale = ftd::rclamp(Pi.step_scale, 0.05f, 1.0f);
            min_step = fmaxf(eps * 0.5f, 1.0e-5f);
            ne = fmaxf(eps * 4.0f, 1.0e-5f);
          } else {
            got = item_ray<kRayYFirst>(P0, item, &d, &idx);
          }
        }
        const DevScene& S = kBatch ? V.scenes[item_of_lane] : S0;
        const RayParams& P = kBatch ? V.params[item_of_lane] : P0;
        const DevBricks& B_of_lane = kBatch ? V.bricks[item_of_lane] : B0;
        (void)B_of_lane;
        if (got) {
          float t0, t1;
          bool inside = ray_aabb(o, d, S.smin, S.smax, &t0, &t1);
          traveled = fmaxf(0.0f, fmaxf(t0, 0.0f));
          max_t = fminf(P.max_dist, t1);
          if (inside && P.max_steps > 0 && !(traveled > max_t)) {
            live = true;
            ray_iters = 0;
            prev = traveled;
            steps = 0;
            phase = kBricks && B_of_lane.free_far ? kFar : kMarch;
            mat_known = false;
          } else {
            write_miss();
          }
        }
      }
    }
    if (__ballot_sync(0xffffffffu, live) == 0u) {
      if (queue_done) break;
      continue;
    }
    if (!live) continue;
    const DevScene& S = kBatch ? V.scenes[item_of_lane] : S0;
    const RayParams& P = kBatch ? V.params[item_of_lane] : P0;
    const DevBricks& B = kBatch ? V.bricks[item_of_lane] : B0;
    if (++ray_iters > P.max_steps + 64u) {
      atomicOr(&next_item[1], 1ull << (phase & 7));
      write_miss();
      continue;
    }

    if (kBricks && phase == kFar) {
      bool exact = false, missed = false;
      for (int f = 0; f < B.far_batch; ++f) {
        float b;
        if (!far_bound(S, B, o + d * traveled, &b, cx) || b < B.band) {
          exact = true;
          break;
        }
        traveled += b - 0.5f * B.band;
        cx.far_step();
        ++steps;  // a far-field step is one step of the march
        if (steps >= P.max_steps || traveled > max_t) {
          missed = true;
          break;
        }
      }
      if (missed) {
        write_miss();
        continue;
      }
      if (!exact) continue;
      phase = kMarch;  // exact evaluation at `traveled` in this iteration
      prev = traveled;
    }

    // The point this lane evaluates in this iteration.
    F3 q;
    float mid = 0.0f;
    if (phase == kMarch) {
      q = o + d * traveled;
      cx.step();
    } else if (phase == kRefine) {
      mid = 0.5f * (lo + hi);
      q = o + d * mid;
    } else if (kBricks && phase == kSecant) {
      // crossing of d = eps on the line through (lo, dlo) and (hi, dhi),
      // aimed 1/64 eps inside the shell so rounding keeps it there
      const float target = eps * (1.0f - 1.0f / 64.0f);
      mid = lo + (dlo - target) / (dlo - dhi) * (hi - lo);
      mid = fminf(fmaxf(mid, lo), hi);
      q = o + d * mid;
    } else if (phase == kNormal) {
      float sgn = (k & 1) ? -ne : ne;
      q = pos;
      if (k < 2) q.x += sgn;
      else if (k < 4) q.y += sgn;
      else q.z += sgn;
    } else {
      q = pos;
    }
    Info info = scene_distance_inl<kForm>(S, q, cx);

    if (phase == kMarch) {
      if (fabsf(info.d) < eps) {
        // the plain method's ten bisections between the last two samples: the
        // reference's depth (the eps-shell crossing found by bisection)
        lo = prev;
        hi = traveled;
        k = 0;
        phase = kRefine;
      } else {
        // the nearest leaf is the ground and the ray descends: the cached
        // bound decides whether the rest of the approach is a plane descent
        if (kBricks && !B.free_far && B.plane_leaf >= 0 && d.y < 0.0f && surface_ids(S, info.ref).x == B.plane_obj &&
            plane_jump(B, q, d, info.d, cached_lb(B, q, cx), eps, scale, min_step)) {
          // The rest of the plain march descends on the plane: after n more
          // steps it first samples inside the eps shell (heights shrink by
          // 1 - scale*s per step).  Same outcome as the plain march: a miss
          // when it would run out of steps or distance on the way.
          const float sdn = -d.y;
          const float g = info.d;
          float along = 0.0f;
          const int n = plane_descent_steps(g, sdn, scale, eps, &along);
          cx.far_step();
          if (n < 0 || static_cast<uint64_t>(steps) + static_cast<uint64_t>(n) >= P.max_steps ||
              traveled + along > max_t) {
            write_miss();
            continue;
          }
          // bracket: here (distance g) and the plane crossing (distance 0)
          lo = traveled;
          dlo = g;
          hi = traveled + g / sdn;
          dhi = 0.0f;
          k = 0;
          phase = kSecant;
          mat_known = false;  // hi is not a verified sample: the material comes from an evaluation
          continue;
        }
        prev = traveled;
        traveled += fmaxf(fabsf(info.d) * scale, min_step);
        ++steps;
        if (kBricks && B.free_far && fabsf(info.d) > B.band_exit) phase = kFar;
        if (steps >= P.max_steps || traveled > max_t) write_miss();
      }
    } else if (kBricks && phase == kSecant) {
      bool accept = true;
      if (fabsf(info.d) < eps) {
        hi = mid;
        hit_mat = surface_ids(S, info.ref).y;
        mat_known = true;
      } else if (info.d > 0.0f && ++k < 3) {
        lo = mid;
        dlo = info.d;
        accept = false;
      }
      if (accept) {
        pos = o + d * hi;
        k = 0;
        if (want_normal) phase = kNormal;
        else if (mat_known) write_hit(hit_mat);
        else phase = kFinal;
      }
    } else if (phase == kRefine) {
      if (fabsf(info.d) < eps) hi = mid;
      else lo = mid;
      if (++k == 10) {
        pos = o + d * hi;
        phase = want_normal ? kNormal : kFinal;
        k = 0;
      }
    } else if (phase == kNormal) {
      // dx = d(p + e x) - d(p - e x), one subtraction as in the reference
      if (k == 0) nx = info.d;
      else if (k == 1) nx = nx - info.d;
      else if (k == 2) ny = info.d;
      else if (k == 3) ny = ny - info.d;
      else if (k == 4) nz = info.d;
      else nz = nz - info.d;
      if (++k == 6) {
        if (kBricks && mat_known) write_hit(hit_mat);
        else phase = kFinal;
      }
    } else {
      write_hit(surface_ids(S, info.ref).y);
    }
  }
  if (kStats) flush_stats(cx.c, stats);
}

#ifndef FT_JIT
// Depth preview pixels (render_depth_tile R:3931-3971, depth_preview_value
// R:5215-5219, spectrum_to_rgb8 R:5221-5227).
__device__ __forceinline__ float depth_pixel_value(const float* __restrict__ t, const uint8_t* __restrict__ mask,
                                                   size_t first, uint32_t aa, float max_dist) {
  float sum = 0.0f;
  float md = fmaxf(max_dist, 1.0e-6f);
  for (uint32_t s = 0; s < aa; ++s) {
    size_t k = first + s;
    float depth = 0.0f;
    if (mask[k]) {
      float d = ftd::rclamp(t[k] / md, 0.0f, 1.0f);
      float shaped = 1.0f - d;
      depth = shaped * shaped;
    }
    sum += depth;
  }
  return sum * (1.0f / static_cast<float>(aa));
}

// spectrum_to_rgb8 (R:5221-5227): gamma 2.2, clamped, truncated
__device__ __forceinline__ uint8_t gamma_u8(float v) {
  float mapped = fminf(powf(fmaxf(v, 0.0f), 1.0f / 2.2f), 1.0f);
  return static_cast<uint8_t>(mapped * 255.0f);
}

// spectrum_to_rgb8_reinhard (R:5229-5239)
__device__ __forceinline__ uint8_t reinhard_u8(float v) {
  float x = fmaxf(v, 0.0f);
  float t = x / (1.0f + x);
  float mapped = fminf(powf(t, 1.0f / 2.2f), 1.0f);
  return static_cast<uint8_t>(mapped * 255.0f);
}

__global__ void depth_rgb8_kernel(const float* __restrict__ t, const uint8_t* __restrict__ mask, uint32_t n_pixels,
                                  uint32_t aa, float max_dist, uint8_t* __restrict__ rgb) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_pixels) return;
  uint8_t g = gamma_u8(depth_pixel_value(t, mask, static_cast<size_t>(i) * aa, aa, max_dist));
  rgb[3 * static_cast<size_t>(i)] = g;
  rgb[3 * static_cast<size_t>(i) + 1] = g;
  rgb[3 * static_cast<size_t>(i) + 2] = g;
}

#endif  // FT_JIT

#include "ft_trace.cuh"

struct TraceHit {
  float t;
  F3 pos, normal;
  uint32_t mat, obj;  // the hit's material and object ids (RayHit, R:440-452)
  int leaf;
};

// environment_color (R:4328-4333), falling back to the sum of EnvLight
// radiances (env_radiance, R:4318-4326).
__device__ F3 environment(const DevScene& S, F3 dir) {
  if (S.env_program >= 0) return scene_program(S, S.env_program, &dir, nullptr);
  F3 s = f3(0.0f, 0.0f, 0.0f);
  for (int i = 0; i < S.n_lights; ++i)
    if (S.lights[i].kind == FT_LIGHT_ENV) s = s + f3(S.lights[i].intensity[0], S.lights[i].intensity[1], S.lights[i].intensity[2]);
  return s;
}

// Shading of one hit (trace_hit_with_material, ray.rs:41-222, for each
// material of the hit, ray.rs:31-35): the radiance it adds, its light samples
// and its secondary rays, reported to `sink`:
//   sink.emit(rgb)                          radiance added at this hit,
//   sink.light(contrib, origin, dir, max_t) a light sample whose contribution
//                                           is contrib x shadow_visibility,
//   sink.push(job)                          a reflected or refracted ray.
// shade_color (R:4217-4276) is distributed over the light samples:
// W (sum_s f rad ndotl vis inv) local_w = sum_s W f rad ndotl inv local_w vis.
template <bool kStats, class Sink>
__device__ __forceinline__ void shade_hit(const DevScene& S, const RayParams& P, const RayJob& J, const TraceHit& h,
                                          Sink& sink, Ctx<kStats>& cx) {
  const float eps = P.eps;
  bool front = ftd::dot3(h.normal, J.d) < 0.0f;
  F3 normal = front ? ftd::normalize3(h.normal) : ftd::normalize3(h.normal * -1.0f);
  const HookCtx hc{h.pos, normal, ftd::normalize3(J.d * -1.0f), front ? 1.0f : 0.0f};
  Resolved rs;
  resolve_hit(S, h.leaf, h.pos, hc, &rs, cx);
  F3 shading_n = normal;
  if (rs.ok) shading_n = ftd::normalize3(front ? rs.normal : rs.normal * -1.0f);
  // build_bsdf_context (R:4397-4449): the shading normal through the hit
  // material's bump and normal hooks, and the context of the BSDF hooks
  BsdfCtx bc;
  bc.pos = h.pos;
  bc.local = object_local(S, h.obj, h.pos);
  bc.normal = shading_n;
  bc.wo = ftd::normalize3(J.d * -1.0f);
  bc.front = front ? 1.0f : 0.0f;
  bc.obj = static_cast<float>(h.obj);
  bc.mat = static_cast<float>(h.mat);
  bc.current_ior = J.med.ior;
  shading_n = hooked_shading_normal(S, bc, J.d * -1.0f, h.mat);
  bc.normal = shading_n;
  // The hit's materials are read where resolve_hit left them (no copies).
  const DMat* mats[2];
  float ws[2];
  int nm = 0;
  if (rs.ok && rs.split) {
    float tt = clamp01(rs.t);  // lerp_spectrum(a, b, t): a (1 - t) + b t
    if (tt != 1.0f) { mats[nm] = &rs.m; ws[nm++] = 1.0f - tt; }
    if (tt != 0.0f) { mats[nm] = rs.mb_same ? &rs.m : &rs.mb; ws[nm++] = tt; }
  } else {
    if (!rs.ok) rs.m = mat_of_id(S, h.mat);
    mats[0] = &rs.m;
    ws[0] = 1.0f;
    nm = 1;
  }
  F3 att = transmittance(J.med, h.t);
  F3 wo = ftd::normalize3(J.d * -1.0f);
  for (int mi = 0; mi < nm; ++mi) {
    const DMat& mat = *mats[mi];
    F3 W = mul3(J.w * ws[mi], att);
    const DParams& Pm = dom_params(mat);
    float rough = clamp01(Pm.roughness);
    int model = dom_model(mat);
    float transmission, ior, metallic, clearcoat, specular_strength;
    bool thin;
    F3 spec_color, base_color;
    if (model == FT_MAT_STANDARD) {
      transmission = clamp01(Pm.transmission); ior = ftd::rclamp(Pm.ior, 1.0f, 3.0f); thin = Pm.thin != 0;
      spec_color = Pm.spec_color; base_color = Pm.color; metallic = clamp01(Pm.metallic);
      clearcoat = clamp01(Pm.clearcoat); specular_strength = clamp01(Pm.specular * Pm.specular_weight);
    } else if (model == FT_MAT_LAMBERT) {
      transmission = 0.0f; ior = 1.0f; thin = false; spec_color = f3(0.0f, 0.0f, 0.0f); base_color = Pm.color;
      metallic = 0.0f; clearcoat = 0.0f; specular_strength = 0.0f;
    } else if (model == FT_MAT_METAL) {
      transmission = 0.0f; ior = 1.0f; thin = false; spec_color = Pm.color; base_color = Pm.color;
      metallic = 1.0f; clearcoat = 0.0f; specular_strength = 1.0f;
    } else {
      transmission = 1.0f; ior = ftd::rclamp(Pm.ior, 1.0f, 3.0f); thin = Pm.thin != 0;
      spec_color = f3(1.0f, 1.0f, 1.0f); base_color = Pm.color; metallic = 0.0f; clearcoat = 0.0f;
      specular_strength = 1.0f;
    }
    float eta_i, eta_t, next_ior;
    if (thin) { eta_i = 1.0f; eta_t = 1.0f; next_ior = J.med.ior; }
    else if (front) { eta_i = J.med.ior; eta_t = ior; next_ior = ior; }
    else { eta_i = J.med.ior; eta_t = 1.0f; next_ior = 1.0f; }
    float cosv = fabsf(ftd::dot3(normal, wo));
    float fresnel;
    if (transmission > 1.0e-4f) {
      fresnel = fresnel_dielectric(cosv, eta_i, eta_t);
    } else {
      float f0 = clamp01(f0_from_ior(ior));
      float x = 1.0f - clamp01(cosv);
      float m5 = x * x * x * x * x;
      fresnel = clamp01(f0 + (1.0f - f0) * m5);
    }
    float reflect_w;
    if (transmission > 1.0e-4f) {
      reflect_w = clamp01(fresnel);
    } else {
      float base = metallic > 0.5f ? 1.0f : clamp01(specular_strength);
      reflect_w = clamp01(base * fresnel + metallic * 0.8f + clearcoat * 0.2f);
    }
    float local_w = clamp01((1.0f - transmission) * (1.0f - reflect_w));
    // shade_color (R:4217-4276), light by light
    if (S.n_lights == 0) {
      sink.emit(W * local_w);
    } else {
      F3 n = ftd::normalize3(shading_n);
      for (int li = 0; li < S.n_lights; ++li) {
        const ft_light& L = S.lights[li];
        uint32_t samples = L.kind == FT_LIGHT_SPHERE ? (L.samples > 0 ? L.samples : 1u) : 1u;
        float inv = 1.0f / static_cast<float>(samples);
        for (uint32_t smp = 0; smp < samples; ++smp) {
          F3 wi, rad;
          float dist;
          sample_light(L, h.pos, smp, samples, &wi, &rad, &dist);
          wi = ftd::normalize3(wi);
          float ndotl = n.x * wi.x + n.y * wi.y + n.z * wi.z;
          if (ndotl <= 0.0f) continue;
          F3 so = offset_origin(h.pos, normal, wi, eps);
          float max_t = isfinite(dist) ? fmaxf(dist - eps * 8.0f, 0.0f) : P.max_dist;
          if (max_t <= 0.0f) continue;
          F3 f = bsdf_eval(S, mat, bc, wi);
          sink.light(mul3(W, mul3(f, rad) * (ndotl * inv * local_w)), so, wi, max_t);
        }
      }
    }
    sink.emit(mul3(W, mat_emission(mat)));
    if (reflect_w > 1.0e-4f) {
      F3 rd = ftd::normalize3(J.d - normal * (2.0f * ftd::dot3(J.d, normal)));
      F3 tint = lerp_sp(spec_color, base_color, clamp01(metallic));
      if (transmission > 1.0e-4f && rough > 0.06f) {
        // trace_rough_dielectric_reflection (ray.rs:296-322): the average of
        // the lobe around the mirror direction
        F3 dirs[kMaxLobes];
        const int n = rough_lobe_directions(rd, rough, rough_reflection_samples(rough), dirs);
        const F3 w = mul3(W, tint * (reflect_w / static_cast<float>(n)));
        for (int k = 0; k < n; ++k)
          sink.push(RayJob{offset_origin(h.pos, normal, dirs[k], eps * (8.0f + rough * 12.0f)), dirs[k], w, J.med,
                           J.depth + 1});
      } else {
        F3 ro = offset_origin(h.pos, normal, rd, eps * (1.0f + rough * 6.0f));
        sink.push(RayJob{ro, rd, mul3(W, tint * reflect_w), J.med, J.depth + 1});
      }
    }
    if (transmission > 1.0e-4f) {
      MediumD next = thin ? J.med : transition(mat, front, J.med);
      next.ior = ftd::rclamp(next_ior, 1.0f, 3.0f);
      F3 td;
      if (refract_dir(J.d, normal, eta_i / eta_t, &td)) {
        float tt = clamp01(transmission);
        F3 tint = f3(1.0f - (1.0f - clamp01(base_color.x)) * tt, 1.0f - (1.0f - clamp01(base_color.y)) * tt,
                     1.0f - (1.0f - clamp01(base_color.z)) * tt);
        const F3 wt = mul3(W, tint * (transmission * (1.0f - fresnel)));
        if (rough > 0.06f) {
          // trace_rough_dielectric_refraction (ray.rs:324-352)
          F3 dirs[kMaxLobes];
          const int n = rough_lobe_directions(ftd::normalize3(td), rough, rough_refraction_samples(rough), dirs);
          const F3 w = wt * (1.0f / static_cast<float>(n));
          for (int k = 0; k < n; ++k)
            sink.push(RayJob{offset_origin(h.pos, normal, dirs[k], eps * (8.0f + rough * 12.0f)), dirs[k], w, next,
                             J.depth + 1});
        } else {
          F3 to = offset_origin(h.pos, normal, td, eps * (8.0f + rough * 12.0f));
          sink.push(RayJob{to, ftd::normalize3(td), wt, next, J.depth + 1});
        }
      }
    }
  }
}

#include "ft_wavefront.cuh"

#ifndef FT_JIT  // batch, pixel, adjoint and measurement kernels: precompiled only
// AA average per pixel and spectrum_to_rgb8_reinhard (R:3908-3921, R:5229-5239).
__global__ void trace_pixels_kernel(const float* __restrict__ sample_rgb, uint32_t n_pixels, uint32_t aa,
                                    float* __restrict__ rgb_out, uint8_t* __restrict__ rgb8_out) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_pixels) return;
  float s[3] = {0.0f, 0.0f, 0.0f};
  for (uint32_t k = 0; k < aa; ++k)
    for (int c = 0; c < 3; ++c) s[c] += sample_rgb[(static_cast<size_t>(i) * aa + k) * 3 + c];
  float inv = 1.0f / static_cast<float>(aa);
  for (int c = 0; c < 3; ++c) {
    float v = s[c] * inv;
    if (rgb_out) rgb_out[3 * static_cast<size_t>(i) + c] = v;
    if (rgb8_out) rgb8_out[3 * static_cast<size_t>(i) + c] = reinhard_u8(v);
  }
}

// Pixels of a batch: each item's depth preview or AA-averaged trace in the
// concatenated image arrays (rgb holds the linear value: the preview value of
// depth items, the averaged radiance of traces).
struct BatchPixItem {
  uint64_t pix_first;  // first pixel of the item in the image arrays
  uint64_t out_first;  // first sample in the depth (t, mask) or trace sample arrays
  uint32_t aa, kind;   // kind 0: depth preview, 1: trace
  float max_dist;
  uint32_t pad;
};

__global__ void batch_pixels_kernel(const BatchPixItem* __restrict__ items, uint32_t n_items, uint64_t n_pixels,
                                    const float* __restrict__ t, const uint8_t* __restrict__ mask,
                                    const float* __restrict__ sample_rgb, float* __restrict__ rgb_out,
                                    uint8_t* __restrict__ rgb8_out) {
  for (uint64_t g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; g < n_pixels;
       g += (uint64_t)gridDim.x * blockDim.x) {
    uint32_t lo = 0, hi = n_items;
    while (hi - lo > 1) {
      uint32_t mid = (lo + hi) >> 1;
      if (items[mid].pix_first <= g) lo = mid;
      else hi = mid;
    }
    const BatchPixItem& it = items[lo];
    uint64_t local = g - it.pix_first;
    size_t first = it.out_first + local * it.aa;
    if (it.kind == 0) {
      float v = depth_pixel_value(t, mask, first, it.aa, it.max_dist);
      uint8_t c8 = gamma_u8(v);
      for (int c = 0; c < 3; ++c) {
        rgb_out[3 * g + c] = v;
        rgb8_out[3 * g + c] = c8;
      }
    } else {
      float s[3] = {0.0f, 0.0f, 0.0f};
      for (uint32_t k = 0; k < it.aa; ++k)
        for (int c = 0; c < 3; ++c) s[c] += sample_rgb[(first + k) * 3 + c];
      float inv = 1.0f / static_cast<float>(it.aa);
      for (int c = 0; c < 3; ++c) {
        float v = s[c] * inv;
        rgb_out[3 * g + c] = v;
        rgb8_out[3 * g + c] = reinhard_u8(v);
      }
    }
  }
}

#include "ft_diff.cuh"
#include "ft_grid.cuh"

// Dependent-FMA chains, 8 per thread, for the FP32 roofline denominator.
__global__ void fma_peak_kernel(float* out, int iters, float a, float b) {
  float x0 = threadIdx.x * 1e-3f, x1 = x0 + 1, x2 = x0 + 2, x3 = x0 + 3, x4 = x0 + 4, x5 = x0 + 5, x6 = x0 + 6,
        x7 = x0 + 7;
  for (int i = 0; i < iters; ++i) {
    x0 = fmaf(x0, a, b); x1 = fmaf(x1, a, b); x2 = fmaf(x2, a, b); x3 = fmaf(x3, a, b);
    x4 = fmaf(x4, a, b); x5 = fmaf(x5, a, b); x6 = fmaf(x6, a, b); x7 = fmaf(x7, a, b);
  }
  float s = x0 + x1 + x2 + x3 + x4 + x5 + x6 + x7;
  if (s == 12345.678f) out[0] = s;
}

#include "ft_path.cuh"

#endif  // FT_JIT

}  // namespace
