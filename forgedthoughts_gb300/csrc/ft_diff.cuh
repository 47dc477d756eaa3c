// Differentiation form: multi-view depth + soft silhouette and the adjoint
// march (ft_render_views / ft_render_backward).  No counterpart in the
// reference.  Definitions, shared with the FP64 CPU restatement:
//
//   forward, per ray: the plain march (step rule, eps hit, ten bisections);
//   on a hit the depth is the zero of f(o + t d), three secant steps from the
//   bisection bracket; on a miss m = the local minimum of f along the ray
//   next to the smallest march sample (its bracket continued past either end
//   of the samples while f falls, then a 40-step golden-section search), and
//   silhouette = exp(-max(m, 0) / tau) (1 on a hit).
//
//   backward: the march is recomputed (nothing per step is stored); at the
//   hit point  d depth / d theta = -(df/dtheta) / (grad_p f . d), at the
//   miss minimum  d sil / d theta = -(sil / tau) df/dtheta  (its position
//   is stationary along the ray, and is polished by secant steps on
//   grad_p f . d = 0 before the derivative is taken); df/dtheta comes from a full fold of the
//   winning union_round tree with reverse-mode derivatives of op_union_round
//   and of the sphere / box distances.  Per-parameter sums across pixels are
//   FP64: shared-memory accumulators per block, one global atomic per block
//   and parameter.
//
// Included by ft_render.cu inside its anonymous namespace.
#pragma once

constexpr int kMaxDiffPrims = 512;  // union_round trees the adjoint folds (primitives)
constexpr int kGoldenSteps = 40;
constexpr int kSecantSteps = 3;
constexpr int kMinPolishSteps = 4;  // secant steps on df/dt at the silhouette minimum (backward)

struct DiffTables {
  const int32_t* slot;         // node * 8 + field -> parameter index, -1 if none
  const int32_t* tree_radius;  // per union_round tree: radius parameter index, -1 if none
  uint32_t n_params;
};

// A ray of the forward definitions as a state machine: every state asks for
// the scene distance at one t of the ray and next(f) takes it, so a warp's
// lanes share one evaluation site whatever their rays are doing.
struct ViewRay {
  enum State : int { kMarch, kRefine, kSecLo, kSecHi, kSecant, kAhead, kBack, kGolden, kHit, kMiss, kEmpty };
  int state = kEmpty, k = 0;
  uint32_t steps = 0;
  float t = 0.0f;  // the distance is asked for here
  // march: prev and the smallest sample's neighbours; hit: bracket lo, hi with
  // values fa, fb; miss: bracket a < x < b with fx at x
  float prev = 0.0f, best = kInf, lo = 0.0f, x = 0.0f, hi = 0.0f, fa = 0.0f, fb = 0.0f;
  bool need_next = false;

  __device__ __forceinline__ bool live() const { return state < kHit; }
  __device__ __forceinline__ static float step_of(const RayParams& P, float f) {
    return fmaxf(fabsf(f) * ftd::rclamp(P.step_scale, 0.05f, 1.0f), fmaxf(P.eps * 0.5f, 1.0e-5f));
  }
  // End of the march without a hit: the local minimum next to the smallest
  // sample (best at x, neighbours lo and hi), bracketed first.
  __device__ __forceinline__ void miss(const RayParams& P) {
    if (!(best < kInf)) {
      state = kEmpty;
      return;
    }
    if (need_next) hi = x + step_of(P, best);
    k = 0;
    state = kAhead;
    t = hi;
  }
  __device__ __forceinline__ void start(const RayParams& P, float t0, float max_t) {
    t = prev = fmaxf(t0, 0.0f);
    lo = x = hi = t;
    state = kMarch;
    if (P.max_steps == 0 || t > max_t) miss(P);
  }
  // Continue the descent past the low end of the bracket while f falls.
  __device__ __forceinline__ void back(const RayParams& P) {
    if (!(lo < x)) lo = fmaxf(x - step_of(P, best), 0.0f);
    k = 0;
    state = kBack;
    t = lo;
  }
  __device__ __forceinline__ void golden() {
    if (k == kGoldenSteps) {
      state = kMiss;
      return;
    }
    t = (hi - x > x - lo) ? x + 0.3819660112501051f * (hi - x) : x - 0.3819660112501051f * (x - lo);
  }
  __device__ __forceinline__ void secant() {
    if (k == kSecantSteps || fb == fa) {
      state = kHit;
      return;
    }
    const float tn = hi - fb * (hi - lo) / (fb - fa);
    lo = hi;
    fa = fb;
    t = hi = tn;
  }
  __device__ __forceinline__ void next(const RayParams& P, float max_t, float f) {
    switch (state) {
      case kMarch:
        if (need_next) {
          hi = t;
          need_next = false;
        }
        if (f < best) {
          best = f;
          lo = prev;
          x = t;
          hi = t;
          need_next = true;
        }
        if (fabsf(f) < P.eps) {
          lo = prev;
          hi = t;
          k = 0;
          state = kRefine;
          t = 0.5f * (lo + hi);
          break;
        }
        prev = t;
        t += step_of(P, f);
        if (++steps >= P.max_steps || t > max_t) miss(P);
        break;
      case kRefine:
        if (fabsf(f) < P.eps) hi = t;
        else lo = t;
        if (++k < 10) {
          t = 0.5f * (lo + hi);
        } else {
          state = kSecLo;
          t = lo;
        }
        break;
      case kSecLo:
        fa = f;
        state = kSecHi;
        t = hi;
        break;
      case kSecHi:
        fb = f;
        k = 0;
        state = kSecant;
        secant();
        break;
      case kSecant:
        fb = f;
        ++k;
        secant();
        break;
      case kAhead:
        if (k < 64 && f < best && hi < P.max_dist) {
          ++k;
          lo = x;
          x = hi;
          best = f;
          t = hi = x + step_of(P, best);
        } else {
          back(P);
        }
        break;
      case kBack:
        if (k < 64 && f < best && lo > 0.0f) {
          ++k;
          hi = x;
          x = lo;
          best = f;
          t = lo = fmaxf(x - step_of(P, best), 0.0f);
        } else {
          k = 0;
          state = kGolden;
          golden();
        }
        break;
      default:  // kGolden
        if (f < best) {
          if (t > x) lo = x;
          else hi = x;
          x = t;
          best = f;
        } else {
          if (t > x) hi = t;
          else lo = t;
        }
        ++k;
        golden();
    }
  }
  __device__ __forceinline__ float silhouette(float tau) const {
    return state == kHit ? 1.0f : (state == kMiss ? expf(-fmaxf(best, 0.0f) / tau) : 0.0f);
  }
};

// A ray whose gradient the adjoint takes: its index, the hit's or minimum's
// t, the weight of its depth or silhouette, and its silhouette (misses).
struct AdjointRay {
  unsigned long long ray;
  float t, w, sil, pad;
};

// Counters of a views pass: work items taken, self-check flags, hit and miss
// records.
constexpr int kViewCounters = 4;

// Gradient sink: parameter partials scaled by `scale` into FP64 accumulators
// (shared memory when the block holds one per parameter), and grad_p f.
struct GradSink {
  double* acc;      // shared or global
  const DiffTables* T;
  float scale;      // multiplies every parameter partial (0: gradient in p only)
  F3 gp;
  __device__ void add(int node, int field, float v) {
    if (scale == 0.0f) return;
    int k = __ldg(&T->slot[node * 8 + field]);
    if (k >= 0) atomicAdd(&acc[k], static_cast<double>(scale * v));
  }
};

// Reverse-mode derivative of one sphere / box primitive (no x / z rotation,
// rounding or shell: the parameter layout guarantees it).
__device__ void prim_backprop(const DevNode& n, int node, F3 p, float adj, GradSink& g) {
  F3 dpc = f3(p.x - n.c[0], p.y - n.c[1], p.z - n.c[2]);
  // DevNode keeps sin / cos of -rot.y
  const float c = n.has_rot ? n.cy : 1.0f, s = n.has_rot ? n.sy : 0.0f;
  F3 q = f3(c * dpc.x + s * dpc.z, dpc.y, -s * dpc.x + c * dpc.z);
  F3 dq;
  if (n.kind == FT_NODE_SPHERE) {
    float l = ftd::len3(q);
    dq = l > 0.0f ? q * (1.0f / l) : f3(0.0f, 0.0f, 0.0f);
    g.add(node, FT_PARAM_S0, -adj);
  } else {
    float qv[3] = {q.x, q.y, q.z}, qa[3], o[3];
    for (int i = 0; i < 3; ++i) {
      qa[i] = fabsf(qv[i]) - n.f[i];
      o[i] = fmaxf(qa[i], 0.0f);
    }
    float outside = sqrtf(o[0] * o[0] + o[1] * o[1] + o[2] * o[2]);
    float dqa[3] = {0.0f, 0.0f, 0.0f};
    if (outside > 0.0f) {
      for (int i = 0; i < 3; ++i) dqa[i] = o[i] / outside;
    } else {
      int m = 0;
      for (int i = 1; i < 3; ++i)
        if (qa[i] > qa[m]) m = i;
      dqa[m] = 1.0f;
    }
    dq = f3(qv[0] < 0.0f ? -dqa[0] : dqa[0], qv[1] < 0.0f ? -dqa[1] : dqa[1], qv[2] < 0.0f ? -dqa[2] : dqa[2]);
    g.add(node, FT_PARAM_S0, -adj * dqa[0]);
    g.add(node, FT_PARAM_S1, -adj * dqa[1]);
    g.add(node, FT_PARAM_S2, -adj * dqa[2]);
  }
  F3 dp = f3(c * dq.x - s * dq.z, dq.y, s * dq.x + c * dq.z);
  g.gp = g.gp + dp * adj;
  g.add(node, FT_PARAM_CX, -adj * dp.x);
  g.add(node, FT_PARAM_CY, -adj * dp.y);
  g.add(node, FT_PARAM_CZ, -adj * dp.z);
  g.add(node, FT_PARAM_ROT_Y, adj * (dq.x * q.z - dq.z * q.x) * (-3.14159265358979323846f / 180.0f));
}

// op_union_round partials (value = max(r, min(a, b)) - |max(r - (a, b), 0)|).
__device__ __forceinline__ void union_round_partials(float a, float b, float r, float* pa, float* pb, float* pr) {
  float ux = fmaxf(r - a, 0.0f), uy = fmaxf(r - b, 0.0f);
  float l = sqrtf(ux * ux + uy * uy);
  if (l > 0.0f) {
    *pa = ux / l;
    *pb = uy / l;
    *pr = 1.0f - (ux + uy) / l;
  } else {
    *pa = a < b ? 1.0f : 0.0f;
    *pb = a < b ? 0.0f : 1.0f;
    *pr = 0.0f;
  }
}

// Full fold of union_round tree `ti` at p with reverse-mode derivatives.
// `vals` holds the two child values of every inner node (2 * (n - 1)).  Out of
// line: only trees without candidate grids and points with more near
// primitives than urtree_backprop keeps come here.
// Returns false for trees the adjoint does not handle.
__device__ __noinline__ bool urtree_backprop_full(const DevScene& S, int ti, F3 p, const DiffTables& T, GradSink& g) {
  const DevUrTree& t = S.urtrees[ti];
  float vals[2 * (kMaxDiffPrims - 1)];
  float adjs[kMaxDiffPrims - 1];
  const int n_inner = t.n_prims - 1;
  if (t.n_prims > kMaxDiffPrims || n_inner < 1) return false;
  const int base = t.inner_root;
  const float r0 = t.r;
  const float r = fmaxf(fabsf(r0), 1.0e-6f);
  auto prim_value = [&](int pos) {
    const DevNode& pn = S.nodes[S.ur_prims[t.prim_first + pos]];
    return ftd::prim_distance(pn, p);
  };
  // Pre-order numbering: children of inner i have larger indices, so a
  // reverse sweep evaluates every inner node after its children.
  for (int i = n_inner - 1; i >= 0; --i) {
    const DevUrInner& in = S.ur_inner[base + i];
    for (int c = 0; c < 2; ++c) {
      int ch = in.child[c];
      float v;
      if (ch < 0) {
        v = prim_value(-ch - 1);
      } else {
        const float a = vals[2 * (ch - base)], b = vals[2 * (ch - base) + 1];
        v = ftd::op_union_round(a, b, r0);
      }
      vals[2 * i + c] = v;
    }
  }
  for (int i = 0; i < n_inner; ++i) adjs[i] = 0.0f;
  adjs[0] = 1.0f;
  float dr = 0.0f;
  for (int i = 0; i < n_inner; ++i) {
    float ai = adjs[i];
    if (ai == 0.0f) continue;
    float pa, pb, pr;
    union_round_partials(vals[2 * i], vals[2 * i + 1], r, &pa, &pb, &pr);
    dr += ai * pr;
    const DevUrInner& in = S.ur_inner[base + i];
    float pc[2] = {pa, pb};
    for (int c = 0; c < 2; ++c) {
      if (pc[c] == 0.0f) continue;
      int ch = in.child[c];
      if (ch < 0) {
        int node = S.ur_prims[t.prim_first + (-ch - 1)];
        prim_backprop(S.nodes[node], node, p, ai * pc[c], g);
      } else {
        adjs[ch - base] += ai * pc[c];
      }
    }
  }
  int kr = __ldg(&T.tree_radius[ti]);
  if (kr >= 0 && g.scale != 0.0f && fabsf(r0) > 1.0e-6f)
    atomicAdd(&g.acc[kr], static_cast<double>(g.scale * dr * (r0 < 0.0f ? -1.0f : 1.0f)));
  return true;
}

// The same derivatives from the primitives that carry any: a subtree holding
// no primitive closer than r has partial 0 beside one that does (its term of
// the round is max(r - b, 0) = 0), and where no primitive is that close the
// whole derivative is the nearest primitive's.  So the candidates of the
// point's cell replace the fold of all primitives and its two arrays of n
// floats in local memory, which bound the adjoint.  With the marches below, a
// fitting step of 64 primitives and 32 views at 256^2 takes 10.9 ms, against
// 183 with the full fold and a thread per ray.
//
// The near primitives are joined as in ur_fold_many with every subtree's value
// kept (ids 0..nn-1 the primitives in order, then the joins), and the adjoints
// go down from the last join with the partials the full fold would use.
__device__ __noinline__ bool urtree_backprop(const DevScene& S, int ti, F3 p, const DiffTables& T, GradSink& g) {
  const DevUrTree& t = S.urtrees[ti];
  int cell = 0;
  if (t.n_prims > kMaxDiffPrims || t.n_prims < 2) return false;
  if (t.fine.dims[0] <= 0) return urtree_backprop_full(S, ti, p, T, g);
  constexpr int kNear = ftgpu::kUrNear;
  int idx[kNear];
  int nn = 0;
  Info best{kInf, ftd::kNoRef};
  bool tie = false;
  Ctx<false> cx;
  cx.c = Counters{};
  if (grid_cell(t.fine, p, &cell) || grid_cell(t.outer, p, &cell)) {
    const uint2 range = __ldg(S.cells + cell);
    for (uint32_t k = range.x, end = range.x + range.y; k < end; ++k) {
      const uint2 e = __ldg(S.entries + k);
      if (__uint_as_float(e.x) >= ftd::rmax(t.r, best.d)) break;
      const int i = static_cast<int>(e.y & ~ftd::kRareFlag);
      const float d = ftd::prim_distance(S.nodes[S.ur_prims[i]], p);
      const int ref = d < best.d ? ~i : min(~i, best.ref);
      if (d <= best.d) best = Info{d, ref};  // (equal: the later one's, as in the fold)
      if (d < t.r) {
        if (nn < kNear) idx[nn] = i;
        ++nn;
      }
    }
  } else {
    best = far_nearest<false>(S, t, p, best, &tie, cx);
  }
  if (nn > kNear || best.ref == ftd::kNoRef || tie) return urtree_backprop_full(S, ti, p, T, g);
  if (nn == 0) {
    const int node = S.ur_prims[~best.ref];
    prim_backprop(S.nodes[node], node, p, 1.0f, g);
    return true;
  }
#pragma unroll 1
  for (int i = 1; i < nn; ++i) {
    const int v = idx[i];
    int j = i - 1;
    for (; j >= 0 && idx[j] > v; --j) idx[j + 1] = idx[j];
    idx[j + 1] = v;
  }
  const float r = fmaxf(fabsf(t.r), 1.0e-6f);
  struct Sub {
    float val, top, adj;  // value, value lifted to its parent join (or the root), adjoint
    int lifts, left, right;
  };
  Sub sub[2 * kNear - 1];
  int open[kNear], at[kNear], sp = 0, n_sub = nn, root = 0;
  uint4 path = __ldg(S.ur_paths + idx[0]);
#pragma unroll 1
  for (int i = 0; i < nn; ++i) {
    float cur = ftd::prim_distance(S.nodes[S.ur_prims[idx[i]]], p);
    int id = i, dep = static_cast<int>(path.z), l = -1;
    if (i + 1 < nn) {
      const uint4 nxt = __ldg(S.ur_paths + idx[i + 1]);
      l = ur_lca(path, nxt);
      path = nxt;
    }
#pragma unroll 1
    for (;;) {
      // up to the ancestor that joins it: the open subtree's, or this one's
      const bool join = sp > 0 && at[sp - 1] > l;
      const int to = join ? at[sp - 1] : l;
      sub[id].val = cur;
      sub[id].lifts = dep - to - 1;
      cur = ur_lifts(cur, dep - to - 1, t.r, cx);
      sub[id].top = cur;
      if (!join) break;
      --sp;
      const int lhs = open[sp];
      cur = ftd::op_union_round(sub[lhs].top, cur, t.r);
      sub[n_sub].left = lhs;
      sub[n_sub].right = id;
      id = n_sub++;
      dep = to;
    }
    if (l >= 0) {
      open[sp] = id;
      at[sp++] = l;
    }
    root = id;
  }
  float dr = 0.0f;
  sub[root].adj = 1.0f;
  constexpr int kSteps = 12;
  float v[kSteps];
#pragma unroll 1
  for (int id = root; id >= 0; --id) {
    // down the lifts: their inputs are val, its successive lifts, and from the
    // first that a lift leaves unchanged on that one
    const int lifts = sub[id].lifts;
    int m = 0;
    v[0] = sub[id].val;
#pragma unroll 1
    while (m < lifts) {
      const float up = ur_lift(v[m], t.r);
      if (up == v[m]) break;
      if (m + 1 == kSteps) return urtree_backprop_full(S, ti, p, T, g);
      v[++m] = up;
    }
    float a = sub[id].adj, pa, pb, pr;
#pragma unroll 1
    for (int k = lifts - 1; k >= 0; --k) {
      union_round_partials(v[k < m ? k : m], kInf, r, &pa, &pb, &pr);
      dr += a * pr;
      a *= pa;
    }
    sub[id].adj = a;
    if (id >= nn) {
      const int lhs = sub[id].left, rhs = sub[id].right;
      union_round_partials(sub[lhs].top, sub[rhs].top, r, &pa, &pb, &pr);
      dr += a * pr;
      sub[lhs].adj = a * pa;
      sub[rhs].adj = a * pb;
    }
  }
  // in the full fold's order: by their parents in pre-order, left child first
  bool done[kNear] = {};
#pragma unroll 1
  for (int n = 0; n < nn; ++n) {
    int pick = -1;
    uint4 pp{};
    for (int i = 0; i < nn; ++i) {
      if (done[i]) continue;
      const uint4 pi = __ldg(S.ur_paths + idx[i]);
      if (pick >= 0) {
        const int l = ur_lca(pp, pi);
        const bool first_at = static_cast<int>(pp.z) - 1 == l, second_at = static_cast<int>(pi.z) - 1 == l;
        if (first_at || !second_at) continue;  // (the kept one is to the left)
      }
      pick = i;
      pp = pi;
    }
    done[pick] = true;
    if (sub[pick].adj == 0.0f) continue;
    const int node = S.ur_prims[idx[pick]];
    prim_backprop(S.nodes[node], node, p, sub[pick].adj, g);
  }
  const int kr = __ldg(&T.tree_radius[ti]);
  if (kr >= 0 && g.scale != 0.0f && fabsf(t.r) > 1.0e-6f)
    atomicAdd(&g.acc[kr], static_cast<double>(g.scale * dr * (t.r < 0.0f ? -1.0f : 1.0f)));
  return true;
}

// df/dtheta and grad_p f at p through the winning leaf of the scene.
__device__ __noinline__ bool scene_backprop(const DevScene& S, F3 p, const DiffTables& T, GradSink& g) {
  int leaf = 0;
  if (!(S.fast.kind == kFastTree && S.fast.entry[0] == kNoPrim)) {  // (a tree alone is its only leaf)
    Ctx<false> cx;
    cx.c = Counters{};
    scene_distance_leaf(S, p, &leaf, cx);
  }
  const DevLeaf& lf = S.leaves[leaf];
  if (lf.kind == ftgpu::kLeafUrTree) return urtree_backprop(S, lf.first, p, T, g);
  if (lf.kind == ftgpu::kLeafPrim) {
    const DevNode& n = S.nodes[lf.node];
    if (n.kind != FT_NODE_SPHERE && n.kind != FT_NODE_BOX) return false;
    prim_backprop(n, lf.node, p, 1.0f, g);
    return true;
  }
  return false;
}

// The rays of work items [first, first + n_work) of all views (items_per_view
// each), persistent: lanes whose ray ended take the next item once kWfRefill
// are idle.  Forward (kAdjoint false): depth, mask and silhouette.  Adjoint:
// the rays that carry an upstream gradient march again and leave a record for
// views_adjoint_kernel, hits from the front of `records` and misses from its
// end.  Self-check: a ray ends after at most max_steps march steps and some 200
// of refinement; a lane past max_steps + 256 sets a bit in counters[1] and
// gives up.  There is no time limit: a call is one launch over all its views,
// however long these take.
//
// One thread per ray to the end left a warp waiting for its longest search: a
// miss takes 40 golden-section steps after its march, and an adjoint ray its
// gradient.  Eight blocks per SM (64 registers): 11.4 ms for the step above
// against 12.4 with five.
template <bool kAdjoint, int kForm>
__global__ void __launch_bounds__(128, 8) views_march_persistent(
    const __grid_constant__ DevScene S, const RayParams* __restrict__ views, uint64_t items_per_view, uint64_t first,
    uint64_t n_work, float tau, float* __restrict__ t_out, uint8_t* __restrict__ mask_out, float* __restrict__ sil_out,
    const float* __restrict__ dl_dt, const float* __restrict__ dl_dsil, AdjointRay* __restrict__ records,
    unsigned long long* __restrict__ counters) {
  const unsigned lane = threadIdx.x & 31u;
  Ctx<false> cx;
  cx.c = Counters{};
  uint32_t ray_iters = 0, view = 0;
  bool queue_done = false;
  ViewRay ray;
  uint64_t item = 0;
  size_t idx = 0;
  F3 o = f3(0.0f, 0.0f, 0.0f), d = o;
  float max_t = 0.0f, wt = 0.0f, ws = 0.0f;
  auto finish = [&]() {
    if (!kAdjoint) {
      if (t_out) t_out[idx] = ray.state == ViewRay::kHit ? ray.hi : 0.0f;
      if (mask_out) mask_out[idx] = ray.state == ViewRay::kHit ? 1 : 0;
      if (sil_out) sil_out[idx] = ray.silhouette(tau);
    } else if (ray.state == ViewRay::kHit) {
      if (wt != 0.0f) records[atomicAdd(&counters[2], 1ull)] = AdjointRay{item, ray.hi, wt, 1.0f, 0.0f};
    } else if (ray.state == ViewRay::kMiss) {
      const float sil = ray.silhouette(tau);
      if (ws != 0.0f && ray.best > 0.0f && sil > 0.0f)
        records[n_work - 1 - atomicAdd(&counters[3], 1ull)] = AdjointRay{item, ray.x, ws, sil, 0.0f};
    }
  };
  for (;;) {
    const unsigned idle = __ballot_sync(0xffffffffu, !ray.live());
    if (!queue_done && (__popc(idle) >= kWfRefill || idle == 0xffffffffu)) {
      unsigned long long base = 0;
      if (lane == 0) base = atomicAdd(&counters[0], static_cast<unsigned long long>(__popc(idle)));
      base = __shfl_sync(0xffffffffu, base, 0);
      if (base >= n_work) queue_done = true;
      const uint64_t k = base + __popc(idle & ((1u << lane) - 1u));
      if (!ray.live() && k < n_work) {
        item = first + k;
        view = static_cast<uint32_t>(item / items_per_view);
        const RayParams& P = views[view];
        if (item_ray<kAdjoint>(P, item - static_cast<uint64_t>(view) * items_per_view, &d, &idx)) {
          idx += static_cast<size_t>(view) * P.width * P.height;
          bool march = true;
          if (kAdjoint) {
            wt = dl_dt ? dl_dt[idx] : 0.0f;
            ws = dl_dsil ? dl_dsil[idx] : 0.0f;
            march = wt != 0.0f || ws != 0.0f;
          }
          if (march) {
            o = f3(P.origin[0], P.origin[1], P.origin[2]);
            ray = ViewRay{};
            ray_iters = 0;
            float t0, t1;
            if (ray_aabb(o, d, S.smin, S.smax, &t0, &t1)) {
              max_t = fminf(P.max_dist, t1);
              ray.start(P, t0, max_t);
            }
            if (!ray.live()) finish();
          }
        }
      }
    }
    if (__ballot_sync(0xffffffffu, ray.live()) == 0u) {
      if (queue_done) break;
      continue;
    }
    if (!ray.live()) continue;
    const RayParams& P = views[view];
    if (++ray_iters > 256u && ray_iters - 256u > P.max_steps) {
      atomicOr(&counters[1], 1ull);
      ray.state = ViewRay::kEmpty;
      finish();
      continue;
    }
    ray.next(P, max_t, scene_distance_inl<kForm>(S, o + d * ray.t, cx).d);
    if (!ray.live()) finish();
  }
}

// The recorded rays' parameter gradients, hits first, then misses, a ray per
// thread.  Dynamic shared memory: n_params doubles when `shared_acc`.
__global__ void __launch_bounds__(128) views_adjoint_kernel(
    const __grid_constant__ DevScene S, const RayParams* __restrict__ views, uint64_t items_per_view, uint64_t n_work,
    float tau, DiffTables T, const AdjointRay* __restrict__ records, const unsigned long long* __restrict__ counters,
    double* __restrict__ grad, int shared_acc, int* __restrict__ unsupported) {
  extern __shared__ double sacc[];
  if (shared_acc) {
    for (uint32_t k = threadIdx.x; k < T.n_params; k += blockDim.x) sacc[k] = 0.0;
    __syncthreads();
  }
  double* acc = shared_acc ? sacc : grad;
  const unsigned long long first = static_cast<unsigned long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  const unsigned long long stride = static_cast<unsigned long long>(gridDim.x) * blockDim.x;
  auto setup = [&](const AdjointRay& r, F3* o, F3* d) {
    const uint32_t v = static_cast<uint32_t>(r.ray / items_per_view);
    size_t idx;
    item_ray<true>(views[v], r.ray - static_cast<uint64_t>(v) * items_per_view, d, &idx);
    *o = f3(views[v].origin[0], views[v].origin[1], views[v].origin[2]);
  };
  for (unsigned long long k = first, n = counters[2]; k < n; k += stride) {
    const AdjointRay r = records[k];
    F3 o, d;
    setup(r, &o, &d);
    const F3 p = o + d * r.t;
    GradSink probe{acc, &T, 0.0f, f3(0.0f, 0.0f, 0.0f)};
    if (!scene_backprop(S, p, T, probe)) {
      atomicOr(unsupported, 1);
      continue;
    }
    const float den = ftd::dot3(probe.gp, d);
    if (fabsf(den) <= 1.0e-8f) continue;
    GradSink sink{acc, &T, -r.w / den, f3(0.0f, 0.0f, 0.0f)};
    scene_backprop(S, p, T, sink);
  }
  for (unsigned long long k = first, n = counters[3]; k < n; k += stride) {
    const AdjointRay r = records[n_work - 1 - k];
    F3 o, d;
    setup(r, &o, &d);
    // The minimum is flat along the ray, so its FP32 position is only known
    // to ~1e-3: polish it with secant steps on df/dt = grad_p f . d = 0.
    float tm = r.t;
    bool ok = true;
    auto slope = [&](float tt) {
      GradSink probe{acc, &T, 0.0f, f3(0.0f, 0.0f, 0.0f)};
      ok &= scene_backprop(S, o + d * tt, T, probe);
      return ftd::dot3(probe.gp, d);
    };
    const float dt0 = 1.0e-3f * fmaxf(1.0f, tm);
    const float g0 = slope(tm);
    float ta = tm - dt0, tb = tm + dt0;
    float ga = slope(ta), gb = slope(tb);
    for (int s = 0; s < kMinPolishSteps && ok && gb != ga; ++s) {
      float tn = tb - gb * (tb - ta) / (gb - ga);
      tn = fminf(fmaxf(tn, tm - 4.0f * dt0), tm + 4.0f * dt0);
      ta = tb;
      ga = gb;
      tb = tn;
      gb = slope(tb);
    }
    if (ok && fabsf(gb) < fabsf(g0)) tm = tb;
    GradSink sink{acc, &T, -r.w * r.sil / tau, f3(0.0f, 0.0f, 0.0f)};
    if (!ok || !scene_backprop(S, o + d * tm, T, sink)) atomicOr(unsupported, 1);
  }
  if (shared_acc) {
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < T.n_params; k += blockDim.x)
      if (sacc[k] != 0.0) atomicAdd(&grad[k], sacc[k]);
  }
}
