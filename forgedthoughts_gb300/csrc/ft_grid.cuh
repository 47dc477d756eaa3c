// Candidate grids built on the device.
//
// For a cell C with centre m and half diagonal h, and a primitive i with
// distance d_i (1-Lipschitz: the host admits no other to a grid), centre c_i
// and outer radius R_i,
//
//     d_i(m) - h  and  |C - c_i| - R_i  bound d_i from below over C,
//     d_i(m) + h                        bounds it from above,
//
// and C lists {i : max(0, lower bounds) < max(r, min_j d_j(m) + h)}, sorted by
// the lower bound.  A primitive left out is at least r away at every point of
// C and at least as far as the nearest one, so it cannot change a point's
// distance; the walk of a list ends at the first entry whose bound reaches the
// running limit.  All in FP32: `slack` covers the rounding of the bounds and
// of the device's evaluation, and cells are padded by a thousandth of their
// size against rounding in the cell lookup.
//
// Blocks of 4^3 cells, one thread per cell.  The block first keeps the
// primitives that pass the same test for the block as a whole (its cells'
// centres and half diagonals lie inside the block's), so a cell tests a few
// dozen primitives instead of all.  A hard union's walk gives up inside its
// solids (see union_distance), so a cell that lies inside one primitive keeps
// no list there.  Two passes of the same kernel: the first
// counts a cell's entries, the second, with the memory in place, writes them.
//
// Bound by the distance evaluations of the block's primitives (a few million
// for 512 primitives).  Opening the 512-primitive field and rendering its
// 800x600 preview takes 8.4 ms; it took 38 when 16 host threads built the lists
// and a slower march rendered it.
//
// Included by ft_kernels.cuh (precompiled only).
#pragma once

struct GridJob {
  float gmin[3], cell;
  int32_t dims[3];
  int32_t first;   // of the grid's cells
  int32_t prim_first, n_prims;
  float r, slack;
  int32_t skip_inside;  // cells inside one primitive keep no list (kInsideCell)
};

constexpr int kGridBlockEdge = 4;
constexpr int kGridKeep = 2048;  // primitives a block of cells keeps; past it every cell tests all

struct GridBound {
  float d, low;   // distance at m, lower bound over the box around m
  uint32_t rare;  // the compact entry's rare flag
};

// Primitive `i` against the box of half size `half` at m.  Out of line: both
// passes run the same instructions, so the entries counted are the entries
// written.
__device__ __noinline__ GridBound grid_bound(const DevScene& S, int i, F3 m, float half) {
  const float4* w = S.cprims + 3 * static_cast<size_t>(i);
  const float4 a = __ldg(w), b = __ldg(w + 1), e = __ldg(w + 2);
  const F3 c = f3(a.x, a.y, a.z);
  GridBound g;
  g.rare = __float_as_uint(e.w) & ftd::kRareFlag;
  float radius;
  if (g.rare) {
    const DevNode& n = S.nodes[__float_as_int(e.z)];
    radius = 0.5f * (n.bmax[0] - n.bmin[0]);
    g.d = rare_distance(n, m);
  } else {
    radius = ftd::len3(f3(b.x, b.y, b.z)) + b.w;
    g.d = ftd::compact_distance<false>(a, b, e.x, e.y, m);
  }
  const float dx = fmaxf(fabsf(m.x - c.x) - half, 0.0f), dy = fmaxf(fabsf(m.y - c.y) - half, 0.0f),
              dz = fmaxf(fabsf(m.z - c.z) - half, 0.0f);
  g.low = fmaxf(g.d - half * 1.7320509f, sqrtf(dx * dx + dy * dy + dz * dz) - radius);
  return g;
}

template <bool kFill>
__global__ void __launch_bounds__(64) grid_cells_kernel(const __grid_constant__ DevScene S,
                                                        const __grid_constant__ GridJob J, uint2* __restrict__ cells,
                                                        uint2* __restrict__ entries,
                                                        unsigned long long* __restrict__ total) {
  __shared__ int keep[kGridKeep];
  __shared__ int n_keep;
  __shared__ float bound[2];
  __shared__ unsigned int warp_sum;
  __shared__ unsigned long long base;
  const int t = threadIdx.x;
  const int nbx = (J.dims[0] + kGridBlockEdge - 1) / kGridBlockEdge, nby = (J.dims[1] + kGridBlockEdge - 1) / kGridBlockEdge;
  const int b0[3] = {static_cast<int>(blockIdx.x % nbx) * kGridBlockEdge,
                     static_cast<int>(blockIdx.x / nbx % nby) * kGridBlockEdge,
                     static_cast<int>(blockIdx.x / nbx / nby) * kGridBlockEdge};
  const float pad = J.cell * 1.0e-3f;
  if (t == 0) n_keep = 0;
  {
    const float half = 0.5f * kGridBlockEdge * J.cell + pad;
    const F3 m = f3(J.gmin[0] + (b0[0] + 0.5f * kGridBlockEdge) * J.cell, J.gmin[1] + (b0[1] + 0.5f * kGridBlockEdge) * J.cell,
                    J.gmin[2] + (b0[2] + 0.5f * kGridBlockEdge) * J.cell);
    float best = kInf;
    for (int k = t; k < J.n_prims; k += 64) best = fminf(best, grid_bound(S, J.prim_first + k, m, half).d);
    for (int off = 16; off > 0; off >>= 1) best = fminf(best, __shfl_xor_sync(0xffffffffu, best, off));
    if ((t & 31) == 0) bound[t >> 5] = best;
    __syncthreads();
    const float limit = fmaxf(J.r, fminf(bound[0], bound[1]) + half * 1.7320509f) + J.slack;
    for (int k = t; k < J.n_prims; k += 64) {
      if (grid_bound(S, J.prim_first + k, m, half).low - J.slack < limit) {
        const int at = atomicAdd(&n_keep, 1);
        if (at < kGridKeep) keep[at] = k;
      }
    }
    __syncthreads();
  }
  const bool all = n_keep > kGridKeep;
  const int n = all ? J.n_prims : n_keep;
  const int x = b0[0] + (t & 3), y = b0[1] + (t >> 2 & 3), z = b0[2] + (t >> 4);
  bool mine = x < J.dims[0] && y < J.dims[1] && z < J.dims[2];
  const int cell = J.first + x + J.dims[0] * (y + J.dims[1] * z);
  const float half = 0.5f * J.cell + pad;
  const F3 m = f3(J.gmin[0] + (x + 0.5f) * J.cell, J.gmin[1] + (y + 0.5f) * J.cell, J.gmin[2] + (z + 0.5f) * J.cell);
  float limit = 0.0f;
  unsigned count = 0;
  if (mine && kFill) {
    // the count pass left the cell's limit beside its count
    const uint2 c = cells[cell];
    limit = __uint_as_float(c.x);
    count = c.y;
    if (count == kInsideCell) {
      count = 0;
      mine = false;
    }
  } else if (mine) {
    float best = kInf;
    for (int k = 0; k < n; ++k) best = fminf(best, grid_bound(S, J.prim_first + (all ? k : keep[k]), m, half).d);
    limit = fmaxf(J.r, best + half * 1.7320509f) + J.slack;
    const bool inside = J.skip_inside && best + half * 1.7320509f < -J.slack;
    for (int k = 0; k < (inside ? 0 : n); ++k)
      count += grid_bound(S, J.prim_first + (all ? k : keep[k]), m, half).low - J.slack < limit;
    cells[cell] = make_uint2(__float_as_uint(limit), inside ? kInsideCell : count);
  }
  // the block's entries: counted into the total, or allocated from it
  unsigned scan = count;
  for (int off = 1; off < 32; off <<= 1) {
    const unsigned up = __shfl_up_sync(0xffffffffu, scan, off);
    if ((t & 31) >= off) scan += up;
  }
  if (t == 31) warp_sum = scan;
  __syncthreads();
  if (t >= 32) scan += warp_sum;
  if (t == 63) base = atomicAdd(total, static_cast<unsigned long long>(scan));
  if (!kFill) return;
  __syncthreads();
  if (!mine) return;
  const unsigned at = static_cast<unsigned>(base) + scan - count;
  cells[cell] = make_uint2(at, count);
  // Ascending by (bound, index): a short list by insertion as it is written, a
  // long one by heap sort in place.
  auto before = [](uint2 u, uint2 v) { return u.x < v.x || (u.x == v.x && (u.y & ~ftd::kRareFlag) < (v.y & ~ftd::kRareFlag)); };
  uint2* list = entries + at;
  const bool insert = count <= 24;
  unsigned w = 0;
  for (int k = 0; k < n && w < count; ++k) {
    const int i = J.prim_first + (all ? k : keep[k]);
    const GridBound g = grid_bound(S, i, m, half);
    const float low = g.low - J.slack;
    if (!(low < limit)) continue;
    const uint2 u = make_uint2(__float_as_uint(fmaxf(low, 0.0f)), static_cast<uint32_t>(i) | g.rare);
    unsigned j = w++;
    for (; insert && j > 0 && before(u, list[j - 1]); --j) list[j] = list[j - 1];
    list[j] = u;
  }
  if (insert) return;
  auto sift = [&](unsigned root, unsigned end) {
    const uint2 v = list[root];
    for (unsigned child = 2 * root + 1; child < end; child = 2 * root + 1) {
      if (child + 1 < end && before(list[child], list[child + 1])) ++child;
      if (!before(v, list[child])) break;
      list[root] = list[child];
      root = child;
    }
    list[root] = v;
  };
  for (unsigned k = w / 2; k-- > 0;) sift(k, w);
  for (unsigned k = w; k-- > 1;) {
    const uint2 v = list[0];
    list[0] = list[k];
    list[k] = v;
    sift(0, k);
  }
}
