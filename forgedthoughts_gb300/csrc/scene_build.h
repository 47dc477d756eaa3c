// Host-side construction of the GPU scene image: device node table, hard-union
// leaves, the leaf BVH, generic leaf programs and the culled union_round-tree
// structures.  Pure C++ (no CUDA) so it is shared by the renderer and the
// structure tests.
#pragma once

#include <cstdint>
#include <string>
#include <vector>

#include "forgedthoughts_gb300.h"
#include "ft_layout.h"

namespace ftgpu {

struct HostNode {  // mirrors ftd::DevNode (128 bytes)
  int32_t kind, a, b, program;
  uint32_t object_id, material_id;
  int32_t ival, has_rot;
  float c[3];
  float sz, cz, sy, cy, sx, cx;
  float f[6];
  float bmin[3], bmax[3];
  float pad[3];
};
static_assert(sizeof(HostNode) == 128, "HostNode layout");

struct HostLeaf {
  float bmin[3], bmax[3];
  int32_t kind;
  int32_t node;
  int32_t first;
  int32_t count;
};

struct HostBvhNode {  // leaf BVH in the reference's build order (R:693-732)
  float bmin[3], bmax[3];
  int32_t lhs, rhs, leaf, pad;
};

struct CompactPrim {  // the device's three 16-byte words (compact_distance)
  float c[3], cos;
  float h[3], rd;  // (h[0] is -0 for a sphere)
  float sin, shell;
  int32_t node;
  uint32_t leaf;  // leaf index, high bit: not a compact kind, evaluated through its node
};
static_assert(sizeof(CompactPrim) == 48, "CompactPrim layout");

struct UrPath {  // a tree primitive's way from the root: bit k is the side taken at depth k
  uint64_t sides;
  uint32_t depth;
  uint32_t pad;
};

struct HostUrTree {
  float r;
  int32_t n_prims;
  int32_t prim_first;   // into ur_prims (in-order position -> node index)
  int32_t bvh_root;     // into ur_bvh
  int32_t inner_root;   // into ur_inner
  int32_t depth;
  int32_t fallback_first, fallback_count;  // generic program of the whole tree
  // Candidate grid: cell c lists every primitive that can be the nearest or
  // lie within r of some point of c.  dims[0] == 0 disables the grid.
  float gmin[3];
  float cell, inv_cell;
  int32_t dims[3];
  int32_t cell_first;  // into ur_cell_offsets (dims product + 1 entries)
  // Outer grid: coarser cells over a box around the first grid, for points
  // outside it (there every primitive is at least 2r away, so a cell lists
  // the primitives that can be the nearest).  odims[0] == 0: none.
  float ogmin[3];
  float ocell, oinv_cell;
  int32_t odims[3];
  int32_t ocell_first;
};

struct HostUrBvh {
  float bmin[3], bmax[3];
  int32_t left, right;
  int32_t prim_begin, prim_count;  // into ur_bvh_prims (in-order positions)
};

struct HostUrInner {
  int32_t child[2];  // >= 0: ur_inner index; < 0: -(position + 1) of a primitive
  int32_t lo, hi;    // in-order primitive range covered (relative to the tree)
};

struct SceneImage {
  std::vector<HostNode> nodes;
  std::vector<HostLeaf> leaves;
  std::vector<HostBvhNode> bvh;
  int32_t bvh_root = -1;
  std::vector<uint32_t> gops;
  std::vector<HostUrTree> urtrees;
  std::vector<HostUrBvh> ur_bvh;
  std::vector<int32_t> ur_bvh_prims;
  std::vector<int32_t> ur_prims;
  std::vector<HostUrInner> ur_inner;
  std::vector<uint32_t> ur_cell_offsets;  // per grid cell: begin into ur_cell_prims
  std::vector<int32_t> ur_cell_prims;     // in-order primitive positions
  // per ur_cell_prims entry: a lower bound of the distance from any point of
  // the cell to the primitive's box (the lists are sorted by it)
  std::vector<float> ur_cell_gaps;
  // A scene of one union_round tree, alone or beside one primitive whose box
  // bounds its distance: their leaves, -1 for other scenes (and no primitive).
  int32_t fast_tree = -1, fast_prim = -1;
  // All leaves are primitives whose boxes bound their distances.
  bool fast_union = false;
  // compact records: of the union_round trees' primitives, indexed as ur_prims,
  // then that of fast_prim; of every leaf, in leaf order, of a fast_union scene.
  // Root paths of the trees' primitives.
  std::vector<CompactPrim> cprims;
  std::vector<UrPath> ur_paths;
  // per ur_inner node: 1 when its primitives use more than one material model
  // (blend_materials then yields a Blend whatever the weights)
  std::vector<int32_t> ur_inner_blend;
  std::vector<int32_t> node_op_begin, node_op_end;  // postfix op range of each node's subtree
  // per object id: the primitive or Custom node carrying it (its transform is
  // the object's, object_transforms R:485-555), -1 for none
  std::vector<int32_t> obj_node;
  std::vector<ft_material> materials;
  std::vector<ft_light> lights;
  int32_t environment_program = -1;
  std::vector<ft_program> programs;
  std::vector<ft_instr> instrs;
  float scene_min[3], scene_max[3];
  float scene_center[3];
  ft_camera camera;
  int32_t has_camera = 0;
  int32_t max_value_stack = 0, max_point_stack = 0;
};

// Build the image; returns false with `error` set on an invalid description.
// With `lists` the candidate lists of the union_round grids are built here
// (ft_scene_build_info reports them); without, only the grids' geometry: a
// scene on a device builds its own lists there.
bool build_scene_image(const ft_scene_desc& desc, SceneImage* out, std::string* error, bool lists);

// Compact record of a primitive node (rare-flagged where its kind or turn has
// none).
CompactPrim compact_prim(const SceneImage& img, int node, uint32_t leaf);

// Tree over compact primitives for points outside their candidate grids, in
// depth-first order: a walk goes to the next node, or past a subtree whose box
// is out of reach, and needs no stack.
struct FarNode {
  float bmin[3];
  int32_t skip;  // the node after the subtree
  float bmax[3];
  int32_t prims;  // -1: inner; else (first far entry << 3) | entries
};
static_assert(sizeof(FarNode) == 32, "FarNode layout");
constexpr int kFarLeaf = 4;
// Appends the tree of the compact primitives [first, first + n) and its
// entries (compact index | rare flag).
void build_far_tree(const SceneImage& img, const std::vector<CompactPrim>& prims, int32_t first, int32_t n,
                    std::vector<FarNode>* nodes, std::vector<uint32_t>* entries);

// Camera basis (R:6263-6286, render_api.rs:132-144) in f32.
struct CameraBasis {
  float origin[3], forward[3], right[3], up[3];
  float tan_fov;
};
CameraBasis resolve_camera(const SceneImage& img, const ft_render_options& opt);
// Basis of a camera at `org` looking at `tgt` (up (0, 1, 0)).
CameraBasis camera_basis(const float org[3], const float tgt[3], float fov);

}  // namespace ftgpu
