"""Where the short scene forms, the candidate grids, the material resolve, the
views passes and the path tracer's passes reach their limits: primitives whose
distance is not bounded by their box, hits that lie farther from the surface
than the blend radius, scenes of very many trees, marches of unbounded length,
large sample counts, ties."""
import ctypes

import numpy as np
import pytest

import forgedthoughts_gb300 as ft
import oracle
from forgedthoughts_gb300 import _native, workloads
from parity import radiance_rmse

pytestmark = pytest.mark.gpu

LIGHTS = ("let camera = Camera { origin: vec3(0, 1.2, -5), target: vec3(0, 0.6, 0), fov_y: 45.0 };\n"
          "let light = PointLight { position: vec3(3, 6, -3), intensity: 60.0 };\n")


def _points(n, reach, seed=11):
    rng = np.random.default_rng(seed)
    return rng.uniform([-reach, -0.5 * reach, -reach], [reach, reach, reach], size=(n, 3)).astype(np.float32)


def _distances(st, pts):
    g = st.gpu()
    g.build_bricks(0.25)
    return g.brick_bounds(pts)[1].astype(np.float64)


def _tree(names, k, tag="u"):
    """A balanced pairwise union_round(k) tree: its lines and its root."""
    lines, cur, level = [], list(names), 0
    while len(cur) > 1:
        nxt = []
        for j in range(0, len(cur) - 1, 2):
            lines.append(f"let {tag}{level}_{j // 2} = {cur[j]}.union_round({cur[j + 1]}, {k});")
            nxt.append(f"{tag}{level}_{j // 2}")
        cur, level = nxt + cur[len(cur) - len(cur) % 2:], level + 1
    return lines, cur[0]


SPHERES = [f"let s{i} = Sphere {{ radius: 0.3, pos: vec3({x}, 0.5, {z}) }};"
           for i, (x, z) in enumerate([(-2.2, -1.9), (1.7, -2.1), (-1.8, 2.0), (2.1, 1.6)])]


@pytest.mark.parametrize("tree_first", [False, True])
@pytest.mark.parametrize("sides", [3, 6])
def test_tree_beside_an_extruded_polygon(sides, tree_first):
    """An extruded polygon's distance is measured to its edge lines and can be
    less than its box's, so it must not bound the walk of a tree beside it.
    Tolerance as for the other distances of a scene: 1e-5 of the value or 1."""
    lines, root = _tree([f"s{i}" for i in range(4)], 0.3)
    prism = f"let prism = ExtrudePolygon {{ sides: {sides}, radius: 1.0, height: 0.6, pos: vec3(0.3, 0.4, -0.2) }};"
    src = "\n".join(SPHERES + lines + [prism]) + "\nlet scene = " + (
        f"{root} + prism;\n" if tree_first else f"prism + {root};\n")
    st = ft.parse_and_eval(src)
    pts = _points(60000, 9.0)
    ref, _, _ = oracle.distance(st, pts, accel=1, precision=32)
    err = np.abs(_distances(st, pts) - ref)
    # (which leaf the walk visits hangs on comparisons of box bounds: a point
    # within a rounding step of one may go either way)
    assert (err > 1e-5 * np.maximum(1.0, np.abs(ref))).sum() <= 2, (float(err.max()), pts[err.argmax()])


def test_tree_beside_a_box_rounded_past_its_size():
    """A node record may hold a rounding above the half size; its box does not
    bound its distance either."""
    lines, root = _tree([f"s{i}" for i in range(4)], 0.3)
    src = "\n".join(SPHERES + lines + ["let b = Box { size: vec3(0.4, 0.4, 0.4), round: 0.1, pos: vec3(0, 0.6, 0) };"])
    st = ft.parse_and_eval(src + f"\nlet scene = {root} + b;\n")
    box = [i for i in range(st.desc.n_nodes) if st.desc.nodes[i].kind == _native.FT_NODE_BOX]
    ctypes.cast(st.desc.nodes, ctypes.POINTER(_native.NodeC))[box[0]].f[3] = 0.9
    pts = _points(60000, 9.0)
    ref, _, _ = oracle.distance(st, pts, accel=1, precision=32)
    err = np.abs(_distances(st, pts) - ref)
    assert (err > 1e-5 * np.maximum(1.0, np.abs(ref))).sum() <= 2, (float(err.max()), pts[err.argmax()])


def test_material_of_a_primitive_nearer_than_the_tree():
    """A hit (of a large epsilon) on the primitive beside a tree, at a point
    outside the tree's grids where the tree's box is the nearer one: the
    tree's walk ends without a surface below the primitive's distance, and the
    hit carries the primitive's material."""
    lines = [f"let s{i} = Sphere {{ radius: 0.01, pos: vec3({x}, {y}, 0.0), material: Metal {{ roughness: 0.1 }} }};"
             for i, (x, y) in enumerate([(-0.05, -1.5), (0.05, -1.5), (-0.05, 1.5), (0.05, 1.5)])]
    ups, root = _tree([f"s{i}" for i in range(4)], 0.01)
    ball = "let ball = Sphere { radius: 0.1, pos: vec3(0, 0, -3.6), material: Lambert { color: vec3(1, 0, 0) } };"
    camera = "let camera = Camera { origin: vec3(-6, 0, -1.7), target: vec3(0, 0, -1.7), fov_y: 3.0 };"
    st = ft.parse_and_eval("\n".join(lines + ups + [ball, camera]) + f"\nlet scene = {root} + ball;\n")
    opts = ft.RenderOptions(width=64, height=64, max_steps=64, max_dist=20.0, epsilon=1.85, step_scale=0.5)
    img = ft.render_depth(st, opts, ft.AccelMode.Bvh, 1, want_material=True)
    _, m, mat, _, _ = oracle.render_depth(st, opts, 1, 1, 32)
    both = (img.mask == 1) & (m == 1)
    assert both.mean() > 0.5 and (mat[both] != 0).all()
    assert (img.material[both] == mat[both]).all()


@pytest.mark.parametrize("n", [6, 14])
def test_resolve_of_hits_farther_off_than_the_blend_radius(n):
    """An epsilon above the blend radius stops a ray where no primitive is
    within it: the gather widens instead of giving up (the general resolve of
    the fallback holds eight open subtrees, a chain of 14 needs more, and its
    material's hooks were lost)."""
    from test_frontend import HOOK_MATERIALS

    lines = [f"let s{i} = Sphere {{ radius: 0.35, pos: vec3({-1.6 + 3.2 * i / (n - 1):.4f}, "
             f"{0.6 + 0.2 * (i % 3):.2f}, {0.1 * (i % 4):.2f}), material: Stripe {{}} }};" for i in range(n)]
    lines.append(f"let u{n - 1} = s{n - 1};")
    for i in range(n - 2, -1, -1):  # every left child a sphere: a chain to the right
        lines.append(f"let u{i} = s{i}.union_round(u{i + 1}, 0.005);")
    st = ft.parse_and_eval(HOOK_MATERIALS + LIGHTS + "\n".join(lines) + "\nlet scene = u0;\n")
    opts = ft.RenderOptions(width=120, height=80, max_steps=256, max_dist=30.0, epsilon=0.01, step_scale=0.7)
    lin, _ = ft.render_trace(st, opts, ft.AccelMode.Bvh, 1, 1)
    ref, _, _ = oracle.render_trace(st, opts, 1, 1, 1, 32)
    assert ref.max() > 0.1
    # the Whitted bar; silhouette pixels whose hit flips count as everywhere
    assert radiance_rmse(lin, ref) <= 1e-3, radiance_rmse(lin, ref)


def test_grids_of_very_many_trees_are_bounded():
    """Each union_round tree asks for its own cells; past 2^26 of them, or
    2^26 list entries, further trees keep no grid and take their BVH."""
    n, lines, roots = 2400, [], []
    for k in range(n):
        x, z = (k % 49 - 24) * 0.4, (k // 49 - 24) * 0.4
        names = [f"s{k}_{i}" for i in range(4)]
        lines += [f"let {v} = Sphere {{ radius: 0.08, pos: vec3({x + 0.1 * (i % 2):.3f}, {0.1 * (i // 2):.3f}, {z:.3f}) }};"
                  for i, v in enumerate(names)]
        ups, root = _tree(names, 0.05, f"u{k}_")
        lines += ups
        roots.append(root)
    st = ft.parse_and_eval(LIGHTS + "\n".join(lines) + "\nlet scene = " + " + ".join(roots) + ";\n")
    size = ctypes.c_uint64()
    assert _native.lib().ft_scene_device_bytes(st.gpu().handle, ctypes.byref(size)) == 0
    assert size.value <= 2 * 8 * 2 ** 26 + 2 ** 26  # cells and entries of 8 bytes; the scene's records
    opts = ft.RenderOptions(width=64, height=48, max_steps=256, max_dist=40.0, epsilon=1e-4, step_scale=0.7)
    img = ft.render_depth(st, opts, ft.AccelMode.Bvh, 1)
    t, m, _, _, _ = oracle.render_depth(st, opts, 1, 1, 32)
    both = (img.mask == 1) & (m == 1)
    assert (img.mask == m).mean() >= 0.999 and both.mean() > 0.1
    assert (np.abs(img.t[both] - t[both]) <= 1e-4).mean() >= 0.999


def _hard_fit_scene():
    return ft.ParamScene(workloads.shape_fit(n=16))


def test_views_take_any_step_limit():
    """A march ends by its own distance limit; a step limit near 2^32 changes
    nothing."""
    ps, vs = _hard_fit_scene(), ft.ring_views(2)
    got = []
    for steps in (100000, 2 ** 32 - 1):
        opts = ft.RenderOptions(width=64, height=64, max_steps=steps, max_dist=100.0, epsilon=1e-4, step_scale=0.05)
        t, mask, sil = ps.render(vs, opts)
        g = ps.backward(vs, opts, (mask == 1).astype(np.float32), (mask == 0).astype(np.float32))
        got.append((t, mask, sil, g))
    assert got[0][1].any()
    for a, b in zip(got[0][:3], got[1][:3]):
        assert np.array_equal(a, b)
    assert np.allclose(got[0][3], got[1][3], rtol=1e-6, atol=1e-6 * np.abs(got[0][3]).max())  # atomics' order


def test_views_take_as_long_as_they_need():
    """A views call is one launch however long it takes (here about 28 s: a
    thousand shells around one centre, interpreted hooks, short steps)."""
    lines = ["let twist = fn(p) { return rotate_y(p, p.y * 18.0); };",
             "let ripple = fn(d, p) { return abs(d + sin(p.y * 120.0) * 0.004) - 0.03; };"]
    lines += [f"let s{i} = Sphere {{ radius: {1.0 + 0.0001 * i:.4f}, domain: twist, distance_post: ripple }};"
              for i in range(1300)]
    ps = ft.ParamScene("\n".join(lines) + "\nlet scene = " + " + ".join(f"s{i}" for i in range(1300)) + ";\n")
    opts = ft.RenderOptions(width=1024, height=1024, max_steps=4000, max_dist=100.0, epsilon=1e-6, step_scale=0.05)
    _, mask, _ = ps.render(ft.ring_views(1), opts)
    assert 0.1 < mask.mean() < 0.4


def _path(st, opts, spp, min_spp, threshold):
    return ft.render_pathtrace(st, opts, ft.AccelMode.Bvh,
                               ft.PathtraceSettings(spp=spp, min_spp=min_spp, noise_threshold=threshold))


def test_path_ends_with_its_last_pixel():
    """Once every pixel has reached its noise threshold no further pass is
    launched, whatever the sample limit, and the result is the one at a limit
    that the last pixel just reaches."""
    w = workloads.union_round_field(n=16, seed=2, width=24, height=16, aa=1)
    st = ft.parse_and_eval(w.source)
    many = _path(st, w.options, 65536, 2, 0.5)
    launches = ctypes.c_uint32()
    assert _native.lib().ft_scene_last_launches(st.gpu().handle, ctypes.byref(launches)) == 0
    most = int(many[2].max())
    assert most < 1024
    assert launches.value <= 2 * (most // 4 + 1) + 64
    few = _path(st, w.options, most, 2, 0.5)
    for a, b in zip(many, few):
        assert np.array_equal(a, b)


def test_path_buffers_do_not_grow_with_the_frame():
    """A large frame is traced in bands: beyond the frame's own buffers (which
    the depth preview has too) at most 2^24 samples of 12 bytes and the state
    of a band.  Rows of every band against the f32 oracle, at the bars of the
    path tracer's other comparisons."""
    torch = pytest.importorskip("torch")
    st = ft.parse_and_eval(LIGHTS + "let scene = Sphere { radius: 0.9, pos: vec3(0, 0.6, 0) };")
    opts = ft.RenderOptions(width=6144, height=4096, max_steps=64, max_dist=20.0, epsilon=1e-3, step_scale=0.9)
    h, o = st.gpu().handle, opts.to_c()
    lib = _native.lib()
    assert lib.ft_render_depth(h, ctypes.byref(o), 1, 1, None, None, None, None, None, 0, None) == 0
    count = torch.zeros(opts.height, opts.width, dtype=torch.int32, device="cuda")
    rgb = torch.zeros(opts.height, opts.width, 3, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    settings = _native.PathtraceSettingsC(2, 1, 1, 0.0)
    assert lib.ft_render_pathtrace(h, ctypes.byref(o), 1, ctypes.byref(settings), ctypes.c_void_p(rgb.data_ptr()),
                                   None, ctypes.c_void_p(count.data_ptr()), _native.FT_FLAG_DEVICE_POINTERS, None) == 0
    assert free - torch.cuda.mem_get_info()[0] <= 12 * 2 ** 24 + 2 ** 27
    assert (count == 2).all()
    ref, _, _, _ = oracle.render_path(st, opts, 1, spp=2, max_bounces=1, min_spp=1, noise_threshold=0.0,
                                      rows=(300, 4096, 500))
    rows = np.arange(300, 4096, 500)
    got, ref = rgb.cpu().numpy()[rows].astype(np.float64), ref[rows]
    assert ref.max() > 0.1
    assert (np.abs(got - ref).max(axis=-1) <= 1e-3).mean() >= 0.99 and radiance_rmse(got, ref) <= 2e-2


@pytest.mark.parametrize("n", [4, 64])
def test_a_new_scene_is_complete_for_every_stream(n):
    """A scene rendered straight after its creation on a stream that does not
    wait for the default stream: the frame it gives later."""
    torch = pytest.importorskip("torch")
    w = workloads.union_round_field(n=n, seed=4, width=320, height=180, aa=1)
    stream, o = torch.cuda.Stream(), w.options.to_c()
    st = ft.parse_and_eval(w.source)
    t = [torch.zeros(180 * 320, dtype=torch.float32, device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    for x in t:
        assert _native.lib().ft_render_depth(st.gpu().handle, ctypes.byref(o), 1, 1, ctypes.c_void_p(x.data_ptr()), None,
                                             None, None, None, _native.FT_FLAG_DEVICE_POINTERS,
                                             ctypes.c_void_p(stream.cuda_stream)) == 0
        torch.cuda.synchronize()
    assert (t[0] > 0).any() and torch.equal(t[0], t[1])


@pytest.mark.parametrize("extra", [0, 1, 5])
def test_adjoint_of_equally_near_primitives(extra):
    """Where two primitives are equally far and none within the blend radius,
    the whole derivative is the later one's (the folds take `a < b ? a : b`),
    as in the FP64 adjoint: mirrored spheres seen along their plane."""
    lines = [f"let p{i} = Sphere {{ radius: 0.3, pos: vec3({x}, {y}, 0.0) }};"
             for i, (x, y) in enumerate([(-1.0, 0.0), (1.0, 0.0), (-1.0, 1.5), (1.0, 1.5)])]
    lines += [f"let p{4 + i} = Sphere {{ radius: 0.2, pos: vec3({6 + i}, 4, 0.5) }};" for i in range(extra)]
    ups, root = _tree([f"p{i}" for i in range(4 + extra)], 0.1)
    ps = ft.ParamScene("\n".join(lines + ups) + f"\nlet scene = {root};\n")
    vs = [((0.0, 0.0, -5.0), (0.0, 0.0, 0.0), 40.0)]
    opts = workloads.shape_fit_options(33)  # odd: the middle column looks along x = 0
    _, mask, sil = ps.render(vs, opts, 0.2)
    ws = np.zeros(mask.shape, np.float32)
    ws[0, 14:19, 16] = 1.0
    assert (mask[ws > 0] == 0).all() and (sil[ws > 0] > 1e-3).all()
    g = ps.backward(vs, opts, None, ws, 0.2)
    ref = oracle.render_backward(ps.state, vs, opts, ps.layout, None, ws, 0.2, 64)
    # FP32 positions of the minima: the bound of the other gradient comparisons
    assert np.abs(g - ref).max() <= 2e-2 * np.abs(ref).max(), (g, ref)


def test_round_boxes_and_spheres_keep_their_own_summation():
    """A box rounded to its half size has an empty core like a sphere's, but
    its squares are summed in a box's order: among hard-unioned primitives it
    has the distance, to the bit, that it has beside a boolean, where every
    primitive is evaluated from its node."""
    lines = ["let a = Box { size: vec3(0.8, 0.8, 0.8), round: 0.4, pos: vec3(-0.7, 0.5, 0.1) };",
             "let b = Box { size: vec3(0.6, 1.2, 0.7), round: 0.3, pos: vec3(0.7, 0.6, -0.2), rot: vec3(0, 25, 0) };",
             "let c = Sphere { radius: 0.35, pos: vec3(0.1, 0.4, 0.9) };",
             "let d = Box { size: vec3(20, 0.2, 20), pos: vec3(0, 60, 0) };",
             "let e = Box { size: vec3(20, 0.2, 20), pos: vec3(0, 61, 0) };"]
    pts = _points(40000, 2.5)
    fast = ft.parse_and_eval("\n".join(lines) + "\nlet scene = a + b + c + d;\n")
    general = ft.parse_and_eval("\n".join(lines) + "\nlet scene = a + b + c + (d - e);\n")
    assert np.array_equal(_distances(fast, pts), _distances(general, pts))


def test_the_adjoint_marches_the_forward_rays():
    """The adjoint re-marches each ray, so it must find what the forward pass
    found: a silhouette gradient on the forward pass's hits alone, or a depth
    gradient on its misses alone, reaches no parameter."""
    ps, vs = ft.ParamScene(workloads.shape_fit(n=64)), ft.ring_views(24)
    opts = workloads.shape_fit_options(512)
    _, mask, _ = ps.render(vs, opts)
    assert 0.02 < mask.mean() < 0.98
    assert not ps.backward(vs, opts, None, (mask == 1).astype(np.float32)).any()
    assert not ps.backward(vs, opts, (mask == 0).astype(np.float32), None).any()


def test_crowded_hard_union():
    """More primitives in one block of cells than a block keeps (2048), and
    lists long enough for the heap sort: spheres around nearly one centre."""
    rng = np.random.default_rng(3)
    lines = [f"let s{i} = Sphere {{ radius: {0.5 + 4e-5 * i:.5f}, pos: vec3({x:.4f}, {y:.4f}, {z:.4f}) }};"
             for i, (x, y, z) in enumerate(rng.uniform(-0.05, 0.05, size=(2500, 3)))]
    st = ft.parse_and_eval("\n".join(lines) + "\nlet scene = " + " + ".join(f"s{i}" for i in range(2500)) + ";\n")
    pts = np.concatenate([_points(6000, r) for r in (0.8, 1.5, 8.0)])
    ref, _, _ = oracle.distance(st, pts, accel=1, precision=32)
    err = np.abs(_distances(st, pts) - ref)
    assert (err <= 1e-5 * np.maximum(1.0, np.abs(ref))).all(), (float(err.max()), pts[err.argmax()])


def test_tree_whose_grids_are_dropped():
    """1200 nearly concentric spheres pass the cap of 2^26 list entries: the
    tree keeps no grid and is evaluated through its BVH or its whole fold."""
    from test_scene_build import _overlapping_spheres

    st = ft.parse_and_eval(_overlapping_spheres(1200))
    size = ctypes.c_uint64()
    assert _native.lib().ft_scene_device_bytes(st.gpu().handle, ctypes.byref(size)) == 0
    assert size.value < 8 * 2 ** 26
    pts = np.concatenate([_points(700, r) + np.float32([0, 1, 0]) for r in (0.8, 1.5, 8.0)])
    ref, _, _ = oracle.distance(st, pts, accel=1, precision=32)
    err = np.abs(_distances(st, pts) - ref)
    assert (err <= 1e-5 * np.maximum(1.0, np.abs(ref))).all(), (float(err.max()), pts[err.argmax()])


def test_adjoint_in_chunks_of_rays():
    """More rays than one pass of the adjoint takes (2^22): the sum of the
    views' own gradients, up to the order of the FP32-weighted FP64 sums."""
    ps, vs = ft.ParamScene(workloads.shape_fit(n=16)), ft.ring_views(5)
    opts = workloads.shape_fit_options(1024)
    rng = np.random.default_rng(2)
    w = [rng.normal(size=(5, 1024, 1024)).astype(np.float32) for _ in range(2)]
    whole = ps.backward(vs, opts, w[0], w[1])
    parts = sum(ps.backward(vs[k:k + 1], opts, w[0][k:k + 1], w[1][k:k + 1]) for k in range(5))
    assert np.abs(whole).max() > 0
    assert np.abs(whole - parts).max() <= 1e-9 * np.abs(parts).max()


LEAVES = {"boolean": "let {n} = (Sphere {{ radius: 0.8, pos: vec3({x}, 0.6, 0) }}) - "
                     "(Box {{ size: vec3(0.9, 0.9, 0.9), pos: vec3({x}, 1.0, -0.3) }});",
          "prism": "let {n} = ExtrudePolygon {{ sides: 3, radius: 0.7, height: 0.8, pos: vec3({x}, 0.5, 0) }};",
          "turned": "let {n} = Box {{ size: vec3(0.9, 0.5, 0.7), round: 0.1, pos: vec3({x}, 0.7, 0), rot: vec3(20, 30, 10) }};",
          "hooked": "let {n} = Sphere {{ radius: 0.6, pos: vec3({x}, 0.6, 0), "
                    "distance_post: fn(d, p) {{ return abs(d) - 0.05; }} }};",
          "sphere": "let {n} = Sphere {{ radius: 0.6, pos: vec3({x}, 0.6, 0) }};"}


@pytest.mark.parametrize("kinds", [("boolean",), ("hooked",), ("prism",), ("boolean", "sphere"), ("sphere", "boolean"),
                                   ("prism", "sphere"), ("prism", "prism"), ("hooked", "turned"), ("boolean", "hooked")])
def test_scenes_of_one_or_two_leaves(kinds):
    """Every pairing of leaf kinds in the short form of one or two leaves:
    distances around the scene, and a depth frame and a trace whose hits find
    their leaves, against the f32 oracle."""
    lines = [LEAVES[k].format(n=f"l{i}", x=-0.9 + 1.8 * i) for i, k in enumerate(kinds)]
    st = ft.parse_and_eval(LIGHTS + "\n".join(lines) + "\nlet scene = " + " + ".join(f"l{i}" for i in range(len(kinds))) + ";\n")
    pts = np.concatenate([_points(8000, r) for r in (1.5, 6.0)])
    ref, _, _ = oracle.distance(st, pts, accel=1, precision=32)
    err = np.abs(_distances(st, pts) - ref)
    assert (err > 1e-5 * np.maximum(1.0, np.abs(ref))).sum() <= 2, (float(err.max()), pts[err.argmax()])
    opts = ft.RenderOptions(width=96, height=64, max_steps=256, max_dist=30.0, epsilon=1e-4, step_scale=0.7)
    img = ft.render_depth(st, opts, ft.AccelMode.Bvh, 1, want_material=True)
    t, m, mat, _, _ = oracle.render_depth(st, opts, 1, 1, 32)
    both = (img.mask == 1) & (m == 1)
    assert (img.mask == m).mean() >= 0.999 and both.mean() > 0.02
    assert (np.abs(img.t[both] - t[both]) <= 1e-4).mean() >= 0.999 and (img.material[both] == mat[both]).all()
    lin, _ = ft.render_trace(st, opts, ft.AccelMode.Bvh, 1, 2)
    rad, _, _ = oracle.render_trace(st, opts, 1, 1, 2, 32)
    assert radiance_rmse(lin, rad) <= 1e-3, radiance_rmse(lin, rad)
    # the same frames from a batch of such scenes alone, and mixed with a scene of a short form
    ball = ft.parse_and_eval(LIGHTS + "let scene = Sphere { radius: 0.5, pos: vec3(0, 0.6, 0) };\n")
    for others in ([], [ball]):
        b = ft.Batch([(x, opts, 1, depth) for x in [st, *others] for depth in (0, 2)])
        b.launch()
        assert np.array_equal(b.read(0)["t"], img.t) and np.array_equal(b.read(0)["mask"], img.mask)
        assert np.allclose(b.read(1)["rgb"], lin, rtol=1e-3, atol=1e-4)  # the sums' order varies
        b.close()
