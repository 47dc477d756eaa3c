"""The short scene forms and the structures behind them, where they can go
wrong: the GPU's FP32 distance in every region of the candidate grids (cells,
cells inside a solid, the outer grid, the far walk) against the f32 oracle,
which walks the leaf BVH and folds whole trees; the path tracer's passes
against one pass.  (The adjoint's near-primitive fold is held to FP64 by the
differentiation tests.)"""
import numpy as np
import pytest

import forgedthoughts_gb300 as ft
import oracle
from forgedthoughts_gb300 import workloads

pytestmark = pytest.mark.gpu

GROUND = workloads.GROUND


def _points(n=6000, reach=2.5, far=30.0):
    rng = np.random.default_rng(5)
    near = rng.uniform([-reach, -0.4, -reach], [reach, reach, reach], size=(2 * n, 3))
    outer = rng.uniform([-2 * reach, -0.4, -2 * reach], [2 * reach, 2 * reach, 2 * reach], size=(n, 3))
    beyond = rng.uniform([-far, 0.0, -far], [far, far, far], size=(n, 3))
    return np.concatenate([near, outer, beyond]).astype(np.float32)


def _assert_distances(src, what):
    # two FP32 evaluations of one formula differ by a few rounding steps of the
    # coordinates (up to 110 for the ground): 1e-5 of the distance or of 1, as
    # for the union_round grids
    st = ft.parse_and_eval(src)
    g = st.gpu()
    g.build_bricks(0.25)
    pts = _points()
    _, exact = g.brick_bounds(pts)
    ref, _, _ = oracle.distance(st, pts, accel=1, precision=32)
    err = np.abs(exact.astype(np.float64) - ref)
    assert (err <= 1e-5 * np.maximum(1.0, np.abs(ref))).all(), (what, float(err.max()), pts[err.argmax()])


KINDS = ["Sphere {{ radius: 0.4, pos: vec3({x}, 0.5, {z}) }}",
         "Box {{ size: vec3(0.5, 0.7, 0.3), pos: vec3({x}, 0.4, {z}), rot: vec3(0, 35, 0) }}",
         "Box {{ size: vec3(0.6, 0.5, 0.4), round: 0.1, pos: vec3({x}, 0.6, {z}) }}",
         "Cylinder {{ radius: 0.3, height: 0.8, pos: vec3({x}, 0.5, {z}) }}",
         "Torus {{ major_radius: 0.4, minor_radius: 0.1, pos: vec3({x}, 0.5, {z}) }}",
         "Box {{ size: vec3(0.4, 0.6, 0.5), pos: vec3({x}, 0.5, {z}), rot: vec3(20, 15, 40) }}",
         "Sphere {{ radius: 0.5, shell: 0.1, pos: vec3({x}, 0.4, {z}) }}"]


def _objects(n):
    rng = np.random.default_rng(n)
    return [f"let p{i} = " + KINDS[i % len(KINDS)].format(x=f"{rng.uniform(-1.8, 1.8):.4f}",
                                                         z=f"{rng.uniform(-1.8, 1.8):.4f}") + ";" for i in range(n)]


@pytest.mark.parametrize("ground", [False, True])
@pytest.mark.parametrize("n", [1, 2, 4, 5, 40])
def test_hard_union_distance(n, ground):
    """One primitive, a pair, all evaluated at every point, and candidate
    grids; overlapping solids, whose inside depends on the walk's order."""
    src = "\n".join(([GROUND] if ground else []) + _objects(n)) + "\nlet scene = " + " + ".join(
        (["ground"] if ground else []) + [f"p{i}" for i in range(n)]) + ";\n"
    _assert_distances(src, (n, ground))


@pytest.mark.parametrize("ground", [False, True])
@pytest.mark.parametrize("n,k", [(4, 0.05), (7, 0.3), (33, 0.15)])
def test_union_round_distance_of_all_kinds(n, k, ground):
    """A tree alone and beside a ground, with primitives outside the compact
    record's kinds, and blends of one, two and many near primitives."""
    lines, cur, level = _objects(n), [f"p{i}" for i in range(n)], 0
    while len(cur) > 1:
        nxt = []
        for j in range(0, len(cur) - 1, 2):
            lines.append(f"let u{level}_{j // 2} = {cur[j]}.union_round({cur[j + 1]}, {k});")
            nxt.append(f"u{level}_{j // 2}")
        cur, level = nxt + cur[len(cur) - len(cur) % 2:], level + 1
    src = "\n".join(([GROUND] if ground else []) + lines) + f"\nlet scene = {'ground + ' if ground else ''}{cur[0]};\n"
    _assert_distances(src, (n, k, ground))


@pytest.mark.parametrize("hooks", ["domain: twist", "distance_post: ripple", "domain: twist, distance_post: ripple"])
def test_hooked_leaf_forms(hooks):
    """Each form of the register evaluation of a hooked leaf, against depth
    frames of the oracle: same hits on 99.9 % of the pixels, depth within 1e-4."""
    from parity import assert_depth_parity

    w = workloads.twisted_shells(24, 3, 96, 64)
    st = ft.parse_and_eval(w.source.replace("domain: twist, distance_post: ripple", hooks))
    img = ft.render_depth(st, w.options, ft.AccelMode.Bvh, 1)
    t, m, _, _, _ = oracle.render_depth(st, w.options, 1, 1, 32)
    assert_depth_parity(img.t, img.mask, t, m, hooks)


@pytest.mark.parametrize("spp", [1, 4, 5, 9])
def test_path_passes_add_up(spp):
    """A threshold that no pixel reaches splits the samples into passes of
    min_spp; without one they are a single pass.  The same samples in the same
    order: equal to the bit."""
    w = workloads.union_round_field(n=16, seed=2, width=40, height=24, aa=1)
    st = ft.parse_and_eval(w.source)
    one = ft.render_pathtrace(st, w.options, w.accel, ft.PathtraceSettings(spp=spp, min_spp=4, noise_threshold=0.0))
    many = ft.render_pathtrace(st, w.options, w.accel,
                               ft.PathtraceSettings(spp=spp, min_spp=min(4, spp), noise_threshold=1e-30))
    moved = many[2] == spp  # a black pixel has no error and stops at min_spp
    assert (one[2] == spp).all() and moved.any()
    assert np.array_equal(one[0][moved], many[0][moved]) and np.array_equal(one[1][moved], many[1][moved])
