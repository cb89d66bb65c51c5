"""Runs of pull steps (several steps a launch on tiles) against single steps.

The contract: lbgpu_step(n) leaves the state that n calls of lbgpu_step(1) leave, bit for bit, ghost ring
and stale slots included, in every storage type, whatever tile shape the size takes.  Sizes lie at
tile edges (one node more or less than a tile, one or two columns in the last tile) and on either
side of the node counts where the shape changes.
"""
import numpy as np
import pytest

import lbgpu
import oracle as O
from helpers import describe_diff, same

pytestmark = pytest.mark.gpu

SCALE = {"f16": 10, "bf16": 6}


def run(st, plan, precision, rs=None):
    with lbgpu.Lattice(st.lx, st.ly, precision, "pull") as lat:
        if precision in SCALE:
            lat.set_offset_scale(SCALE[precision])
        lat.set_geometry(st.omega, st.tag, st.bc, st.zgb)
        lat.set_populations(st.lat, st.tmp)
        if rs is not None:
            lat.set_stochastic_rounding(True, rs)
        for n in plan:
            lat.step(n)
        assert lat.steps_done == sum(plan)
        return lat.populations(), lat.macros(), lat.moments()


def agree(st, precision, plan, rs=None):
    one = run(st, [1] * sum(plan), precision, rs)
    got = run(st, plan, precision, rs)
    assert same(got[0], one[0]), (precision, st.lx, st.ly, describe_diff(got[0], one[0]))
    for a, b in zip(got[1], one[1]):
        assert same(a, b)
    assert same(got[2], one[2])
    return got[0]


EDGES = [(5, 4), (16, 8), (17, 9), (31, 25), (66, 33), (129, 17)]


@pytest.mark.parametrize("precision", ["f64", "f32", "f16", "bf16"])
@pytest.mark.parametrize("size", EDGES)
def test_every_boundary_rule_anywhere(precision, size):
    lx, ly = size
    st = O.random_boundary_lattice(lx, ly, seed=lx * 7 + ly)
    for i, t in enumerate(range(3, 19)):     # and off the perimeter
        st.tag[2 + (5 * i) % (lx - 2), 2 + (3 * i) % (ly - 2)] = t
    got = agree(st, precision, [1, 2, 9, 13, 20])
    if precision == "f64":
        exp = O.run(st, 45).lat
        assert same(got, exp), describe_diff(got, exp)


@pytest.mark.parametrize("precision", ["f64", "f32", "f16"])
@pytest.mark.parametrize("size", [(1, 1), (1, 9), (9, 1), (2, 2), (2, 17), (3, 3), (18, 2)])
def test_lattices_narrower_than_their_perimeter(precision, size):
    """One or two rows or columns: nodes with several sides at once, no interior at all."""
    st = O.random_boundary_lattice(size[0], size[1], seed=size[0] + 40 * size[1])
    got = agree(st, precision, [1, 2, 11])
    if precision == "f64":
        assert same(got, O.run(st, 14).lat)


# one and two columns past a multiple of every tile width, and a width below four columns
@pytest.mark.parametrize("precision", ["f64", "f32", "f16", "bf16"])
@pytest.mark.parametrize("size", [(17, 12), (34, 11), (65, 23), (130, 31), (67, 29)])
def test_extrapolated_outlet(precision, size):
    st = O.build_cylinder(O.Cylinder.reference_driver(*size))
    got = agree(st, precision, [1, 7, 12, 23])
    if precision == "f64":
        exp = O.run(st, 43).lat
        assert same(got, exp), describe_diff(got, exp)


def test_extrapolated_outlet_of_a_custom_geometry():
    """A pressure node of an extrapolated row before the row's end keeps single steps."""
    st = O.build_cylinder(O.Cylinder.reference_driver(40, 20))
    st.tag[20, 10] = 18
    got = agree(st, "f64", [3, 14])
    assert same(got, O.run(st, 17).lat)


# either side of the node counts where the tile shape changes
@pytest.mark.parametrize("precision,sizes", [
    ("f64", [(230, 90), (257, 160), (401, 310), (2100, 1500)]),
    ("f32", [(230, 90), (257, 240), (700, 200), (1030, 700)]),
    ("f16", [(230, 90), (401, 160), (1030, 130), (2100, 1500)]),
    ("bf16", [(230, 90), (401, 160), (1030, 130), (2100, 1500)]),
    ("f16r", [(401, 160), (1030, 130), (2100, 1500)]),
    ("bf16r", [(401, 160), (1030, 130)]),
    ("f16br", [(401, 160), (1030, 130), (2100, 1500)]),
    ("bf16s", [(401, 161), (1030, 129), (2100, 1500)]),
])
def test_every_tile_shape(precision, sizes):
    for lx, ly in sizes:
        def go(plan):
            with lbgpu.Lattice(lx, ly, lbgpu.storage_form(precision)[0], "pull") as lat:
                lbgpu.configure_storage(lat, precision, 0.03, 9)
                lat.setup_cylinder(lx // 5 + 1, ly // 2 + 1, ly // 10 + 1, 0.03, 80.0, lbgpu.WALL_REGULARIZED,
                                   lbgpu.OUTLET_CONST)
                for n in plan:
                    lat.step(n)
                return lat.populations()
        a, b = go([3, 15]), go([1] * 18)
        assert same(a, b), (precision, lx, ly, describe_diff(a, b))


@pytest.mark.parametrize("precision", ["f16", "bf16"])
def test_stochastic_rounding(precision):
    st = O.build_cylinder(O.Cylinder.baseline(150, 41))
    agree(st, precision, [1, 8, 13, 21], rs=7)


def test_infinite_and_nan_velocities_as_the_reference_has_them():
    """The short forms of the FP64 rules stand aside where 0 times a velocity is not 0."""
    st = O.random_boundary_lattice(40, 24, seed=11)
    f = st.lat.reshape(42, 26, 9)
    f[5, 5, 1] = np.inf
    f[20, 12, 2] = -np.inf
    f[30, 20, 0] = np.nan
    f[12, 18] = 0.0
    f[12, 18, 1] = 1e-3        # a density that nearly cancels
    f[12, 18, 3] = -1e-3
    f[33, 6, 5] = 1e200        # a velocity whose square overflows
    for steps in (1, 2, 5):
        got = run(st, [steps], "f64")[0]
        exp = O.run(st, steps).lat
        assert same(got, exp), steps


def test_row_shift_set_and_cleared_between_runs():
    """Row-shifted lattices keep a fourth slot of stale values with their table: clearing the shift moves what
    it holds."""
    st = O.random_boundary_lattice(70, 40, seed=4)

    def go(plan):
        with lbgpu.Lattice(70, 40, "f16", "pull") as lat:
            lat.set_offset_scale(12)
            lat.set_offset_shift(lbgpu.poiseuille_profile(40, 0.03))
            lat.set_geometry(st.omega, st.tag, st.bc, st.zgb)
            lat.set_populations(st.lat, st.tmp)
            seen = []
            for part in plan:
                for n in part:
                    lat.step(n)
                seen.append(lat.populations())
                lat.set_offset_shift(None)      # the stored values now mean something else; the bits stay
                seen.append(lat.populations())
                lat.set_offset_shift(lbgpu.poiseuille_profile(40, 0.03))
            return seen

    for a, b in zip(go([[3], [9], [2]]), go([[1] * 3, [1] * 9, [1] * 2])):
        assert same(a, b)


def test_steps_in_a_captured_graph_replay():
    """A caller that captures an even number of steps on the lattice's stream can replay them."""
    import torch

    def channel():
        lat = lbgpu.Lattice(150, 41, "f64", "pull")
        lat.setup_cylinder(31, 21, 5, 0.03, 60.0, lbgpu.WALL_BOUNCEBACK, lbgpu.OUTLET_CONST)
        lat.step(5)
        lat.synchronize()
        return lat

    torch.zeros(1, device="cuda")
    with channel() as lat, channel() as ref:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=torch.cuda.ExternalStream(lat.stream), capture_error_mode="thread_local"):
            lat.step(4)
        for _ in range(3):
            graph.replay()
        torch.cuda.synchronize()
        ref.step(12)
        assert same(lat.populations(), ref.populations())
        del graph
