"""Which way runs of pull steps take: tiles with and without boundary rules off the perimeter, and lattices whose
shape decides between tiles and single steps, each against single steps bit for bit."""
import numpy as np
import pytest

import lbgpu
from helpers import describe_diff, same

pytestmark = pytest.mark.gpu


def run(lx, ly, storage, plan, outlet=lbgpu.OUTLET_CONST, rules=()):
    """Populations after the runs of `plan`; rules: (X, Y, tag) nodes of boundary rules."""
    obst = (lx // 5 + 1, ly // 2 + 1, max(1, ly // 10))
    with lbgpu.Lattice(lx, ly, lbgpu.storage_form(storage)[0], "pull") as lat:
        lbgpu.configure_storage(lat, storage, 0.03, 9)
        lat.setup_cylinder(*obst, 0.03, 2.0, lbgpu.WALL_REGULARIZED, outlet)
        if rules:
            omega, tag, bc, zgb = lbgpu.build_cylinder(lx, ly, *obst, 0.03, 2.0, lbgpu.WALL_REGULARIZED, outlet,
                                                       populations=False)[:4]
            tag = np.array(tag).reshape(lx + 2, ly + 2)
            for X, Y, t in rules:
                tag[X, Y] = t
            lat.set_geometry(omega, tag, bc, zgb)
        for n in plan:
            lat.step(n)
        return lat.populations()


# sizes with tiles off the perimeter in every shape; left-wall nodes (their table is filled) at and around tile corners
@pytest.mark.parametrize("storage,lx,ly", [
    ("f32", 150, 60), ("f32", 401, 160), ("f32", 700, 200), ("f32", 1030, 700), ("f16", 150, 60), ("f16", 401, 160),
    ("f16", 2100, 1500), ("f16r", 401, 160), ("bf16", 700, 200), ("f16b", 401, 160), ("f16br", 700, 200), ("f64", 401, 160)])
def test_some_tiles_have_boundary_rules(storage, lx, ly):
    rules = [(65, 25, 13), (64, 24, 5), (33, 33, 13), (lx // 2, ly // 2, 13), (lx - 4, ly - 4, 5), (lx // 2 + 40, ly // 2 + 1, 13)]
    got, exp = run(lx, ly, storage, [3, 15], rules=rules), run(lx, ly, storage, [1] * 18, rules=rules)
    assert same(got, exp), describe_diff(got, exp)
    assert not same(exp, run(lx, ly, storage, [1] * 18))      # the rules matter


# either side of the lines between tiles and single steps for lattices of a few long rows
WALLS = {True: lbgpu.WALL_REGULARIZED, False: lbgpu.WALL_BOUNCEBACK}      # rules along the rows, or not


@pytest.mark.parametrize("storage,lx,ly,tiles,rules", [c + (False,) if len(c) == 4 else c for c in [
    ("f64", 20001, 10, False), ("f64", 17001, 10, True), ("f64", 20000, 15, True), ("f64", 263001, 12, True),
    ("f64", 8003, 20, True), ("f64", 8003, 20, False, True), ("f64", 8003, 49, True, True), ("f64", 3001, 40, True, True),
    ("f32", 24003, 8, False), ("f32", 24003, 9, True), ("f32", 20000, 8, True),
    ("f32", 20003, 20, True), ("f32", 20003, 20, False, True), ("f32", 20003, 41, True, True), ("f32", 150001, 17, True, True),
    ("f16", 60001, 10, True), ("f16", 60001, 10, False, True), ("f16r", 60001, 5, False, True), ("f16b", 50001, 64, False, True),
    ("f16", 60001, 20, False), ("f16", 60001, 26, True), ("f16", 90001, 12, True), ("f16", 20003, 20, True),
    ("f16r", 60001, 20, False), ("f16r", 60001, 12, True), ("f16r", 21003, 35, False), ("f16r", 21003, 36, True),
    ("f16b", 20001, 20, False), ("f16b", 20001, 70, True), ("f16b", 5003, 40, True), ("bf16b", 30001, 4, False),
    ("f16br", 20001, 96, False), ("f16br", 5003, 40, True), ("f16br", 6001, 31, False),
    ("f64", 70, 50000, True), ("f64", 70, 62001, False)]])
def test_flat_lattices_take_the_faster_way(storage, lx, ly, tiles, rules):
    got, exp = run(lx, ly, storage, [3, 13]), run(lx, ly, storage, [1] * 16)
    assert same(got, exp), describe_diff(got, exp)
    with lbgpu.Lattice(lx, ly, lbgpu.storage_form(storage)[0], "pull") as lat:
        lbgpu.configure_storage(lat, storage, 0.03, 9)
        lat.setup_cylinder(9, 2, 1, 0.03, 2.0, WALLS[rules], lbgpu.OUTLET_CONST)
        lat.step(1)
        lat.step(16)
        assert (lat.last_launches < 16) == tiles


# channels with an extrapolated outlet in the wide and large shapes, one and two columns past a multiple of the tiles'
# width, and a channel whose many tiles are taken row by row
@pytest.mark.parametrize("storage,lx,ly,outlet", [
    ("f32", 769, 520, lbgpu.OUTLET_ZGB), ("f32", 2114, 1421, lbgpu.OUTLET_ZGB), ("f64", 2114, 1501, lbgpu.OUTLET_ZGB),
    ("f16", 770, 520, lbgpu.OUTLET_ZGB), ("bf16", 2113, 1421, lbgpu.OUTLET_ZGB), ("f32", 4099, 2300, lbgpu.OUTLET_CONST)])
def test_large_channels(storage, lx, ly, outlet):
    got, exp = run(lx, ly, storage, [1, 8, 3], outlet), run(lx, ly, storage, [1] * 12, outlet)
    assert same(got, exp), describe_diff(got, exp)
