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
