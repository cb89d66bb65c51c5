"""Batches whose members take two steps a launch on tiles, against every member stepped alone, one step at a
time: odd and even counts, whole chunks and remainders, sizes at tile edges, AA members beside them, and
members that also step on their own between two batch calls (which leaves their buffers turned over)."""
import pytest

import lbgpu
import oracle as O
from helpers import describe_diff, same

pytestmark = pytest.mark.gpu

SIZES = [(5, 4), (64, 12), (65, 13), (33, 40), (130, 31)]
# batch steps, or (member, steps on its own)
PLANS = [[1, 2, 3, 20, 22], [(1, 2), 4, (2, 3), 5, 40, (0, 1), 2, 21], [6, (3, 4), (4, 5), 46]]


def make(size, precision, scheme):
    st = O.random_boundary_lattice(size[0], size[1], seed=size[0] + 3 * size[1])
    if size[0] > 20:
        st.tag[20, 5] = 14     # a boundary rule off the perimeter
    base, shift, rs = lbgpu.storage_form(precision)
    lat = lbgpu.Lattice(st.lx, st.ly, base, scheme)
    if base == "f16":
        lat.set_offset_scale(10)
    if rs and size[0] != 65:       # and one member that rounds to nearest
        lat.set_stochastic_rounding(True, size[0])
    if shift:
        lat.set_offset_shift(lbgpu.shift_profile(shift, size[1], 0.03))
    lat.set_geometry(st.omega, st.tag, st.bc, st.zgb)
    lat.set_populations(st.lat, st.tmp)
    return lat


@pytest.mark.parametrize("precision", ["f64", "f32", "f16", "f16r", "f16sr"])
@pytest.mark.parametrize("plan", PLANS)
def test_members_equal_single_steps(precision, plan):
    kinds = [(s, "pull") for s in SIZES] + [((70, 20), "aa")]
    lats = [make(s, precision, k) for s, k in kinds]
    alone = [make(s, precision, k) for s, k in kinds]
    done = [0] * len(kinds)
    with lbgpu.Batch(lbgpu.storage_form(precision)[0]) as b:
        for lat in lats:
            b.add(lat)
        for p in plan:
            if isinstance(p, tuple):
                lats[p[0]].step(p[1])
                done[p[0]] += p[1]
            else:
                b.step(p)
                done = [d + p for d in done]
        b.synchronize()
        for lat, ref, n, k in zip(lats, alone, done, kinds):
            assert lat.steps_done == n
            for _ in range(n):
                ref.step(1)
            got, exp = lat.populations(), ref.populations()
            assert same(got, exp), (precision, k, describe_diff(got, exp))
    for lat in lats + alone:
        lat.close()
