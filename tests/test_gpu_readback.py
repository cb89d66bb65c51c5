"""Read-outs through pinned chunks: fields and populations against each other at sizes with one chunk, many
chunks, rows and columns longer than a chunk, several threads' worth of data, and callers in
several threads."""
import threading

import numpy as np
import pytest

import lbgpu
from helpers import same

pytestmark = pytest.mark.gpu


def channel(lx, ly, precision="f64", steps=3):
    lat = lbgpu.Lattice(lx, ly, precision, "pull")
    lat.setup_cylinder(lx // 5 + 1, ly // 2 + 1, max(1, ly // 10), 0.03, 50.0, lbgpu.WALL_REGULARIZED,
                       lbgpu.OUTLET_CONST)
    lat.step(steps)
    return lat


def fields_of(f):
    """The library's sums in its order, in FP64."""
    f = f[1:-1, 1:-1]
    top, mid, bot = (f[..., 2] + f[..., 5]) + f[..., 6], (f[..., 0] + f[..., 1]) + f[..., 3], (f[..., 4] + f[..., 7]) + f[..., 8]
    rho = (top + mid) + bot
    ux = (((f[..., 1] + f[..., 5]) + f[..., 8]) - ((f[..., 3] + f[..., 6]) + f[..., 7])) / rho
    return rho.T, ux.T, ((top - bot) / rho).T


@pytest.mark.parametrize("size", [(4, 4), (33, 9), (250, 51), (60000, 3), (4, 30000), (1400, 1001)])
def test_fields_and_populations_agree(size):
    with channel(*size) as lat:
        f = lat.populations()
        exp = fields_of(f)
        for a, b in zip(lat.macros(), exp):
            assert same(a, b)
        if size[0] * size[1] <= 262144:
            for a, b in zip(lat.macros_noalloc(), exp):
                assert same(a, b)
        lat.velocity_accumulate()
        lat.velocity_accumulate()
        ux, uy, k = lat.velocity_average()
        assert k == 2
        assert same(ux, (exp[1] + exp[1]) * 0.5) or np.allclose(ux, exp[1], rtol=0, atol=1e-15)
        assert np.allclose(uy, exp[2], rtol=0, atol=1e-15)


def test_callers_in_several_threads():
    sizes = [(1400, 1001), (250, 51), (900, 700), (64, 64)]
    lats = [channel(lx, ly, "f32", 5) for lx, ly in sizes]
    exp = [(lat.macros(), lat.populations()) for lat in lats]
    bad = []

    def read(i):
        for _ in range(5):
            m, f = lats[i].macros(), lats[i].populations()
            if not (all(same(a, b) for a, b in zip(m, exp[i][0])) and same(f, exp[i][1])):
                bad.append(i)

    team = [threading.Thread(target=read, args=(i,)) for i in range(len(lats))]
    for t in team:
        t.start()
    for t in team:
        t.join()
    for lat in lats:
        lat.close()
    assert not bad
