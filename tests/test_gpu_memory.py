"""Device memory that the library keeps between lattices is there for the next one, whatever its size."""
import pytest

import lbgpu

pytestmark = pytest.mark.gpu


def test_a_large_lattice_takes_what_the_pool_keeps():
    import torch

    torch.zeros(1, device="cuda")
    with lbgpu.Lattice(64, 64, "f64") as alive:
        alive.setup_cylinder(9, 9, 3)
        free = torch.cuda.mem_get_info()[0]
        fill = torch.empty(free - (400 << 20), dtype=torch.uint8, device="cuda")     # 400 MB are left
        small = [lbgpu.Lattice(1000, 800, "f32") for _ in range(4)]                  # 58 MB each: from the pool
        for lat in small:
            lat.close()
        left = torch.cuda.mem_get_info()[0]
        try:
            with lbgpu.Lattice(2000, 1000, "f64") as lat:                            # 290 MB
                lat.setup_cylinder(400, 500, 100)
                lat.step(3)
                lat.velocity_accumulate()
                assert lat.moments()[0] > 0
        finally:
            del fill
            torch.cuda.empty_cache()
        assert left < 300 << 20       # (or the pool kept nothing and the test shows nothing)
