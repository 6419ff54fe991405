"""Voxelization with a tile's x-slabs on 8, 4 and 2 warps, and with whole tiles (the
number follows from the listed tiles and the grid), bit for bit against the CPU oracle:
overlapping spheres (list order matters), moving over several calls, tiles at ragged
edges, and tiles whose bin overflows (every sphere re-collected by every slab)."""
import numpy as np
import pytest

from helpers import small_suspension

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,n,rmin,rmax,prec", [
    ((24, 20, 28), 6, 3.0, 4.0, 0),            # 8 slabs
    ((17, 33, 9), 5, 2.0, 3.5, 1),             # 8 slabs, ragged tiles
    ((24, 24, 24), 700, 1.0, 2.0, 0),          # 8 slabs, overflowing bins
    ((66, 60, 63), 60, 5.0, 8.0, 1),           # 4 slabs
    ((96, 90, 97), 110, 7.0, 9.0, 0),          # 2 slabs
    ((121, 120, 126), 260, 7.0, 9.0, 1),       # whole tiles
])
def test_slabs_match_oracle(gpu, oracle, shape, n, rmin, rmax, prec):
    p = small_suspension(shape, n, rmin, rmax, seed=n, overlap=True, v_std=0.4)
    gl = gpu.Lattice(*shape, 1.5, precision=prec, max_particles=n, max_tag=n, max_radius=10.0)
    ol = oracle.OracleLattice(*shape, 1.5)
    for step in range(3):
        x = p.x + step * p.v
        gl.set_particles(x, p.v, p.w, p.r, p.tag)
        ol.set_particles(x, p.v, p.w, p.r, p.tag)
        st = ol.state()
        assert np.array_equal(gl.get_field(gpu.FIELD_SUBCELL_COUNT), st["n"])
        assert np.array_equal(gl.get_field(gpu.FIELD_PARTICLE_ID), st["id"])
    assert gl.device_errors() == 0
    gl.close()
