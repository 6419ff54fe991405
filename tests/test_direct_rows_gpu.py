"""The FP32 collide-stream kernel that works without staging (rows that are not 16-byte
aligned): row lengths around the 64-cell segment and its 32-cell halves, one-cell-thick
axes, walls and periodic wraps on every axis, overlapping spheres, with and without a
body force, over two steps of each streaming phase.

Bars of the other FP32 parity tests: populations within 2e-5 of the largest (FP32
rounding of a few 1e-7 a step), forces within 1e-4, against the CPU oracle in double."""
import numpy as np
import pytest

from helpers import rel_err, small_suspension

pytestmark = pytest.mark.gpu

CASES = [((5, 4, 1), (1, 1, 1)), ((1, 7, 2), (1, 1, 1)), ((6, 1, 3), (0, 1, 0)), ((9, 8, 31), (0, 0, 1)),
         ((9, 10, 33), (1, 0, 0)), ((12, 11, 63), (1, 1, 1)), ((11, 12, 65), (0, 0, 0)), ((10, 9, 66), (0, 1, 1)),
         ((9, 12, 97), (1, 0, 1)), ((8, 9, 129), (0, 0, 1)), ((7, 8, 191), (1, 1, 0))]


@pytest.mark.parametrize("force", [(0.0, 0.0, 0.0), (1e-5, -2e-5, 3e-5)])
@pytest.mark.parametrize("shape,per", CASES)
def test_direct_rows(gpu, oracle, shape, per, force):
    omega = 1.0 / 0.7
    rng = np.random.default_rng(sum(shape))
    f0 = rng.standard_normal((19, *shape)) * 1e-3
    n = 4 if min(shape) >= 8 else 0
    p = small_suspension(shape, n, 1.2, 2.2, seed=3, periodic=(1, 1, 1), overlap=True, v_std=0.02) if n else None
    gl = gpu.Lattice(*shape, omega, periodic=per, precision=gpu.PREC_FP32_DEV, body_force=force, max_particles=16,
                     max_tag=16, max_radius=4.0)
    ol = oracle.OracleLattice(*shape, omega, periodic=per, body_force=force)
    gl.set_populations(f0.astype(np.float32))
    ol.set_populations(f0)
    for _ in range(4):
        if p is not None:
            gl.set_particles(p.x, p.v, p.w, p.r, p.tag)
            ol.set_particles(p.x, p.v, p.w, p.r, p.tag)
        gl.collide_and_stream()
        ol.collide_and_stream()
        assert rel_err(gl.get_populations(), ol.get_populations()) <= 2e-5
        if p is not None:
            assert rel_err(gl.get_forces()[0], ol.get_forces()[0]) <= 1e-4
    assert gl.device_errors() == 0
    gl.close()
