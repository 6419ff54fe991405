"""The FP64 collide-stream kernel on rows of an odd number of cells (not 16-byte aligned):
half-way bounce-back and periodic wraps on every axis and their corners, rows shorter than a
segment, of one segment and a remainder, one-cell-thick axes, with and without a body force,
over two steps of each streaming phase.

Bars of the other FP64 parity tests: populations within 1e-12 of the largest, forces
within 1e-11 (both sides round at about 1e-16 per step), against the CPU oracle."""
import numpy as np
import pytest

from helpers import rel_err, small_suspension

pytestmark = pytest.mark.gpu

CASES = [((3, 4, 1), (1, 1, 1)), ((1, 5, 3), (0, 0, 0)), ((4, 1, 5), (0, 1, 1)), ((9, 8, 31), (0, 0, 0)),
         ((9, 10, 33), (1, 0, 0)), ((10, 9, 63), (0, 1, 1)), ((8, 9, 65), (0, 0, 1)), ((9, 9, 67), (0, 0, 0)),
         ((8, 9, 127), (1, 1, 0)), ((9, 8, 129), (0, 0, 1)), ((8, 8, 131), (0, 0, 0)), ((9, 9, 65), (1, 1, 1))]


@pytest.mark.parametrize("force", [(0.0, 0.0, 0.0), (1e-5, -2e-5, 3e-5)])
@pytest.mark.parametrize("shape,per", CASES)
def test_odd_rows(gpu, oracle, shape, per, force):
    omega = 1.0 / 0.7
    rng = np.random.default_rng(sum(shape))
    f0 = rng.standard_normal((19, *shape)) * 1e-3
    n = 4 if min(shape) >= 8 else 0
    p = small_suspension(shape, n, 1.2, 2.2, seed=3, periodic=(1, 1, 1), overlap=True, v_std=0.02) if n else None
    gl = gpu.Lattice(*shape, omega, periodic=per, body_force=force, max_particles=16, max_tag=16, max_radius=4.0)
    ol = oracle.OracleLattice(*shape, omega, periodic=per, body_force=force)
    gl.set_populations(f0)
    ol.set_populations(f0)
    for _ in range(4):
        if p is not None:
            gl.set_particles(p.x, p.v, p.w, p.r, p.tag)
            ol.set_particles(p.x, p.v, p.w, p.r, p.tag)
        gl.collide_and_stream()
        ol.collide_and_stream()
        assert rel_err(gl.get_populations(), ol.get_populations()) <= 1e-12
        if p is not None:
            assert rel_err(gl.get_forces()[0], ol.get_forces()[0]) <= 1e-11
    assert gl.device_errors() == 0
    gl.close()
