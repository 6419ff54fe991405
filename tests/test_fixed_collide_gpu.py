"""FP64 collide-stream on lattices whose cells mix values inside and outside the
fixed-point range, cells at rest (all zero) and solid cells, against the CPU oracle.

Bound: 1e-12 of the largest population, the bar of the other FP64 parity tests (both
sides round at about 1e-16 per step, over four steps).  The oracle runs on the CPU."""
import numpy as np
import pytest

from helpers import rel_err, small_suspension

pytestmark = pytest.mark.gpu

SHAPES = [((20, 18, 64), (1, 1, 1)), ((12, 14, 132), (1, 1, 1)), ((16, 18, 40), (0, 0, 0)), ((14, 16, 67), (1, 0, 1)),
          ((13, 15, 1), (1, 1, 1)), ((9, 11, 33), (0, 1, 0))]


def populations(shape, seed):
    rng = np.random.default_rng(seed)
    f = rng.standard_normal((19, *shape)) * 1e-3
    cells = rng.random(shape)
    f[:, cells < 0.05] = 0.0                                   # at rest
    f[:, (cells >= 0.05) & (cells < 0.08)] *= 1e-200           # below the range once scaled down
    f[:, (cells >= 0.08) & (cells < 0.10)] *= 1e-100
    big = (cells >= 0.10) & (cells < 0.15)                     # |f| >= 1/32
    f[3][big] = 0.04
    f[12][big] = -0.035
    return f


@pytest.mark.parametrize("shape,per", SHAPES)
def test_fixed_point_range_mixed(gpu, oracle, shape, per):
    omega = 1.0 / 0.62
    n = 5 if min(shape) > 10 else 0
    p = small_suspension(shape, n, 2.5, 3.5, seed=5, periodic=per, overlap=True, v_std=0.08, w_std=0.01) if n else None
    f0 = populations(shape, 11)
    gl = gpu.Lattice(*shape, omega, periodic=per, max_particles=64, max_tag=64, max_radius=8.0)
    ol = oracle.OracleLattice(*shape, omega, periodic=per)
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
            for a, b in zip(gl.get_forces(), ol.get_forces()):
                assert rel_err(a, b) <= 1e-11
    gl.close()


def test_rest_stays_at_rest(gpu):
    gl = gpu.Lattice(16, 12, 70, 1.7, periodic=(1, 0, 1))
    for _ in range(3):
        gl.collide_and_stream()
    assert not np.any(gl.get_populations())
    gl.close()
