"""The FP64 form on a fluid whose density lies outside the fixed-point range (|f| >= 1/32 from
a tenth off one on), with and without spheres: warps with solid cells run the double routine
with the solid terms, the others without.

Bars: populations within 1e-12 of the largest and forces within 1e-11 against the CPU oracle
(those of the other FP64 parity tests); a fluid cell with only fluid around it the same bits
whether its warp holds solid cells or not."""
import numpy as np
import pytest

from helpers import rel_err, small_suspension

pytestmark = pytest.mark.gpu

SHAPES = [((12, 14, 64), (1, 1, 1)), ((13, 12, 96), (0, 0, 0)), ((12, 13, 67), (1, 0, 1)), ((12, 12, 33), (0, 1, 0))]


@pytest.mark.parametrize("force", [(0.0, 0.0, 0.0), (1e-5, -2e-5, 3e-5)])
@pytest.mark.parametrize("shape,per", SHAPES)
def test_dense_fluid(gpu, oracle, shape, per, force):
    omega = 1.0 / 0.62
    f0 = np.random.default_rng(sum(shape)).standard_normal((19, *shape)) * 1e-3
    f0[0] += 0.12 / 3 * (1 + 0.5 * np.cos(2 * np.pi * np.arange(shape[0]) / shape[0]))[:, None, None]   # 0.02 to 0.06
    p = small_suspension(shape, 2, 2.0, 2.5, seed=5, periodic=per, overlap=True, v_std=0.05)
    after = []
    for solid in (False, True):
        gl = gpu.Lattice(*shape, omega, periodic=per, body_force=force, max_particles=8, max_tag=8, max_radius=8.0)
        ol = oracle.OracleLattice(*shape, omega, periodic=per, body_force=force)
        gl.set_populations(f0)
        ol.set_populations(f0)
        for step in range(4):
            if solid:
                gl.set_particles(p.x, p.v, p.w, p.r, p.tag)
                ol.set_particles(p.x, p.v, p.w, p.r, p.tag)
            gl.collide_and_stream()
            ol.collide_and_stream()
            got = gl.get_populations()
            assert rel_err(got, ol.get_populations()) <= 1e-12
            if step == 0:
                after.append(got)
            if solid:
                for a, b in zip(gl.get_forces(), ol.get_forces()):
                    assert rel_err(a, b) <= 1e-11
        if solid:
            n = gl.get_field(gpu.FIELD_SUBCELL_COUNT)
        gl.close()
    near = np.zeros(shape, dtype=bool)
    for dx in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dz in (-1, 0, 1):
                near |= np.roll(n > 0, (dx, dy, dz), axis=(0, 1, 2))
    assert near.any() and not near.all()
    assert np.array_equal(after[0][:, ~near], after[1][:, ~near])
