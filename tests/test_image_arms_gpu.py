"""Torques of the FP32 form on rows short enough for one segment of a row to hold both ends
of a sphere that wraps around the periodic z boundary (or that reaches past half of a short
row between walls): the ends take the arms of different images.  Rows on and off 16-byte
boundaries, rows on both sides of the length beyond which this cannot happen, single
lattices and batches, both streaming phases, with and without a body force.

Bar of the FP32 form's forces and torques: 1e-4 of the largest, against the FP64 oracle."""
import numpy as np
import pytest

import workloads as W
from helpers import rel_err

pytestmark = pytest.mark.gpu

OMEGA = 1.0 / 0.7


def scene(shape, per):
    nz = shape[2]
    x = np.array([[9.7, 9.2, nz - 4.6], [10.3, 28.4, 2.1]])
    r = np.array([8.0, 6.3])
    if not per[2]:
        x[:, 2], r[:] = (0.6, nz - 1.4), (nz / 2 + 1.3, nz / 2 + 0.6)
    v = np.array([[0.02, -0.01, 0.015], [-0.01, 0.02, 0.01]])
    w = np.array([[1e-3, 2e-3, -1e-3], [-2e-3, 1e-3, 1e-3]])
    return W.with_ghosts(W.Particles(x, v, w, r, np.array([1, 2], dtype=np.int32)), shape, per)


def populations(shape):
    return np.random.default_rng(shape[2]).standard_normal((19, *shape)) * 1e-3


CASES = [((20, 40, nz), per) for nz in (64, 65, 66, 68, 72, 75, 80, 84, 96, 132) for per in ((1, 1, 1), (0, 0, 1))]
CASES += [((34, 46, 14), (1, 1, 0)), ((34, 46, 16), (0, 0, 0))]


@pytest.mark.parametrize("force", [(0.0, 0.0, 0.0), (1e-5, -2e-5, 3e-5)])
@pytest.mark.parametrize("shape,per", CASES)
def test_image_arms(gpu, oracle, shape, per, force):
    p = scene(shape, per)
    gl = gpu.Lattice(*shape, OMEGA, periodic=per, body_force=force, precision=gpu.PREC_FP32_DEV, max_particles=16,
                     max_tag=16, max_radius=float(p.r.max()))
    ol = oracle.OracleLattice(*shape, OMEGA, periodic=per, body_force=force)
    f = populations(shape)
    gl.set_populations(f)
    ol.set_populations(f)
    for _ in range(4):
        gl.set_particles(p.x, p.v, p.w, p.r, p.tag)
        ol.set_particles(p.x, p.v, p.w, p.r, p.tag)
        gl.collide_and_stream()
        ol.collide_and_stream()
        for a, b in zip(gl.get_forces(), ol.get_forces()):
            assert rel_err(a, b) <= 1e-4
    gl.close()


def test_image_arms_batch(gpu, oracle):
    scenes = [scene(*c) for c in CASES]
    B = gpu.Batch([{"shape": s, "periodic": per, "omega": OMEGA, "max_particles": 16} for s, per in CASES],
                  precision=gpu.PREC_FP32_DEV, max_tag=16, max_radius=10.0)
    B.init_equilibrium(0.01, (0.01, -0.02, 0.015))
    ols = [oracle.OracleLattice(*s, OMEGA, periodic=per) for s, per in CASES]
    for ol in ols:
        ol.init_equilibrium(0.01, (0.01, -0.02, 0.015))
    counts = np.array([p.n for p in scenes], dtype=np.int32)
    rec = np.concatenate([gpu.pack_records(p.x, p.v, p.w, p.r, p.tag) for p in scenes])
    ends = np.cumsum(counts)
    for _ in range(4):
        got = B.cycle(counts, rec)
        for p, ol, e in zip(scenes, ols, ends):
            ol.set_particles(p.x, p.v, p.w, p.r, p.tag)
            ol.collide_and_stream()
            for a, b in zip(got, ol.get_forces()):
                assert rel_err(a[e - p.n:e], b) <= 1e-4
    B.close()
