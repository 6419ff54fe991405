"""An adjoint window runs forward exactly as the same calls of set_particles_device and
collide_and_stream made one by one, also when the spheres have moved since the last list: a
cell shared by two spheres can keep its old owner in the first voxelization of the new
places and change hands in the second.

Bars: voxel state and populations bit for bit, the loss and the last forces within 1e-12 of
the largest (double atomics in another order)."""
import numpy as np
import pytest
import torch

import workloads as W
from helpers import rel_err, small_suspension

pytestmark = pytest.mark.gpu

SHAPE, OMEGA = (32, 30, 36), 1.5


def moved_lists(seed):
    """Four lists of overlapping spheres, each moved from the one before."""
    p = small_suspension(SHAPE, 24, 3.0, 5.0, seed=seed, overlap=True, v_std=0.02)
    return [W.with_ghosts(W.Particles(p.x + 0.35 * k * np.sign(p.v), p.v, p.w, p.r, p.tag), SHAPE) for k in range(4)]


@pytest.mark.parametrize("nsteps,every,steady", [(1, 1, False), (2, 2, False), (5, 2, False), (5, 5, True)])
@pytest.mark.parametrize("form", ["fp64", "fp32"])
def test_window_is_its_calls(gpu, oracle, form, nsteps, every, steady):
    lists = moved_lists(2)
    ol = oracle.OracleLattice(*SHAPE, OMEGA)
    owners = []
    for q in lists + lists[-1:]:
        ol.set_particles(q.x, q.v, q.w, q.r, q.tag)
        owners.append(ol.state()["id"])
    assert np.any(owners[-1] != owners[-2])   # the scene has such cells
    p = lists[-1]
    rec = np.repeat(gpu.pack_records(p.x, p.v, p.w, p.r, p.tag)[None], nsteps, axis=0)
    if not steady:
        rec[:, :, 3:9] *= 1.0 + 0.1 * np.sin(0.7 * np.arange(nsteps))[:, None, None]
    weights = np.random.default_rng(1).normal(size=(nsteps, p.n, 6))
    lats = []
    for _ in range(2):
        lat = gpu.Lattice(*SHAPE, OMEGA, precision=gpu.PREC_FP64 if form == "fp64" else gpu.PREC_FP32_DEV,
                          max_particles=300, max_tag=32, max_radius=6.0)
        lat.init_equilibrium(0.0, (0.01, 0.0, 0.0))
        for q in lists[:-1]:
            lat.set_particles(q.x, q.v, q.w, q.r, q.tag)
            lat.collide_and_stream()
        lats.append(lat)
    calls, window = lats
    table = torch.from_numpy(rec).cuda()
    torch.cuda.synchronize()
    loss = 0.0
    for t in range(nsteps):
        calls.set_particles_device(p.n, table[t].data_ptr())
        calls.collide_and_stream()
        F, T = calls.get_forces()
        loss += float((weights[t] * np.concatenate([F, T], axis=1)).sum())
    scale = float(np.abs(weights).sum() * max(np.abs(F).max(), np.abs(T).max()))
    got = window.adjoint_window(rec, weights, every)
    for field in (gpu.FIELD_SUBCELL_COUNT, gpu.FIELD_PARTICLE_ID, gpu.FIELD_PARTICLE_VELOCITY, gpu.FIELD_POPULATIONS):
        assert np.array_equal(calls.get_field(field), window.get_field(field))
    for a, b in zip(window.get_forces(), calls.get_forces()):
        assert rel_err(a, b) <= 1e-12
    assert abs(got["loss"] - loss) <= 1e-12 * scale
    for lat in lats:
        lat.close()
