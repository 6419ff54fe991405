"""Particle lists that change from call to call: the tag -> slot map and the record table
exist twice and a new list clears the old one's entries, in eager calls and under stream
capture (where the whole map is cleared instead), for both widths of the prepare launch.

Bars as in the other FP64 parity tests: voxel state bit for bit, forces within 1e-11 of
the largest (1e-12 of the sum of the cell forces) against the CPU oracle; a replayed
graph against the same calls made eagerly, 1e-12 (summation order)."""
import numpy as np
import pytest
import torch

from helpers import rel_err, small_suspension

pytestmark = pytest.mark.gpu


def lists(shape, n, rmin, rmax):
    """The same spheres under other slots, tags and counts from call to call."""
    p = small_suspension(shape, n, rmin, rmax, seed=n, overlap=True, v_std=0.01)
    rng = np.random.default_rng(n)
    out = []
    for k in range(6):
        order = rng.permutation(n)
        tag = p.tag[order] + (n if k % 3 == 2 else 0)          # disjoint tags in every third list
        out.append((p.x[order] + 0.05 * k, p.v[order], p.w[order], p.r[order], tag.astype(np.int32)))
    out[3] = tuple(a[: max(1, n // 3)] for a in out[3])         # a shorter list
    return out


@pytest.mark.parametrize("shape,n,rmin,rmax", [((30, 28, 26), 5, 3.0, 4.0), ((64, 60, 52), 4100, 0.6, 1.0)])
def test_changing_lists(gpu, oracle, shape, n, rmin, rmax):
    gl = gpu.Lattice(*shape, 1.5, max_particles=n, max_tag=2 * n, max_radius=6.0)
    ol = oracle.OracleLattice(*shape, 1.5)
    for k, p in enumerate(lists(shape, n, rmin, rmax)):
        if k == 2:   # an empty list in between
            gl.set_particles(*[a[:0] for a in p])
        gl.set_particles(*p)
        ol.set_particles(*p)
        st = ol.state()
        assert np.array_equal(gl.get_field(gpu.FIELD_SUBCELL_COUNT), st["n"])
        assert np.array_equal(gl.get_field(gpu.FIELD_PARTICLE_ID), st["id"])
        named = np.isin(st["id"][st["n"] > 0], p[4]).all()
        gl.collide_and_stream()
        if not named:   # cells left behind by an earlier list: reported, as their tags are not mapped
            assert gl.device_errors() == gpu.DEVERR_UNMAPPED_TAG
            break
        ol.collide_and_stream()
        for a, b in zip(gl.get_forces(), ol.get_forces()):
            assert rel_err(a, b) <= 1e-11
    assert k >= 1
    gl.close()


def test_captured_lists(gpu):
    """Two steps captured once and replayed with other records in the same table."""
    shape, n = (30, 28, 26), 5
    tables = [torch.from_numpy(gpu.pack_records(*p)).cuda() for p in lists(shape, n, 3.0, 4.0) if len(p[3]) == n]
    tables = [t for t in tables if float(t[:, 10].max()) <= n]
    assert len(tables) >= 3
    eager = gpu.Lattice(*shape, 1.5, max_particles=n, max_tag=2 * n, max_radius=6.0)
    graphed = gpu.Lattice(*shape, 1.5, max_particles=n, max_tag=2 * n, max_radius=6.0)
    rec = tables[0].clone()
    ft = torch.zeros(6 * n, dtype=torch.float64, device="cuda")
    want = torch.zeros_like(ft)
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    graphed.set_stream(stream.cuda_stream)

    def two_steps(lat, table, out):
        for _ in range(2):
            lat.set_particles_device(n, table.data_ptr())
            lat.collide_and_stream()
        lat.get_forces_device(out.data_ptr())

    two_steps(graphed, rec, ft)
    two_steps(eager, tables[0], want)
    graphed.synchronize()
    eager.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        two_steps(graphed, rec, ft)
    for t in tables[1:] + tables[:1]:
        rec.copy_(t)
        torch.cuda.synchronize()
        graph.replay()
        two_steps(eager, t, want)
        torch.cuda.synchronize()
        assert rel_err(ft.cpu(), want.cpu()) <= 1e-12
    # an eager list after the replays
    graphed.set_stream(None)
    two_steps(graphed, tables[1], ft)
    two_steps(eager, tables[1], want)
    torch.cuda.synchronize()
    assert rel_err(ft.cpu(), want.cpu()) <= 1e-12
    graphed.close()
    eager.close()
