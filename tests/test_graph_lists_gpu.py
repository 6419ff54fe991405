"""Captured steps mixed with eager ones: a graph holds the addresses it was captured with, so
what it writes and reads has to be what the eager calls around it write and read.

Bars as for captured lists: forces within 1e-12 of the largest against the same calls made
eagerly on another handle (double atomics in another order); lists that change from call to
call within 1e-11 of the CPU oracle's forces, cells left without a particle reported as there."""
import numpy as np
import pytest
import torch

from helpers import rel_err, small_suspension

pytestmark = pytest.mark.gpu

SHAPE, N = (30, 28, 26), 5


class Pair:
    """A handle whose steps go through graphs, and one fed the same calls eagerly."""

    def __init__(self, gpu, form):
        prec = gpu.PREC_FP64 if form == "fp64" else gpu.PREC_FP32_DEV
        self.graphed, self.eager = (gpu.Lattice(*SHAPE, 1.5, precision=prec, max_particles=N, max_tag=2 * N,
                                                max_radius=6.0) for _ in range(2))
        p = small_suspension(SHAPE, N, 3.0, 4.0, seed=N, overlap=True, v_std=0.01)
        rng = np.random.default_rng(7)
        orders = [rng.permutation(N) for _ in range(6)]
        self.tables = [torch.from_numpy(gpu.pack_records(*(a[o] for a in (p.x, p.v, p.w, p.r, p.tag)))).cuda()
                       for o in orders]
        self.rec = self.tables[0].clone()
        self.ft, self.want = (torch.zeros(6 * N, dtype=torch.float64, device="cuda") for _ in range(2))
        self.stream = torch.cuda.Stream()
        torch.cuda.synchronize()
        self.graphed.set_stream(self.stream.cuda_stream)

    def two_steps(self, lat, out, table=None, n=N):
        for _ in range(2):   # the streaming phase comes back
            if table is not None:
                lat.set_particles_device(n, table.data_ptr())
            lat.collide_and_stream()
        lat.get_forces_device(out.data_ptr())

    def both(self, k):
        self.two_steps(self.graphed, self.ft, self.tables[k])
        self.two_steps(self.eager, self.want, self.tables[k])
        self.compare()

    def capture(self, table=None, n=N):
        self.graphed.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=self.stream):
            self.two_steps(self.graphed, self.ft, table, n)
        return graph

    def compare(self):
        self.graphed.synchronize()
        self.eager.synchronize()
        torch.cuda.synchronize()
        assert rel_err(self.ft.cpu(), self.want.cpu()) <= 1e-12
        assert self.graphed.device_errors() == self.eager.device_errors() == 0

    def close(self):
        self.graphed.set_stream(None)
        self.graphed.close()
        self.eager.close()


@pytest.fixture(params=["fp64", "fp32"])
def pair(gpu, request):
    p = Pair(gpu, request.param)
    yield p
    p.close()


@pytest.mark.parametrize("eager_first", [1, 2])
def test_replays_between_eager_lists(pair, eager_first):
    pair.both(0)
    graph = pair.capture(pair.rec)

    def replay(k):
        pair.rec.copy_(pair.tables[k])
        torch.cuda.synchronize()
        graph.replay()
        pair.two_steps(pair.eager, pair.want, pair.tables[k])
        pair.compare()

    def eager_list(k):
        for lat in (pair.graphed, pair.eager):
            lat.set_particles_device(N, pair.tables[k].data_ptr())

    for k in range(eager_first):
        eager_list(1 + k)
    replay(3)
    eager_list(4)   # an odd number of eager lists between the replays
    pair.two_steps(pair.graphed, pair.ft)
    pair.two_steps(pair.eager, pair.want)
    pair.compare()
    replay(5)
    pair.two_steps(pair.graphed, pair.ft)   # and a step of the list that the replay left
    pair.two_steps(pair.eager, pair.want)
    pair.compare()
    replay(2)
    pair.both(1)


def test_captured_steps_alone(pair):
    """A graph of the steps, replayed for lists that eager calls set."""
    pair.both(0)
    graph = pair.capture()
    for k in (1, 2, 3, 4):
        for lat in (pair.graphed, pair.eager):
            lat.set_particles_device(N, pair.tables[k].data_ptr())
        pair.graphed.synchronize()
        graph.replay()
        pair.two_steps(pair.eager, pair.want)
        pair.compare()


def test_capture_of_a_shorter_list(pair):
    """Capturing runs nothing: the lists before and after it follow one another."""
    pair.both(0)
    pair.capture(pair.rec, 2)
    pair.both(5)
    pair.both(2)
    pair.both(3)


def test_lists_of_other_lengths(gpu, oracle):
    """Longer, shorter, empty and disjoint lists, each compared in full."""
    p = small_suspension(SHAPE, N, 3.0, 4.0, seed=3, overlap=True, v_std=0.01)
    rng = np.random.default_rng(1)
    gl = gpu.Lattice(*SHAPE, 1.5, max_particles=N, max_tag=2 * N, max_radius=6.0)
    ol = oracle.OracleLattice(*SHAPE, 1.5)
    ft = torch.zeros(6 * N, dtype=torch.float64, device="cuda")
    for length, shift in ((N, 0), (N, 0), (2, 0), (N, N), (0, 0), (3, 0), (N, 0), (N, N), (N, 0)):
        o = rng.permutation(N)[:length]
        q = (p.x[o], p.v[o], p.w[o], p.r[o], (p.tag[o] + shift).astype(np.int32))
        gl.set_particles(*q)
        ol.set_particles(*q)
        gl.collide_and_stream()
        ol.collide_and_stream()
        gl.get_forces_device(ft.data_ptr())
        gl.synchronize()
        for got, want in zip(ft[:6 * length].cpu().numpy().reshape(2, length, 3), ol.get_forces()):
            assert rel_err(got, want) <= 1e-11
        st = ol.state()
        named = np.isin(st["id"][st["n"] > 0], q[4]).all()
        assert gl.device_errors() == (0 if named else gpu.DEVERR_UNMAPPED_TAG)
    gl.close()
