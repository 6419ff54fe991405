"""Batched FP32 domains whose rows end in a segment of at most half its cells (the odd phase
takes those tails two rows at a time): row lengths on both sides of every limit, odd and even
numbers of rows, walls and periodic wraps, one-row domains; each domain against a single
handle fed the same calls, over two steps of each streaming phase.

Bars: populations bit for bit (a cell's result does not depend on its place in a segment),
forces within 1e-5 of the largest (float partial sums in another order, 1e-7 each)."""
import numpy as np
import pytest

from helpers import rel_err
from test_batch import TAU, advance, make_batch, packed, particles, singles

pytestmark = pytest.mark.gpu

ROWS = [(1, 7), (20, 9), (32, 8), (33, 9), (64, 8), (65, 9), (96, 10), (97, 9), (130, 11), (161, 8)]


@pytest.mark.parametrize("per", [(0, 0, 1), (1, 1, 0)])
def test_batch_row_tails(gpu, per):
    doms = [{"shape": (8, ny, nz), "periodic": per, "omega": 1 / TAU, "max_particles": 8 if nz > 8 else 0,
             "n": 2 if nz > 8 else 0, "r": (1.5, 2.5)} for nz, ny in ROWS]
    doms.append({"shape": (6, 1, 70), "periodic": per, "omega": 1 / TAU, "max_particles": 0, "n": 0, "r": (1, 1)})
    parts = particles(doms, 3)
    B = make_batch(gpu, doms, gpu.PREC_FP32_DEV)
    Ls = singles(gpu, doms, gpu.PREC_FP32_DEV)
    for it in range(4):
        counts, rec = packed(gpu, parts)
        FB, TB = B.cycle(counts, rec, init_vel=(it == 0))
        FS, TS = [], []
        for k, (L, p) in enumerate(zip(Ls, parts)):
            if p is None:
                L.set_particles(np.zeros((0, 3)), np.zeros((0, 3)), np.zeros((0, 3)), np.zeros(0), np.zeros(0, np.int32))
                L.collide_and_stream()
            else:
                L.set_particles(p.x, p.v, p.w, p.r, p.tag, init_vel=(it == 0))
                L.collide_and_stream()
                F, T = L.get_forces()
                FS.append(F)
                TS.append(T)
            np.testing.assert_array_equal(B.get_populations(k), L.get_populations())
        assert rel_err(FB, np.concatenate(FS)) <= 1e-5
        assert rel_err(TB, np.concatenate(TS)) <= 1e-5
        advance(doms, parts)
    B.close()
    for L in Ls:
        L.close()
