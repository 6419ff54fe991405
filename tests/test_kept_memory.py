"""Device memory that stays with a handle between adjoint windows: bounded over all handles,
given back on request, with the handle and when an allocation needs it."""
import subprocess

import numpy as np
import pytest

from conftest import PKG, ROOT
from helpers import rel_err


def test_kept_blocks(tmp_path):
    exe = tmp_path / "kept_memory_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", f"-I{PKG / 'csrc'}", str(ROOT / "tests" / "kept_memory_check.cpp"),
                    "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True).stdout.strip() == "ok"


@pytest.mark.gpu
def test_window_memory_is_given_back(gpu):
    torch = pytest.importorskip("torch")
    rec = np.repeat(gpu.pack_records([[20.0, 21.0, 22.0]], [[0.01, 0.0, 0.0]], [[0.0, 0.0, 0.0]], [5.0], [1])[None], 6, axis=0)
    weights = np.ones((6, 1, 6))

    def window(lat):
        lat.init_equilibrium(0.0, (0.01, 0.0, 0.0))
        return lat.adjoint_window(rec, weights, 3)

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info(0)[0]

    lat = gpu.Lattice(64, 64, 64, 1.5, max_particles=4, max_tag=4, max_radius=6.0)
    lat.adjoint_release()   # nothing kept yet
    first = window(lat)     # (and first-use costs)
    lat.adjoint_release()
    own, before = lat.device_bytes(), free()
    second = window(lat)
    kept = lat.device_bytes() - own
    assert kept > 5 * 19 * 8 * 64**3 and before - free() >= kept
    third = window(lat)
    assert lat.device_bytes() - own == kept
    lat.adjoint_release()
    assert lat.device_bytes() == own and free() == before
    for k in first:   # (double atomics in another order)
        assert rel_err(second[k], first[k]) <= 1e-10 and rel_err(third[k], first[k]) <= 1e-10
    window(lat)
    lat.close()
    assert free() > before
