"""The reverse step's row addresses: rows longer than one 64-cell run, walls and periodic wraps
on every axis and their corners, both streaming phases, against the float64 PyTorch model
differentiated over its full tape.  Bar of the other FP64 adjoint parity tests, 1e-10 of the
largest gradient (rounding of about 1e-16 a step and operation)."""
import pytest

pytest.importorskip("torch")

from helpers import rel_err  # noqa: E402
from test_adjoint import case, gpu_window, torch_grads, torch_model  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,periodic", [((14, 12, 67), (0, 0, 0)), ((12, 13, 130), (0, 1, 1)),
                                            ((13, 12, 64), (1, 0, 1)), ((12, 14, 65), (1, 1, 0)),
                                            ((12, 13, 129), (1, 1, 1))])
def test_adjoint_long_rows(gpu, oracle, shape, periodic):
    c = case(shape, periodic, 3, 21, 5)
    L, g_out, ol = gpu_window(gpu, oracle, c, K=3)
    ref = torch_grads(torch_model(ol, c), ol.get_populations(), c)
    with L:
        assert abs(g_out["loss"] - ref["loss"]) <= 1e-12 * abs(ref["loss"])
        assert rel_err(g_out["grad_vel"], ref["grad_vel"]) <= 1e-10
        assert rel_err(g_out["grad_body_force"], ref["grad_body_force"]) <= 1e-10
        assert abs(g_out["grad_tau"] - ref["grad_tau"]) <= 1e-10 * abs(ref["grad_tau"])
        assert rel_err(g_out["grad_f0"].reshape(19, -1), ref["grad_f0"].reshape(19, -1)) <= 1e-10
