"""A wait of the cooperative FP32 loops that runs out ends the solve as an error,
also where the iteration was its last one."""
import pytest

from test_gpu_failures import _apply_still_works

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [1, 2], ids=["mixed", "x64"])
@pytest.mark.parametrize("max_iterations", [1, 100])
def test_a_wait_that_runs_out_is_an_error(precision, max_iterations, gpu_lib):
    assert gpu_lib.esf_selftest_loop_wait(precision, max_iterations) == 3  # ESF_ERR_CUDA
    assert b"ran out" in gpu_lib.esf_last_error()
    _apply_still_works(gpu_lib)


def test_arguments(gpu_lib):
    assert gpu_lib.esf_selftest_loop_wait(0, 1) == 1
    assert gpu_lib.esf_selftest_loop_wait(1, 0) == 1
