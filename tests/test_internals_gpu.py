"""States that the C ABI cannot set, through a driver that sees the library's internals (internals_driver.cu), on a
B200. A wait that has timed out is not made to happen: the flag that it leaves is written by the host.
"""
import os
import shutil
import subprocess

import pytest

from conftest import PKG, ROOT

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def driver(nse, cuda, tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path_factory.mktemp("internals") / "internals_driver")
    subprocess.run([nvcc, "-O1", "-std=c++17", "--expt-relaxed-constexpr", "-gencode", "arch=compute_100a,code=sm_100a",
                    os.path.join(ROOT, "tests", "internals_driver.cu"), "-L", PKG, "-lnse2d_b200", "-Xlinker", "-rpath", "-Xlinker", PKG,
                    "-o", exe], check=True, capture_output=True, timeout=600)

    def run(*args):
        r = subprocess.run([exe, *map(str, args)], capture_output=True, text=True, timeout=120)
        assert r.returncode == 0, r.stderr
        return {k: float(v) for k, v in (ln.split() for ln in r.stdout.splitlines())}
    return run


@pytest.mark.parametrize("precision", [64, 32])
def test_a_run_after_a_wait_that_timed_out_says_so(nse, driver, precision):
    """The reason is NSE2D_HALT_NONFINITE (a host loop that waits for t_end would otherwise never end); a new state
    runs as ever."""
    got = driver("gave_up", precision)
    assert got["one_launch"] == 1
    assert int(got["reason"]) & nse.HALT_NONFINITE
    assert got["steps_of_a_void_state"] == 0
    assert got["reason_of_a_new_state"] == nse.HALT_BUDGET and got["steps_of_a_new_state"] == 5


def test_a_model_wait_that_timed_out_is_an_error_once(driver):
    """nse2d_cnn_gradients and nse2d_cnn_train_step return an error, the weights and the step count stay as they were,
    and the calls after it work: the next training step is the first one, to the bit."""
    got = driver("model_wait")
    assert got["gradients"] == -1 and got["train"] == -1
    assert got["gradients_after"] == 0 and got["loss_after_is_right"] == 1
    assert got["weights_kept"] == 1
    assert got["train_after"] == 0 and got["weights_after_are_the_first_steps"] == 1


@pytest.mark.parametrize("precision", [64, 32])
def test_steps_beside_another_channels_are_by_launches(driver, precision):
    """A step while another channel's steps are in flight on another stream is by launches, which overlap, and so is
    the next one of the channel that it came beside; in one launch otherwise. The same bits either way."""
    got = driver("shared", precision)
    assert got["one_launch"] == 1 and got["still_busy"] == 1
    assert got["by_launches_beside_another"] == 1
    assert got["by_launches_alone"] == 0
    assert got["first_channel_by_launches_0"] == 1 and got["first_channel_by_launches_1"] == 0
    assert got["same_bits"] == 1


def test_the_tuner_times_the_steps_that_a_plan_governs(driver):
    """On a grid whose steps go in one launch, every plan would time the same kernel: the tuner replays graphs there."""
    got = driver("autotune")
    assert got["one_launch"] == 1
    assert got["graphs_captured"] == 1
    assert got["one_launch_after"] == 1


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("Nx,Ny,rows", [(64, 65, 1), (64, 514, 4), (128, 129, 1), (128, 300, 3), (256, 514, 4), (512, 257, 2), (512, 514, 4),
                                        (1024, 131, 1), (1024, 300, 3), (1024, 446, 3), (1024, 513, 4), (1024, 514, 4), (1024, 515, 0),
                                        (64, 5, 0), (32, 129, 0), (2048, 257, 0)])
def test_the_grids_whose_steps_go_in_one_launch(driver, Nx, Ny, rows, precision):
    """64 to 1024 points by up to 514 rows, with as many bands as the solve has groups of columns: bands of one to four
    rows on 148 SMs."""
    got = driver("form", Nx, Ny, precision)
    assert got["rows_a_cta"] == rows and got["one_launch"] == (rows > 0)
