"""The C-ABI runtime on the host alone (tests/c/host_runtime.cpp): the CUDA
runtime and the kernel launchers replaced by stand-ins that record what the
library asks for.  Copies happen as late as the CUDA runtime may do them, so a
host buffer that does not outlive its copy shows here and nowhere else."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "worldline-flux-tube-lattice_gb300")


@pytest.fixture(scope="module")
def runtime(tmp_path_factory):
    import build as pkg_build

    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path_factory.mktemp("host") / "host_runtime")
    subprocess.run([cxx, "-std=c++17", "-O1", "-I" + os.path.join(PKG, "csrc"),
                    "-I" + os.path.join(ROOT, "include"), "-I" + pkg_build.cuda_include(),
                    os.path.join(PKG, "csrc", "wl_api.cpp"),
                    os.path.join(PKG, "csrc", "wl_spline.cpp"),
                    os.path.join(ROOT, "tests", "c", "host_runtime.cpp"), "-o", exe],
                   check=True, capture_output=True, text=True)

    def run(scenario):
        r = subprocess.run([exe, scenario], capture_output=True, text=True, timeout=60)
        assert r.returncode == 0, r.stderr
        return {k: float(v) for k, v in (line.split() for line in r.stdout.splitlines())}

    return run


def test_proper_time_inputs_outlive_their_copy(runtime):
    r = runtime("tint_staging")
    assert r["released"] == 0 and r["rewritten"] == 0


def test_one_wait_per_sweep_of_the_loop_parallel_calls(runtime):
    r = runtime("loop_waits")
    assert r["ev"] == 1 and r["loops"] == 1 and r["rewritten"] == 0


def test_reported_launches_are_the_kernels_enqueued(runtime):
    r = runtime("launches")
    assert r["cut"] > 0 and r["off"] == 0


def test_batch_scratch_is_bounded(runtime):
    r = runtime("batch_scratch")
    assert r["largest"] <= r["chunk_sums"] + 256 * 2 ** 20
    assert r["small_per_loop"] == 1


def test_heavy_jobs_do_not_decide_the_cut_of_the_others(runtime):
    r = runtime("batch_side")
    assert r["alone"] == 1 and r["beside"] == 1


def test_ev_launches_nothing_for_the_lattice(runtime):
    """The legacy call holds no bounding boxes, which the lattice's kernels read."""
    r = runtime("ev_lattice")
    assert r["nan"] == 1 and r["kernels"] == 0


def test_sweep_grids_keep_the_unit_index_in_32_bits(runtime):
    assert runtime("sweep_grid")["ok"] == 1


def test_the_clamp_is_left_out_only_where_it_changes_no_bit(runtime):
    """smooth_clamp_idle() itself, against float32 sums over |z|^2 below the clamp."""
    r = runtime("clamp_idle")
    assert r["wrong"] == 0 and r["idle"] > 0


def test_which_launches_are_cut_into_single_loops(runtime):
    """(10: a launch alone on the chip, 1: one among others.)  Full chips of short
    loops, or of several fluxes, keep whole chunks: their loops' sums would cost up
    to a quarter of the walk."""
    assert runtime("cut_rule") == {"short_loops_full_chip": 0, "four_fluxes": 10, "scan": 11,
                                   "long_loops_full_chip": 11, "heavier_nodes": 11,
                                   "just_above_a_wave": 10, "few_units": 11, "many_waves": 0}
