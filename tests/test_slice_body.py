"""The device body of a fused iteration (csrc/gsc_fused_body.cuh) on the CPU,
its threads resumed in chosen orders: what the barriers leave open must not
change a result, whichever thread of a block runs ahead."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NATIVE = os.path.join(ROOT, "tests", "native")
CSRC = os.path.join(ROOT, "gpu-inner-outer_b200", "csrc")
CUDA_INCLUDE = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")


def compiled(tmp_path_factory, name):
    cxx = shutil.which("g++")
    if not cxx or not os.path.exists(os.path.join(CUDA_INCLUDE, "cuda_runtime.h")):
        pytest.skip("no C++ compiler or CUDA headers")
    exe = str(tmp_path_factory.mktemp(name) / name)
    subprocess.run([cxx, "-O1", "-std=c++17", "-w", "-I", CUDA_INCLUDE, "-I", NATIVE, "-I", CSRC, "-o", exe,
                    os.path.join(NATIVE, name + ".cpp")], check=True)
    return exe


@pytest.fixture(scope="module")
def slice_check(tmp_path_factory):
    return compiled(tmp_path_factory, "slice_check")


def run(exe, *args):
    r = subprocess.run([exe] + [str(a) for a in args], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.startswith("ok"), (args, r.returncode, r.stdout)
    return int(r.stdout.split()[1])


@pytest.mark.parametrize("order", range(5))
@pytest.mark.parametrize("rows,cells,inputs,per_pass,threads", [
    (64, 40, 24, 8, 512),    # eight threads a row, more hits in a pass than are noted
    (100, 20, 40, 16, 256),  # two a row
    (4, 40, 24, 8, 32),      # a warp
])
def test_lowest_input_over_passes(slice_check, order, rows, cells, inputs, per_pass, threads):
    """Every input of the second pass satisfies every active state, none of
    the first does: the first of the second pass is the answer."""
    hits = run(slice_check, order, 1, rows, cells, inputs, per_pass, threads, 1)
    assert hits == rows * (cells // 4)


@pytest.mark.parametrize("order", range(3))
@pytest.mark.parametrize("seed", range(1, 4))
@pytest.mark.parametrize("rows,cells,inputs,per_pass,threads", [
    (64, 40, 24, 8, 512), (70, 33, 24, 24, 128), (17, 20, 24, 8, 32), (1, 64, 9, 4, 64),
])
def test_random_boxes(slice_check, order, seed, rows, cells, inputs, per_pass, threads):
    assert run(slice_check, order, seed, rows, cells, inputs, per_pass, threads) > 0


@pytest.mark.parametrize("seed", range(1, 4))
@pytest.mark.parametrize("rows,cells,inputs,per_pass,threads", [(64, 40, 24, 8, 512), (70, 33, 24, 24, 128),
                                                                (17, 20, 24, 8, 32)])
def test_valid_cells_of_windows_read_directly(slice_check, seed, rows, cells, inputs, per_pass, threads):
    """Where D' is read without dilated copies the valid set has none either,
    and its cells are looked up in the set itself."""
    assert run(slice_check, seed, seed, rows, cells, inputs, per_pass, threads, 0, 1) > 0


@pytest.mark.parametrize("order", range(3))
@pytest.mark.parametrize("rows,cells,inputs,per_pass,threads,block_rows", [
    (70, 40, 24, 8, 256, 16), (70, 40, 24, 8, 256, 24), (33, 20, 24, 24, 64, 8), (64, 33, 24, 8, 128, 32),
    (9, 20, 24, 8, 64, 8), (64, 40, 24, 8, 128, 40),
])
def test_rows_of_a_slice_in_several_blocks(slice_check, order, rows, cells, inputs, per_pass, threads, block_rows):
    """Blocks of whole bytes of row-lost bits, the last one shorter: each
    updates its rows alone and records them, and no other's."""
    assert run(slice_check, order, 2, rows, cells, inputs, per_pass, threads, 0, order % 2, block_rows) > 0


@pytest.fixture(scope="module")
def batch_check(tmp_path_factory):
    return compiled(tmp_path_factory, "batch_check")


@pytest.mark.parametrize("order", range(5))
@pytest.mark.parametrize("threads,warp", [(64, 0), (256, 0), (32, 1), (128, 1)])
def test_stopped_instances_beside_running_ones(batch_check, order, threads, warp):
    """A group that skips a stopped instance's tasks goes on to the next
    instance's record while some of its threads still read the stop flag."""
    assert run(batch_check, order, threads, warp) == 3 * 512
