"""Host rules of the fused method's plan, on the CPU."""
import subprocess

import pytest

from test_slice_body import compiled


@pytest.fixture(scope="module")
def plan_check(tmp_path_factory):
    return compiled(tmp_path_factory, "plan_check")


@pytest.mark.parametrize("shape,nk,nl,levels,windows,direct", [
    ((4, 1000, 360, 900), 2, 2, 0b1111, 9, True),    # 2 * 2 * 4 copies of 324 M words: above 32-bit offsets
    ((4, 1000, 360, 900), 2, 2, 0b0111, 9, False),   # three levels: below
    ((4, 1000, 360, 900), 2, 2, 0b0111, 1, True),    # no wider than the set itself
    ((1, 1, 20000, 26000), 2, 1, 0b1, 9, False),     # slices of one word are held as four
    ((1, 1, 20000, 27000), 2, 1, 0b1, 9, True),
])
def test_dilated_copies_stay_within_their_offsets(plan_check, shape, nk, nl, levels, windows, direct):
    """Where a set has dilated copies, every word of them has a 32-bit offset."""
    out = subprocess.run([plan_check] + [str(v) for v in (*shape, nk, nl, levels, windows, 0)], capture_output=True,
                         text=True, check=True).stdout.split()
    assert bool(int(out[0])) == direct
    words = nk * nl * bin(levels).count("1") * shape[2] * shape[3] * ((shape[1] * ((shape[0] + 31) // 32) + 3) // 4 * 4)
    assert int(out[1]) == words
    assert direct or words < 2**32


@pytest.mark.parametrize("shape,cells,batched,direct", [
    ((20, 20, 16, 10), 6, 0, True),       # few further words: directly, whatever the window
    ((20, 20, 16, 10), 6, 1, False),      # beside others: windows of four cells only
    ((20, 20, 16, 10), 4, 1, True),
    ((65, 65, 100, 56), 5, 0, True),      # 16.7 MiB
    ((65, 65, 100, 57), 5, 0, False),     # 17.04
    ((65, 65, 100, 140), 4, 0, True),     # 31.4, of four cells
    ((65, 65, 100, 150), 4, 0, False),
])
def test_windows_read_directly(plan_check, shape, cells, batched, direct):
    out = subprocess.run([plan_check] + [str(v) for v in (*shape, 2, 2, 2, cells, batched)], capture_output=True,
                         text=True, check=True).stdout.split()
    assert bool(int(out[0])) == direct


@pytest.mark.parametrize("n0,n1,reps", [(64, 64, 36), (108, 46, 35), (45, 41, 36), (17, 300, 9), (250, 17, 36)])
@pytest.mark.parametrize("slices", [1, 7, 72, 143, 144, 148, 149, 168, 184, 185, 222, 223, 275, 296, 297, 300])
def test_parts_of_slices_are_resident_at_once(plan_check, n0, n1, reps, slices):
    """The parts that slices are split into (whole bytes of row bits) are one
    wave: at 64 registers a thread an SM holds 1,024 threads."""
    out = subprocess.run([plan_check, "shape"] + [str(v) for v in (n0, n1, slices, reps)], capture_output=True,
                         text=True, check=True).stdout.split()
    threads, rows, parts, wide = map(int, out)
    assert parts > 1 and wide and rows % 8 == 0 and (parts - 1) * rows < n1 <= parts * rows
    assert threads % 32 == 0 and 32 <= threads <= 384
    assert -(-slices * parts // 148) * threads <= 1024
