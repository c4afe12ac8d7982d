"""Host rules of the library that decide sizes and kernels, called directly
(tests/host_rules.cpp, linked against the library; no GPU)."""
import shutil
import subprocess
from pathlib import Path

import pytest

import xpcs_gpu as xg

HERE = Path(__file__).resolve().parent
ROOT = HERE.parent
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"

pytestmark = pytest.mark.skipif(not Path(NVCC).exists(), reason="nvcc not found")


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    xg.lib()
    exe = tmp_path_factory.mktemp("rules") / "host_rules"
    r = subprocess.run([NVCC, "-std=c++17", "-x", "cu", str(HERE / "host_rules.cpp"), "-I",
                        str(ROOT / "include"), "-I", str(xg.HERE / "csrc"), "-L",
                        str(xg.LIB.parent), "-lxpcs_gpu", "-Xlinker", f"-rpath={xg.LIB.parent}",
                        "-o", str(exe)], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr

    def call(*args):
        out = subprocess.run([str(exe), *map(str, args)], capture_output=True, text=True,
                             check=True, timeout=60).stdout
        return [float(x) for x in out.split()]
    return call


def test_no_sort_of_a_series_events_outgrows_its_transposes_histogram(rules):
    """A captured batch graph holds the histogram's address.  Sorts of at most
    the transpose's items fit what the transpose reserved, in tiles of 2,048
    and of 4,096 items, on both sides of where the tile changes."""
    n = [1, 2047, 2048, 4097, 1 << 20, (1 << 27) - 1, 1 << 27, (1 << 27) + 5, 1 << 31]
    words = rules("hist", *n)
    assert words == sorted(words)
    for k, w in zip(n, words):
        assert w >= 256 * -(-k // 2048) + 513


@pytest.mark.parametrize("pixels,mean,cap,by_thread", [
    (1 << 20, 3, 32, True), (1 << 20, 50, 80, True), (36864, 10, 32, True), (16384, 3, 32, True),
    (4096, 10, 32, False), (16384, 80, 112, False),
])
def test_caller_held_rows_choose_their_kernel_by_pixels_and_row_length(rules, pixels, mean, cap,
                                                                       by_thread):
    """Rows without a partition map: every pixel counts, so rows of many pixels
    keep a thread each and the mean row length picks the capacity."""
    assert rules("rows", pixels, pixels * mean, 4000) == [cap, cap if by_thread else 0]


@pytest.mark.parametrize("pixels,by_thread,alone", [(4096, 1, 48), (4096, 0, 0),
                                                    (1 << 20, 1, 48), (1 << 20, 0, 48)])
def test_a_tuned_series_of_few_pixels_keeps_a_capacity_that_was_chosen(rules, pixels, by_thread,
                                                                       alone):
    """The caller's row capacity, also one set after an autotune, and the thread
    form where the autotuner found it faster, hold for few pixels too."""
    assert rules("tuned", pixels, pixels * 20, 1000, by_thread) == [alone, 48]
