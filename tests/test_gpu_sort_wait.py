"""A radix-sort tile that waits in vain for the counts of a tile before it
(csrc/dem_sort.cu): it gives up after a bounded time and counts the records
itself, so the order stays the stable one."""
import pathlib
import subprocess

import pytest

pytestmark = pytest.mark.gpu
HERE = pathlib.Path(__file__).resolve().parent
CSRC = HERE.parent / "discrete-element-method-for-packing-cuda-c-code_b200" / "csrc"


def test_wait_that_runs_out(cuda):
    out = HERE / "lawcheck" / "_build"
    out.mkdir(exist_ok=True)
    exe = out / "sortwait"
    subprocess.run(["nvcc", "-O2", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", f"-I{CSRC}",
                    f"-I{HERE.parent / 'include'}", "-o", str(exe), str(HERE / "sortcheck" / "sortwait.cu")], check=True)
    r = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=120)
    rows = [tuple(map(int, ln.split())) for ln in r.stdout.split("\n") if ln]
    assert rows == [(4096, 0), (20 * 4096 + 1, 0), (39 * 8192 + 5, 0)], rows
