"""The branch-free FP64 quotients, reciprocals and roots of csrc/dem_law.cuh
on the operands where rounding is hardest, and the branch-free contact law
over all constants it is used for (moduli over 18 decades, friction over 6,
rolling lengths from 0 to 1,000, the ends of each range among them): the bits
of CUDA's rounded operations and of contact_law."""
import pathlib
import subprocess

import pytest

pytestmark = pytest.mark.gpu
HERE = pathlib.Path(__file__).resolve().parent
CSRC = HERE.parent / "discrete-element-method-for-packing-cuda-c-code_b200" / "csrc"


def test_hardest_operands_and_all_constants(cuda):
    out = HERE / "lawcheck" / "_build"
    out.mkdir(exist_ok=True)
    exe = out / "lawedge"
    subprocess.run(["nvcc", "-O2", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-fmad=false",
                    f"-I{CSRC}", f"-I{HERE.parent / 'include'}", "-o", str(exe),
                    str(HERE / "lawcheck" / "lawedge.cu")], check=True)
    r = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=120)
    rows = {a: (int(n), int(bad)) for a, n, bad in (ln.split() for ln in r.stdout.split("\n") if ln)}
    assert set(rows) == {"rcp64", "div64", "sqrt64", "law32", "law64"}
    assert all(bad == 0 for _, bad in rows.values()), rows
    assert rows["rcp64"][0] > 10_000_000 and rows["div64"][0] > 500_000 and rows["sqrt64"][0] > 10_000, rows
    assert rows["law32"][0] > 1_000_000 and rows["law64"][0] > 1_000_000, rows
