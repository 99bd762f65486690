"""The branch-free quotients, roots and contact law of csrc/dem_law.cuh
(x_rcp, x_div, x_sqrt, contact_law_fast) give the bits of CUDA's correctly
rounded operations and of contact_law wherever they apply: every FP32
significand, random and nearly halfway FP32 and FP64 quotients, and contacts
over the whole range of overlaps, motions and histories, exact zeros and
values outside the fast form's range among them."""
import pathlib
import subprocess

import pytest

pytestmark = pytest.mark.gpu
HERE = pathlib.Path(__file__).resolve().parent
CSRC = HERE.parent / "discrete-element-method-for-packing-cuda-c-code_b200" / "csrc"


def test_fast_law_is_bit_exact(cuda):
    out = HERE / "lawcheck" / "_build"
    out.mkdir(exist_ok=True)
    exe = out / "lawfast"
    subprocess.run(["nvcc", "-O2", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-fmad=false",
                    f"-I{CSRC}", f"-I{HERE.parent / 'include'}", "-o", str(exe),
                    str(HERE / "lawcheck" / "lawfast.cu")], check=True)
    r = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=120)
    rows = {a: (int(b), int(c)) for a, b, c in (ln.split() for ln in r.stdout.split("\n") if ln)}
    assert set(rows) == {"rcp32", "sqrt32", "div32", "div64", "sqrt64", "law32", "law64"}
    assert all(bad == 0 for bad, _ in rows.values()), rows
    # the fast form takes the ordinary contacts (15.2 M draws, 5 of 16 kinds outside its range)
    assert rows["law32"][1] > 5_000_000 and rows["law64"][1] > 5_000_000, rows
