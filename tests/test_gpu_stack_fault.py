"""A stack whose column pass gave up waiting for a pair's operands has no valid map of that pair: the
collection says so, as zc_shift_map does, instead of returning the pair's peak. The fault word is written
into the pair's record from the host (tests/stack_fault.cpp, built here against the engine); no wait runs out."""
import subprocess
from pathlib import Path

import pytest

from zcmir_b200 import build

pytestmark = pytest.mark.gpu


def test_a_pairs_fault_word_fails_the_collection(tmp_path):
    exe, here = tmp_path / "stack_fault", Path(__file__).resolve().parent
    subprocess.run([build.nvcc(), *build.ARCH, "-std=c++17", "--expt-relaxed-constexpr", "-I", str(build.CSRC), "-I",
                    str(build.ROOT / "include"), "-x", "cu", str(here / "stack_fault.cpp"), "-o", str(exe),
                    "-L", str(build.HERE), "-l:libzcmir.so", "-Xlinker", f"-rpath={build.HERE}"], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    clean, *faults, stage, no_stage, last = r.stdout.splitlines()
    assert clean == no_stage == last == "1"
    assert len(faults) == 3 and all("inverse column pass gave up waiting" in x and f"pair {k + 1}" in x for k, x in enumerate(faults))
    assert "tensor-core column stage gave up waiting" in stage and "pair 2" in stage
