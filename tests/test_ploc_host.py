"""What the PLOC build must keep to on paths that no GPU run takes at will: its
kernels' source run block by block on the CPU, and its sizes at triangle counts
that no test builds."""
import re
import subprocess
from pathlib import Path

import pytest

TESTS = Path(__file__).resolve().parent
CSRC = TESTS.parent / "meturay_b200" / "csrc"
CUDA = Path("/usr/local/cuda")


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    """ploc.cu as C++ for the CPU, its launches replaced, with the checks of
    ploc_blocks.cpp."""
    source = re.sub(r"\b\w+<<<.*?>>>\(", "host_no_launch(", (CSRC / "ploc.cu").read_text(),
                    flags=re.S)
    folder = tmp_path_factory.mktemp("ploc")
    (folder / "ploc.cpp").write_text('#include "host_block.hpp"\n' + source +
                                     (TESTS / "ploc_blocks.cpp").read_text())
    out = folder / "ploc"
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-w", "-ffp-contract=off", f"-I{TESTS}",
                        f"-I{CUDA}/include", "-iquote", str(CSRC), str(folder / "ploc.cpp"), "-o",
                        str(out), f"-L{CUDA}/lib64", "-lcudart"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return out


@pytest.mark.parametrize("check", ["blocks", "arrays"])
def test_on_the_host(program, check):
    """blocks: a block acts on one reading of the give-up word; arrays: a build's
    arrays have their room at any triangle count."""
    r = subprocess.run([str(program), check], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
