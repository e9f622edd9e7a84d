"""The host builder's trees, by area and by cost, are to the bit those of its
first, scalar form (of which the hashes below are), at node widths 2, 5 and 8
and 2 to 700 primitives; boxes with infinite bounds give valid trees."""
import hashlib
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "optix-path-tracer_gb300", "csrc")

TREES = {  # kind of boxes (host_builder_driver.cpp) -> md5 of its lines
    0: "0a3538d09b8ed55ced95c960ba821971",
    1: "8bae8ea974438f3e23471ddb7798d93c",
    2: "34967f043ef6ec6f571411a8e5c4a1eb",
    3: "e32fbc461e7801ab327852553082c13b",
    4: "1c94bb3d21dd2321ff7694f5179065d0",
    5: "134e6e814957af73f1afc38345441f81",
}


@pytest.fixture(scope="module")
def lines(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    exe = str(tmp_path_factory.mktemp("host_builder") / "driver")
    subprocess.run([cxx, "-std=c++17", "-O3", "-ffp-contract=off", "-fsanitize=address,undefined",
                    "-fno-sanitize=float-divide-by-zero", "-fno-sanitize-recover=undefined", "-I", CSRC,
                    os.path.join(HERE, "host_builder_driver.cpp"), os.path.join(CSRC, "bvh_host.cpp"),
                    "-o", exe], check=True)
    return subprocess.run([exe], capture_output=True, text=True, check=True).stdout.splitlines()


@pytest.mark.parametrize("kind", sorted(TREES))
def test_trees(lines, kind):
    own = [l for l in lines if l.startswith(f"hash {kind} ")]
    assert len(own) == 36
    assert hashlib.md5("\n".join(own).encode()).hexdigest() == TREES[kind]


def test_infinite_bounds(lines):
    assert lines[-1] == "nonfinite ok"
