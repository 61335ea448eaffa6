"""The packed traversal against the exact one, both restated on the host
(packed_traversal.cpp): every closest hit and every any-hit answer is the same."""
import subprocess
from pathlib import Path

import pytest

TESTS = Path(__file__).resolve().parent
ROOT = TESTS.parent


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    out = tmp_path_factory.mktemp("packed") / "packed_traversal"
    subprocess.run(["g++", "-O3", "-std=c++20", "-mfma", "-ffp-contract=off", "-I", str(ROOT / "sol_b200" / "csrc"),
                    str(TESTS / "packed_traversal.cpp"), "-o", str(out)], check=True)
    return out


# lengths: directions of length 2^-100 to 2^79, some with components up to 2^-118 of the largest
@pytest.mark.parametrize("family", ["lengths"])
@pytest.mark.parametrize("seed", [1, 2])
def test_same_answers(program, family, seed):
    out = subprocess.run([str(program), family, "400000", str(seed)], check=True, capture_output=True, text=True).stdout
    rays, hits, closest, any_hit = map(int, out.split())
    assert rays == 400_000 and hits > rays // 2
    assert (closest, any_hit) == (0, 0)
