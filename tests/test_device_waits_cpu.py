"""No device wait's outcome is dropped: a kernel that goes on after a wait
expired has marked it, each warp for itself, and the host can see it.  (Read from
the sources: a wait that runs out is not something to provoke on a device.)"""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "cuda-bimp_b200" / "csrc"


def test_every_bounded_wait_is_checked():
    waits = 0
    for f in sorted([*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")]):
        for n, line in enumerate(f.read_text().splitlines(), 1):
            code = line.split("//")[0]
            if re.search(r"\bmbar_wait\(", code) and "mbar_wait(uint32_t" not in code:
                waits += 1
                # tested, or a drain after an expiry that is already marked
                assert re.search(r"(if|&&) \(?!?\(?mbar_wait\(|!mbar_wait\(|\(void\)mbar_wait\(", code), (f.name, n, line)
            assert not re.search(r"if \(t == 0\) atomicOr\(fault", code), (f.name, n, line)
    assert waits >= 4


def test_kernels_that_wait_take_the_fault_word():
    for f in sorted([*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")]):
        for k in re.split(r"(?=__global__ )", f.read_text())[1:]:
            if re.search(r"\bmbar_wait", k):
                head = k[:k.index("{")]
                assert "fault_word" in head, (f.name, head)
