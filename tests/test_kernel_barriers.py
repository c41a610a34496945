"""One lane's arrival on a shared-memory barrier speaks for its whole warp: it hands a stage back to
the copy engine or an accumulator to the tensor cores.  The other lanes' accesses are only ordered
before it by a __syncwarp() directly in front; without one the order rests on the warp happening to
be converged.  Read off the sources, as a missing one shows on no run that can be relied on."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "jdm-ghassan_v1_flach_b200", "csrc")
ARRIVE = re.compile(r"if \((lane|\(threadIdx\.x & 31\)) == 0\) mbar_arrive\(")


def arrivals():
    out = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        lines = [re.sub(r"//.*", "", l).strip() for l in open(path)]
        out += [(os.path.basename(path), i + 1, lines) for i, l in enumerate(lines) if ARRIVE.match(l)]
    return out


def test_the_pattern_finds_the_arrivals():
    """Every one-lane arrival of the sources is written in the form that the next test looks for."""
    text = "".join(open(p).read() for p in glob.glob(os.path.join(CSRC, "*.cu*")))
    assert len(re.findall(r"[^_]mbar_arrive\(&|[^_]mbar_arrive\(empty\)", text)) == len(arrivals()) > 8


@pytest.mark.parametrize("name,line,lines", arrivals(), ids=lambda v: str(v) if not isinstance(v, list) else "")
def test_warp_is_synchronised_before_one_lane_arrives(name, line, lines):
    before = [l for l in lines[:line - 1] if l][-1]
    assert before == "__syncwarp();", f"{name}:{line}: one lane arrives for the warp after '{before}'"
