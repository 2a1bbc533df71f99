"""The kernels take correctly rounded reciprocals from the toolchain
(__frcp_rn), and none refines the hardware's approximation by itself: the only
use of that instruction is the 16-bit z-pass's, as it stands (its error, at
most 1 ulp, is far below the storage's)."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "inverse_solver_b200", "csrc")


def test_hardware_reciprocal_is_used_in_one_place():
    uses = {}
    for path in glob.glob(os.path.join(CSRC, "*.cu*")):
        code = re.sub(r"//[^\n]*", "", open(path).read())
        n = len(re.findall(r"rcp\.approx|__fdividef|__frcp_r[zud]\b", code))
        if n:
            uses[os.path.basename(path)] = n
    assert uses == {"cols_pipe.cu": 1}
