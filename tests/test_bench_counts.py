"""The bench's whole-loop fraction counts the propagations that a solve runs
(bench.propagations): the library's loop starts with iteration 2 from three
iterations on."""
import importlib.util
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _bench():
    spec = importlib.util.spec_from_file_location("bench_module", os.path.join(ROOT, "bench.py"))
    m = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(m)
    return m


def test_propagations_follow_the_loop():
    b = _bench()
    src = open(os.path.join(ROOT, "inverse_solver_b200", "csrc", "odt_api.cu")).read()
    assert re.search(r"const int j0 = B >= 3 && [^;]* \? 2 : 1;", src)   # the loop runs jj = j0 .. B
    assert [b.propagations(n) for n in (0, 1, 2, 3, 40)] == [0, 1, 2, 2, 39]
    assert re.search(r"iteration_frac\": \(ITER_BYTES \* vox_step \* propagations\(s\.Bornmax\)", open(
        os.path.join(ROOT, "bench.py")).read())
