"""The RK3 stages are programmatic dependent launches: a stage's grid is resident
while the stage before still writes the state and the boundary traces it will
read.  The read-only path (ld.global.nc, __ldg) is only defined for memory that
nothing writes during the grid's life, so the stage kernels must not use it."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dg-cfl-less-maxwell-solver_b200", "csrc")


def _code(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def test_no_read_only_loads_in_the_stage_kernels():
    assert not re.search(r"__ldg\s*\(|ld\.global\.nc", _code("rk3.cu"))


def test_no_read_only_qualifiers_on_the_stage_buffers():
    """const __restrict__ lets the compiler choose the read-only path by itself."""
    params = re.search(r"struct Rk3Params\s*{(.*?)};", _code("kernels.h"), re.S).group(1)
    trace = re.search(r"struct Rk3Trace\s*{(.*?)};", _code("kernels.h"), re.S).group(1)
    assert "__restrict__" not in params + trace
