"""The row-driven sweep passes solution values between CTAs of one launch with no
flag beside them: a value is its own readiness mark.  That is sound only if every
value moves whole, by relaxed accesses of its own size, and if the mark is one
pattern of the whole value.  Read from the source (a torn double cannot be made
to appear on demand)."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dg-cfl-less-maxwell-solver_b200", "csrc")


def _source():
    with open(os.path.join(CSRC, "kinetic.cu")) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def _body(src, head):
    """The braces that follow the first match of `head`."""
    m = re.search(head, src)
    assert m, head
    i = src.index("{", m.end())
    depth, j = 0, i
    while True:
        depth += {"{": 1, "}": -1}.get(src[j], 0)
        j += 1
        if depth == 0:
            return src[i:j]


def test_the_mark_is_the_whole_double():
    body = _body(_source(), r"bool unwritten\(double v\)")
    assert "hiint" not in body and "longlong" in body


def test_rows_move_by_relaxed_accesses_of_whole_values():
    src = _source()
    for t, elem in (("double", "v2.f64"), ("float", "v4.f32")):
        part = _body(src, r"struct RowPart<%s>" % t)
        for op in ("load_relaxed", "store_relaxed"):
            ops = re.findall(r"(?:ld|st)\.[a-z.]*global\.[a-z0-9.]+", _body(part, op + r"\("))
            assert ops and all(o.endswith("relaxed.gpu.global." + elem) for o in ops), (t, op, ops)


def test_waiting_and_gathering_use_them():
    src = _source()
    wait = _body(src, r"bool warp_gather_wait\(")
    assert "unwritten(load_relaxed(last))" in wait and ".u32" not in wait
    assert re.search(r"warp_gather<F, T, ACC, (BD, )?true>", wait)
    flow = _body(_body(src, r"void warp_gather\("), r"if \(FLOW\)")
    assert "load_relaxed" in flow and "memcpy_async" not in flow
    assert re.search(r"if \(FLOW\)\s*v\.store_relaxed", _body(src, r"void warp_solve\("))


def test_the_first_level_is_an_ordinary_launch():
    """Levels stage right-hand side and boundary data ahead of their grid dependency
    wait.  The first one's are written by the kernels just before it, so it must not
    start early; the later ones' are then complete."""
    body = _body(_source(), r"int launch_kin_sweep\(")
    assert re.search(r"numAttrs = p\.item_begin > 0 \? 1 : 0;", body)
    stage = _body(_source(), r"void warp_stage\(")
    assert "p.bt" in stage and "p.yacc" in stage  # still staged ahead
