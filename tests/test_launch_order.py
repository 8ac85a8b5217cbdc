"""What the passes of grids that are not powers of two read before their
dependent-launch wait, from their source (no GPU): positions and draw indices of
a call may be written by the kernel directly before the call's first pass, so
that pass (ROW_LOAD_SRC) waits before ``gen_row_op``, which reads them."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "wideanglepropagation_b200", "csrc")


def _body(source, kernel):
    """The text of `kernel` between its braces, without comments."""
    with open(os.path.join(CSRC, source)) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    at = text.index("{", text.index(kernel + "("))
    depth, end = 0, at
    while True:
        depth += {"{": 1, "}": -1}.get(text[end], 0)
        if depth == 0:
            return text[at:end]
        end += 1


@pytest.mark.parametrize("source,kernel", [("wap_generic.cu", "gen_row_kernel"), ("wap_bluestein.cu", "blue_row_kernel")])
def test_first_pass_waits_before_it_reads_positions(source, kernel):
    body = _body(source, kernel)
    before = body[:body.index("gen_row_op(")]
    flag = re.search(r"bool (\w+) = a\.flags & ROW_LOAD_SRC;", before)
    assert flag, "the first pass is not told apart before gen_row_op"
    assert f"if ({flag.group(1)}) pdl_wait_then_release();" in before[flag.end():]
    assert "a.shifts" not in before and "a.draw" not in before
