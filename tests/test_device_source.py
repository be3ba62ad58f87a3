"""Rules of the device code that a run cannot show: a violation depends on how
a warp's lanes happen to be scheduled, and its outcome would be a hang."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pbbsbench_b200", "csrc")


def body_of(source, head):
    """The braces' content of the function whose text starts with `head`."""
    at = source.index(head)
    at = source.index("{", at)
    depth = 0
    for i in range(at, len(source)):
        depth += {"{": 1, "}": -1}.get(source[i], 0)
        if depth == 0:
            return source[at: i + 1]
    raise AssertionError("unbalanced braces after " + head)


def test_the_set_pass_gives_up_by_whole_warps():
    """Each lane of a warp loads the error word, and another warp may set it
    between two of the loads: the loads go through a warp vote before anything
    returns on them, as warp collectives and a block sum follow."""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "mis.cu")).read())
    body = body_of(text, "bool settle(")
    looks = re.findall(r"[^;{}]*sync\.error[^;{}]*;", body)
    loads = [s for s in looks if "ld_" in s or "volatile" in s]
    assert loads and all(re.search(r"__any_sync\(\s*FULL\s*,", s) for s in loads), loads
