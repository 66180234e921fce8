"""The roles of oz_cheb_kernel's CTA decide as one whether an order goes on.  The error word
is set by another CTA at any moment, so threads that each read it can see different values:
the threads of warps 2-7 that went on would wait at their named barrier for those that
left, without a limit, and the lanes of the MMA warp would part at a vote of all 32.  A
failure between two such reads cannot be timed on a device; the rule is checked on the
source."""
import os
import re

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dynemol_gb300", "csrc", "ozaki.cu")


def _text():
    return re.sub(r"//[^\n]*", "", open(SRC).read())


def test_the_grid_barrier_answers_from_one_thread():
    text = _text()
    body = text[text.index("grid_barrier_sub(unsigned *count, unsigned target, int *err,\n"):]
    body = body[:body.index("\n}\n")]
    one = body[body.index("if (threadIdx.x == 64) {"):]
    depth, end = 0, 0
    for end, ch in enumerate(one):
        depth += (ch == "{") - (ch == "}")
        if ch == "}" and depth == 0:
            break
    inside, after = one[:end], one[end:]
    assert '"l"(err)' in inside and "aborted" in inside
    assert "err" not in after and "abort" not in after and "bar.sync 2, 192" in after


def test_the_order_loop_has_one_answer_per_role():
    text = _text()
    loop = text[text.index("for (int k = 1; ok && k <= L.K; ++k) {"):]
    loop = loop[:loop.index("if (threadIdx.x == 0) {")]
    answers = re.findall(r"\bok = ([^;]*);", loop)
    assert len(answers) == 3
    assert answers[1].startswith("__all_sync(0xffffffffu, ")          # warp 1
    assert answers[2].startswith("c.grid_barrier_sub(") and "&&" not in answers[2]  # warps 2-7
