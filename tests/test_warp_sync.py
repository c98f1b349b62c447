"""Barriers that no result shows, looked for in the text.

CUDA orders the lanes' accesses to shared memory at barriers only; shuffles, votes and warp reductions exchange
registers.  A missing barrier shows in no result as long as the lanes run in step.  A block whose warps decide
differently to leave a loop waits at a barrier for ever, which no test may bring about on a GPU."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "poissonrecon_gpu_gb300", "csrc")


def _body(text, head):
    """The braces' contents after the first 'head'."""
    at = text.index("{", text.index(head))
    depth = 0
    for k in range(at, len(text)):
        depth += {"{": 1, "}": -1}.get(text[k], 0)
        if depth == 0:
            return text[at + 1:k], k + 1
    raise ValueError(head)


def _source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def test_bound_box_orders_the_neighbours_before_the_finer_terms():
    # a leaf that is one brick of edge 8 or 4 has no depth of the coarse loop: the path without the loop's body
    text, _ = _body(_source("iso.cu"), "signed char bound_box(")
    loop = "for (int d = r + 1; d <= dpoly; ++d)"
    _, end = _body(text, loop)
    path = text[:text.index(loop)] + text[end:]
    scatter = path.index("sm.id[0][(lane / 9)")
    reads = path.index("sm.id[cur][g]")
    assert scatter < reads
    assert re.search(r"__sync(warp|threads)\(\)", path[scatter:reads])


def test_flexible_cg_leaves_by_one_read_of_the_error_flag():
    # another depth's wait may set the flag between two threads' reads of it
    text, _ = _body(_source("flexcg.cu"), "k_fcg_all(FcgArgs a")
    reads = re.findall(r"[^\n;]*\*\s*\(volatile int\*\)\s*a\.err[^\n;]*", text)
    assert reads
    for r in reads:
        assert re.search(r"__syncthreads_(or|and)\(threadIdx\.x == 0 &&", r), r
