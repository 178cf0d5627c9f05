"""Rules of synchronisation that a missing line would break without a test run
noticing (the hardware mostly gets away with it), checked on the kernels' text."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mille-feuille_b200", "csrc")


def _code(name):
    """The file without comments, so that text about a barrier does not count as one."""
    with open(os.path.join(CSRC, name)) as f:
        s = f.read()
    return re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", s, flags=re.S))


def _body(code, head):
    """The braces' content of the first function whose header starts with `head`."""
    at = code.index(head)
    i = code.index("{", at)
    depth, j = 1, i + 1
    while depth:
        depth += {"{": 1, "}": -1}.get(code[j], 0)
        j += 1
    return code[i + 1:j - 1]


def test_cluster_kernels_meet_before_the_first_remote_store():
    """CUDA allows access to another block's shared memory only once that block has
    started: a cluster barrier comes before everything that can lead to a
    cluster_store."""
    code = _code("solver_dev.cuh")
    assert "cluster_store(" in _body(code, "__device__ void block_partial(")
    body = _body(code, "k_solve(SolverParams P)")
    first_use = min(body.index(w) for w in ("block_partial(", "solve_barrier(", "if (P.x0_given)"))
    assert "if constexpr (CL) cluster_barrier();" in body[:first_use]
