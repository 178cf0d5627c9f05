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


def test_cluster_barrier_takes_whole_warps():
    """`.aligned` barriers need every lane of a warp at the same instruction; lanes that
    come from a branch (the stores of the first few) are not known to be."""
    body = _body(_code("solver_dev.cuh"), "__device__ __forceinline__ void cluster_barrier()")
    assert body.index("__syncwarp();") < body.index(".aligned")


def test_multi_column_reductions_leave_between_two_barriers():
    """Every reduction over several columns copies its sums to registers between two
    block barriers, after its warps' half-warps have met."""
    code = _code("multi.cu")
    for body in (_body(code, "__device__ void grid_collect_m("), _body(_body(code, "struct BlockSync {"), "reduce(")):
        tail = body[body.rindex("sh.bcast[wib] = a;"):]
        at = [m.start() for m in re.finditer(r"__syncthreads\(\);", tail)]
        assert len(at) == 2 and at[0] < tail.index("out[k] = sh.bcast[k]") < at[1]
    for body in (_body(code, "__device__ void block_partial_m("), _body(_body(code, "struct BlockSync {"), "reduce(")):
        assert body.index("__syncwarp();") < body.index("__shfl_xor_sync(")
    assert "sh.bcast" not in _body(code, "__device__ void cg_multi_body(")


def test_team_items_hand_over_without_shared_words():
    """A team's words come from its item, which nothing writes during the launch, and a
    block leaves its list with all its threads or with none."""
    code = _code("multi.cu")
    team = _body(code, "struct TeamSync {")
    assert "const BatchItem &it;" in team and "unsigned epoch;" in team
    body = _body(code, "k_batch(const __grid_constant__ BatchParams B)")
    assert sorted(re.findall(r"__shared__[^;]*;", body)) == ["__shared__ SharedM sh;", "__shared__ int next, stop;"]
    item = body[body.index("TeamSync sy{"):body.index("for (;;)")]
    assert item.index("stop = ") < item.index("__syncthreads();") < item.index("if (stop) return;")
    assert item.count("return;") == 1
