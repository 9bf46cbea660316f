"""The batched solver's on-chip kernel against two rules that no run can be relied on to show broken, read from its
source: a CTA's shared memory may only be touched by others once its cluster has passed a barrier, and a value is
broadcast under a mask that holds the lane it comes from."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _function(name):
    """Body of a function of batch.cu, comments taken out."""
    txt = open(os.path.join(ROOT, "fenics-rs_b200", "csrc", "batch.cu")).read()
    txt = re.sub(r"//[^\n]*", "", txt)
    at = txt.index("{", re.search(rf"\b{name}\(", txt).start())
    depth, end = 0, at
    while True:
        depth += {"{": 1, "}": -1}.get(txt[end], 0)
        end += 1
        if depth == 0:
            return txt[at:end]


def test_cluster_barrier_comes_before_the_first_remote_access():
    body = _function("k_batch_resident")
    assert "map_shared_rank" in _function("resident_sum")
    first = min(body.index("resident_sum<"), body.index("map_shared_rank"))
    # a barrier of the kernel's own top level, not one of a branch that some instances take
    barrier = body.index("cl.sync()")
    assert barrier < first
    assert body[:barrier].count("{") - body[:barrier].count("}") == 1
    assert barrier < body.index("for (")


def test_the_next_instance_is_broadcast_under_a_whole_warps_mask():
    body = _function("k_batch_resident")
    assert "__activemask" not in body
    ticket = body[body.index("atomicAdd(next"):]
    assert ticket.index("__shfl_sync(BFULL, v, 0)") < ticket.index("map_shared_rank(&turn")
