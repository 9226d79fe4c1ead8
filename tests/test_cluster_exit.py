"""A kernel whose CTAs write into one another's shared memory (shared::cluster) must not
let a CTA exit while another may still send to it, also where a bounded wait gave up
and the CTAs run apart.  Such a failure is not produced on a device: the sources are
read instead."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "differentiable-flowmap_b200", "csrc")


def _kernels(text):
    """(name, body) of every __global__ function."""
    for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\s*\(", text):
        i = text.index("{", m.end())
        depth, j = 1, i + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[j], 0)
            j += 1
        yield m.group(1), text[i:j]


@pytest.mark.parametrize("name", ["k_mg_coarse", "k_pcg_cluster"])
def test_ends_with_a_cluster_barrier(name):
    with open(os.path.join(CSRC, "fm_mg_cluster.cuh")) as f:
        bodies = dict(_kernels(f.read()))
    body = re.sub(r"//[^\n]*", "", bodies[name])
    after = body[max(body.rindex(s) for s in ("vcycle();", "cl_sum<", "cl_st_async") if s in body):]
    both = "cl_cluster_sync();" in after
    assert both or after.find("cl_cluster_arrive();") >= 0
    assert both or after.find("cl_cluster_wait();") > after.find("cl_cluster_arrive();")
    end = after.rindex("cl_cluster_sync();" if both else "cl_cluster_wait();")
    assert "return" not in after[:end]  # every thread reaches it
