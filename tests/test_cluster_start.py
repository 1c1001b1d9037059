"""The order of the cluster GMRES's barriers, read from its source (none of it shows on a GPU except by chance).

A block of a cluster may store to another block's shared memory only after that block has started, which a
barrier of the whole cluster ensures: on every path it comes before the first of the stores (put_part), both
outside the functions that only define them.  And a warp reaches an .aligned barrier converged: after a branch
of single threads a __syncwarp or __syncthreads comes first."""
import os
import re

import cms2d_b200

SRC = os.path.join(os.path.dirname(cms2d_b200.__file__), "csrc", "cms_gmres_cluster.cuh")


def _kernel_body(text):
    start = text.index("{", text.index("k_gmres_cluster(GmcArgs<T> Ain)"))
    depth = 0
    for k in range(start, len(text)):
        depth += {"{": 1, "}": -1}.get(text[k], 0)
        if depth == 0:
            return text[start + 1:k]


def _without_local_functions(body):
    """The statements the kernel runs itself: the bodies of its named lambdas taken out."""
    out, k = "", 0
    for m in re.finditer(r"auto \w+ = \[[^\]]*\]\([^;{]*\{", body):
        if m.start() < k:
            continue
        out += body[k:m.start()]
        depth, k = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(body[k], 0)
            k += 1
    return out + body[k:]


def test_cluster_barrier_before_first_remote_store():
    body = re.sub(r"//[^\n]*", "", open(SRC).read())
    body = _without_local_functions(_kernel_body(body))
    first_store, barrier = body.index("put_part("), body.index("gmc_sync()")
    assert "map_shared_rank" not in body  # remote stores are made by put_part only
    assert barrier < first_store
    assert body[:barrier].count("{") == body[:barrier].count("}")  # not inside a branch or a loop


def test_warps_reach_aligned_barriers_converged():
    body = re.sub(r"//[^\n]*", "", open(SRC).read())
    fn = body[body.index("void gmc_sync()"):]
    fn = fn[:fn.index("\n}")]
    assert fn.count(".aligned") == 2
    before = fn[:fn.index("barrier.cluster.arrive")]
    assert max(before.rfind("__syncwarp()"), before.rfind("__syncthreads()")) > before.rfind("if (")
