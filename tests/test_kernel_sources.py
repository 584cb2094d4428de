"""Rules of the kernels that a run cannot show to be broken."""
import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_cluster_barrier_before_first_and_after_last_remote_access():
    """Another CTA's shared memory may be touched only once that CTA is known
    to run and while it has not left: every kernel that maps it passes a
    barrier of the whole cluster before the first access and after the last."""
    seen = 0
    for path in sorted(glob.glob(os.path.join(ROOT, "mxc_b200", "csrc", "*.cu"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for body in re.split(r"\b__global__\b", text)[1:]:
            body = body[:body.index("\n}")]
            use = [x.start() for x in re.finditer(r"\bmap_shared_rank\b", body)]
            if not use:
                continue
            seen += 1
            sync = [x.start() for x in re.finditer(r"\bcl\.sync\(\)", body)]
            assert sync and sync[0] < use[0] and sync[-1] > use[-1], path
    assert seen


def test_warps_with_tasks_of_their_own_do_not_meet_at_syncthreads():
    """__syncthreads() has to be the same statement for every thread of a
    block: a kernel whose preparing warp returns from its own loop uses the
    barrier instruction instead."""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(ROOT, "mxc_b200", "csrc", "k_sketch.cu")).read())
    body = next(x for x in re.split(r"\b__global__\b", text)[1:] if "k_sketch(" in x)
    body = body[:body.index("\n}")]
    assert "__syncthreads" not in body and body.count("sk_barrier()") == 4
