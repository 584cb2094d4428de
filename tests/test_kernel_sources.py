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
