"""A CTA may touch another CTA's shared memory only once that one is known to
have started.  In csrc/batch.cu a kernel that works in teams first takes its
cluster from cluster_team(), which therefore has to be a meeting of the whole
cluster.  Read from the source: the fault that a missing meeting would be
depends on how late a CTA starts."""
import os
import re

from conftest import ROOT

SRC = os.path.join(ROOT, "nmag-src_gb300", "csrc", "batch.cu")


def _bodies():
    """Name -> body of each function at file scope, comments removed."""
    text = re.sub(r"//[^\n]*", "", open(SRC).read())
    heads = re.finditer(r"^(?:__device__|__global__)[^;{(]*?(?:__launch_bounds__\([^)]*\)\s*)?(\w+)\([^;{)]*\)\s*\{", text,
                        re.M)
    return {m.group(1): text[m.end():text.index("\n}", m.end())] for m in heads}


def test_the_cluster_meets_before_a_peer_is_touched():
    f = _bodies()
    assert "barrier.cluster.wait" in f["tsync"]
    assert re.search(r"\btsync\(", f["cluster_team"])
    assert "map_shared_rank" not in f["cluster_team"]
    for kernel in ("k_batch_run", "k_batch_eval"):
        assert f[kernel].index("cluster_team()") < f[kernel].index("next_team_particle(")
        assert "map_shared_rank" not in f[kernel]
