"""Order of cluster barriers and remote shared-memory accesses, read from the kernels' source.

A CTA may touch another CTA's shared memory only once every CTA of the cluster has started executing.  A
kernel that skips that wait is right nearly always and loses a value without an error otherwise, so no run
shows it: the rule is checked where it is written."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "instinctflash_b200" / "csrc"
REMOTE = re.compile(r"mapa\.shared::cluster|st\.shared::cluster|ld\.shared::cluster|\bst_dsmem_f32\(|\bld_dsmem_f32\(|\bmap_to_cta\(|\bmbar_arrive_cluster\(")
STARTED = re.compile(r"\bcluster_wait\(\)|\bcluster_sync_all\(\)")


def kernel_bodies(text):
    """(name, body) of every __global__ function, comments removed."""
    text = re.sub(r"//[^\n]*", "", text)
    for head in re.finditer(r"__global__", text):
        brace = text.index("{", head.end())
        name = re.findall(r"(\w+)\s*\(", text[head.end():brace])
        depth, i = 1, brace + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        yield [n for n in name if n not in ("__launch_bounds__", "__cluster_dims__", "conditional_t")][-1], text[brace:i]


def remote_before_started(body):
    """True when the body reaches for another CTA's shared memory before any wait on the cluster barrier."""
    remote, started = REMOTE.search(body), STARTED.search(body)
    return remote is not None and (started is None or started.start() > remote.start())


@pytest.mark.parametrize("source", ["gemm_fp8_sm100.cu", "row_ops.cu", "attn_ops.cu"])
def test_remote_shared_memory_after_the_cluster_has_started(source):
    bodies = list(kernel_bodies((CSRC / source).read_text()))
    assert any(REMOTE.search(body) for _, body in bodies)
    assert [name for name, body in bodies if remote_before_started(body)] == []


def test_the_rule_finds_an_early_store():
    early = 'asm volatile("st.shared::cluster.u32 [%0], %1;"); cluster_sync_all();'
    assert remote_before_started("{" + early + "}")
    assert not remote_before_started("{ cluster_arrive(); cluster_wait(); " + early + "}")
