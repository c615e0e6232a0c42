"""The mixed pair-tensor kernel's hand-over between the two blocks of a cluster, read from its source: block 1
passes the completion of its bulk copies on to block 0, whose products read block 1's shared memory, so the
arrival has to release and block 0's wait to acquire at cluster scope."""
import re
from pathlib import Path

SOURCE = (Path(__file__).resolve().parents[1] / "threebodymdalgorithms_b200" / "csrc" / "tbmd_pairs.cu").read_text()


def body(name):
    m = re.search(r"\b%s\([^;{]*\)\s*\n\{.*?\n\}" % name, SOURCE, re.S)
    assert m, name
    return m.group(0)


def test_arrivals_for_copies_release_at_cluster_scope():
    remote = re.findall(r"(\w+)\(&S\.full\[[^\]]*\], 0\)", SOURCE)
    assert remote, "no arrival at the other block's `full` barriers"
    for name in remote:
        assert "mbarrier.arrive.release.cluster.shared::cluster.b64" in body(name), name


def test_wait_before_products_acquires_at_cluster_scope():
    issue = SOURCE[SOURCE.index("if (warp == 9 && lane == 0 && rank == 0)"):]
    issue = issue[:issue.index("mma_bf16(D")]
    waits = re.findall(r"bar_wait(<\w+>)?\(&S\.full", issue)
    assert waits == ["<true>"]
    assert "CLUSTER ? bar_try_cluster(b, parity) : bar_try(b, parity)" in body("bar_wait")
    assert "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64" in body("bar_try_cluster")


def test_relaxed_arrivals_hand_over_nothing_but_tmem():
    for name in re.findall(r"__device__ __forceinline__ void (\w+)\(", SOURCE):
        if "arrive.relaxed" in body(name):
            used = re.findall(r"\b%s\(&S\.(\w+)" % name, SOURCE)
            assert set(used) == {"acc_empty"}, name
