"""Memory order between the two CTAs of the pair kernel, as its source states it: no test run can show a missing order."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "coalsack_b200", "csrc")


def source(name):
    return re.sub(r"//.*", "", open(os.path.join(CSRC, name)).read())


def test_arrivals_on_the_other_cta_have_cluster_scope():
    arrivals = re.findall(r"mbarrier\.arrive[\w.:]*shared::cluster[\w.]*", source("csk_tile2.cuh"))
    assert arrivals
    for a in arrivals:
        assert re.search(r"\.(release|relaxed)\.cluster\.", a), a  # without: release, but to the arriving CTA only


def test_waits_for_both_ctas_acquire_from_the_cluster():
    s = source("csk_tile2.cuh")
    assert "mbarrier.try_wait.parity.acquire.cluster" in source("csk_common.cuh")
    for bar in ("bar_slot", "bar_acc_early", "bar_acc_free"):
        waits = re.findall(r"(\w+)\(%s\([^;]*?, " % bar, s)
        assert [w for w in waits if w.startswith("wait") or w.startswith("mbar_wait")] == ["wait_for_both"], (bar, waits)


def test_token_rows_report_to_the_cta_that_issues_the_mmas():
    """The other CTA's token rows are read by the leader's MMAs: their copies' own completion (which releases to the cluster) must
    reach the leader, not only an arrival by a thread that saw them land."""
    s = source("csk_tile2.cuh")
    loads = re.findall(r"tma_load_2d\w*\(st\b[^;]*;", s)
    assert len(loads) == 2
    for load in loads:
        assert load.startswith("tma_load_2d_pair(") and "leader_full0" in load, load
    assert "2u * 128u * (uint32_t)half" in s  # the leader expects both halves
