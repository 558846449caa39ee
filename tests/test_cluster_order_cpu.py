"""What one CTA of a cluster hands to another is ordered across the cluster: the default scope of an arrival or a wait is the CTA."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "runnburn_b200" / "csrc"


def sources():
    return {p.name: p.read_text() for p in sorted(CSRC.glob("*")) if p.suffix in (".cuh", ".cu", ".inc", ".hpp")}


def test_arrivals_at_another_cta_release_across_the_cluster():
    found = [(n, m.group(0)) for n, t in sources().items() for m in re.finditer(r"mbarrier\.arrive[\w.:]*shared::cluster[\w.:]*", t)]
    assert found
    fenced = "fence.release.sync_restrict::shared::cta.cluster;\\n\\tmbarrier.arrive.relaxed.cluster.shared::cluster"
    for name, text in sources().items():
        bare = text.replace(fenced, "")
        assert all(".release.cluster." in m for m in re.findall(r"mbarrier\.arrive[\w.:]*shared::cluster[\w.:]*", bare)), name


@pytest.mark.parametrize("file", ["prefill_gemm_pair.cuh", "dense.cuh"])
def test_waits_for_another_cta_acquire_across_the_cluster(file):
    """`full` of the matmuls on pairs of SMs: the odd CTA's stage, the even CTA's MMA warp waits."""
    text = sources()[file]
    mma = text[:text.index("pt_mma(tmem")]
    mma = mma[mma.rindex("if (rank == 0) {"):]
    assert "pt_wait_shared(&full[s]" in mma and "mbar_wait_bounded(&full" not in mma
    text = sources()["prefill_gemm_pair.cuh"]
    wait = text[text.index("bool pt_wait_in("):]
    wait = wait[:wait.index("\n}\n")]
    assert "try_wait.parity.acquire.cluster" in wait and "fence.acquire.sync_restrict::shared::cluster.cluster" in wait
