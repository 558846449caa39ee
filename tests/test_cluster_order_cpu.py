"""What one CTA of a cluster hands to another is ordered across the cluster: the default scope of an arrival or a wait is the CTA."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "runnburn_b200" / "csrc"


def sources():
    return {p.name: p.read_text() for p in sorted(CSRC.glob("*")) if p.suffix in (".cuh", ".cu", ".inc", ".hpp")}


def test_arrivals_at_another_cta_release_across_the_cluster():
    found = [(n, m.group(0)) for n, t in sources().items() for m in re.finditer(r"mbarrier\.arrive[\w.:]*shared::cluster[\w.:]*", t)]
    assert found
    assert not [f for f in found if ".release.cluster." not in f[1]]


def test_waits_for_another_cta_acquire_across_the_cluster():
    """`full` of the K-quant matmul on pairs of SMs: the odd CTA arrives, the even CTA's MMA warp waits."""
    text = sources()["prefill_gemm_pair.cuh"]
    mma = text[text.index("if (rank == 0) {"):]
    mma = mma[:mma.index("pt_mma(")]
    assert "pt_wait(&full[s]" in mma and "mbar_wait_bounded(&full" not in mma
    assert "try_wait.parity.acquire.cluster" in text[text.index("bool pt_wait("):][:500]
