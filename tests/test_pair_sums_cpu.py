"""Which barrier stands between the CTA pair's copies and the warps that read them with ordinary loads. A missing order between two CTAs of a cluster
cannot be shown by running the kernel, so this reads its source."""
import re
from pathlib import Path

SOURCE = Path(__file__).resolve().parents[1] / "gcow_b200" / "csrc" / "ops" / "gemm2_tcgen05.cu"


def test_column_sums_read_only_what_their_own_cta_was_told_of():
    """Copies into a CTA's shared memory complete on CTA 0's full[]. A thread of CTA 0 that has waited there may read CTA 0's part; CTA 1's part would
    need that passed on with a release and an acquire at cluster scope, which an arrival without a scope does not give."""
    text = SOURCE.read_text()
    start = text.index("A_MN && warp >= 2 + EPI_WARPS) {")
    branch = re.sub(r"//[^\n]*", "", text[start:text.index("- epilogue (both CTAs", start)])
    waits = re.findall(r"mbar_(?:try_wait|wait_abortable)(<[^>]*>)?\(([^;]*)\)", branch)
    assert len(waits) == 1 and "&sm->full[s]" in waits[0][1]
    assert re.search(r"if \(rank == 0 && p\.aux\) \{", branch[:branch.index("mbar_wait_abortable")])
    assert "mbar_arrive_cluster" not in branch and "ld.shared::cluster" not in branch
    # CTA 1's stages have no other reader than the MMAs, so only CTA 0's wait for the warps that add up
    assert re.search(r"readers = A_MN && p\.aux && rank == 0 \? 1 \+ SUM_WARPS : 1;", text)
