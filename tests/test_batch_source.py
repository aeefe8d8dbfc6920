"""How the batch kernel loads what it writes itself: nothing that runs can show a
wrong choice reliably, so the source is read."""
import os
import re

from conftest import ROOT

CSRC = os.path.join(ROOT, "block_matrix_format_performance_gb300", "csrc")


def test_batch_products_load_their_vector_coherently():
    """The vector of a product is rewritten within the launch, and the read-only
    path may return an older line: every row routine takes the coherent loads,
    and no read-only load takes the vector."""
    text = open(os.path.join(CSRC, "batch.cu")).read()
    calls = re.findall(r"core::(?:flat|csr|tpr|rowown)_row<([^>]*)>", text)
    assert len(calls) == 3
    for args in calls:
        assert args.split(",")[-1].strip() == "dev::XCoh", args
    for args in re.findall(r"(?:__ldg|__ldcs|ld_cached\w*|ld_stream\w*) \((.*)\)", text):
        assert not re.search(r"\bx\b", args), args
