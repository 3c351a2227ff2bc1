"""The kernels of the CG loop's bodies, read from their source.

A turn of the graph's loop runs several bodies, and the host-driven loop queues
several between two looks at the flag, so bodies run after the solve has ended:
every kernel of one has to leave at once then (a whole SpMV past the end would
change no result, only take its time).
"""
import re
from pathlib import Path

import pytest

SRC = (Path(__file__).resolve().parents[1] / "alien_b200" / "csrc" / "krylov.cu").read_text()


@pytest.mark.parametrize("kernel", ["k_cg_px", "k_cg_spmv", "k_cg_spmv_x4", "k_cgj_spmv", "k_cgj_update",
                                    "k_cgj_update_x4"])
def test_a_body_past_the_end_leaves_at_once(kernel):
    m = re.search(rf"__global__[^;{{]*\b{kernel}\([^{{]*\)\s*\{{(?P<first>[^;{{]*[;{{])", SRC)
    assert m, kernel
    assert re.match(r"\s*if \(st->done\)\s*(return;|\{)", m["first"]), m["first"]
