"""Launch order that no run can show reliably: what the kernel sources say about overlapped launches."""
import os
import re

from bitmtp_b200 import native


def _body(source: str, kernel: str) -> str:
    """Text of a kernel from its opening brace to the closing brace in the first column."""
    start = source.index("{", source.index(kernel + "("))
    text = source[start:source.index("\n}\n", start)]
    return re.sub(r"//[^\n]*", "", text)


def test_the_packer_never_lets_a_product_start_early():
    """Products launched with overlap request their weights before they wait for the previous kernel, so the kernel that
    writes weights must not trigger the next launch, and it touches nothing before it has waited itself."""
    source = open(os.path.join(native.CSRC, "fused_ops.cuh")).read()
    body = _body(source, "pack_t2_g128_kernel")
    assert "launch_dependents" not in body
    statements = [s.strip() for s in body.lstrip("{").split(";")]
    assert statements[0] == "pdl_wait()"
