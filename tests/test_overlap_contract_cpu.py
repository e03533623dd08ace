"""What no run can show reliably, from the kernel sources: the order of overlapped launches, and which lanes of a warp meet
in a shuffle."""
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


def test_the_prompt_softmax_takes_whole_warps():
    """The tile kernel's two softmax builds shuffle over whole warps, so the number that chooses between them may depend on
    the warp but on nothing finer.  And one number is enough: the rows of a warp's 16 vectors lie in one slab."""
    source = open(os.path.join(native.CSRC, "prompt_attn.cuh")).read()
    body = _body(source, "prompt_hist_kernel")
    assert "if (lim >= BM_ATTN_SUPER) pa_softmax<true>" in body
    assert re.findall(r"\blim\s*=[^=][^;]*;", body) == ["lim = pa_tile_keys(p.hist0, p.T, row0, p.log_g, warp, key0);"]
    slab, vectors = (int(re.search(rf"{n} = (\d+)", source).group(1)) for n in ("kPaSlab", "kPaQueries"))
    for log_g in range(4):
        for warp in range(vectors // 16):
            for row0 in range(0, 40 * slab, vectors >> log_g):
                rows = [row0 + (v >> log_g) for v in range(16 * warp, 16 * warp + 16)]
                assert rows[0] == row0 + ((16 * warp) >> log_g) and len({r // slab for r in rows}) == 1


def test_kernels_that_wait_promise_no_read_only_memory():
    """A kernel that may start before its predecessor has finished reads memory that is written while it runs, so none of its
    parameters may be declared read-only and unaliased: a load through one may be moved ahead of the wait."""
    seen = 0
    for name in sorted(os.listdir(native.CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        text = re.sub(r"//[^\n]*", "", open(os.path.join(native.CSRC, name)).read())
        for m in re.finditer(r"__global__[^;{]*\{", text):
            body = text[m.end():text.index("\n}\n", m.end())]
            if "pdl_wait()" in body:
                seen += 1
                assert "__restrict__" not in m.group(0), f"{name}: {m.group(0)}"
                assert not re.search(r"const[^;=]*__restrict__", body), f"{name}: {m.group(0)}"
    assert seen >= 10
