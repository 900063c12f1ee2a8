"""Order of `pdl_wait` and `pdl_trigger` in the kernels that head a forward pass, read from their source.

A product of few rows asks for weight tiles in front of its own wait (csrc/gemm_tcgen05.cu).  With every kernel before it in the pass triggering ahead of its wait, it could start
while the kernel in front of the pass, which may have written those weights, is not known to be visible; the first kernel of a pass therefore triggers behind its wait."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "realhf_b200" / "ops" / "csrc"


def body(file: str, kernel: str) -> str:
    """The text of a kernel's body without its comments."""
    text = re.sub(r"//[^\n]*", "", (CSRC / file).read_text())
    at = text.index("{", re.search(r"__global__[^;{]*\b" + kernel + r"\(", text).end())
    depth, end = 0, at
    while True:
        depth += {"{": 1, "}": -1}.get(text[end], 0)
        end += 1
        if depth == 0:
            return text[at:end]


@pytest.mark.parametrize("file,kernel", [("embed_grad.cu", "rows_kernel"), ("embed_grad.cu", "rows_warp_kernel"), ("posenc.cu", "embed_sinusoid_kernel")])
def test_the_first_kernel_of_a_pass_triggers_behind_its_wait(file, kernel):
    text = body(file, kernel)
    assert text.count("pdl_wait()") == 1 and text.count("pdl_trigger()") == 1
    assert text.index("pdl_wait()") < text.index("pdl_trigger()")
