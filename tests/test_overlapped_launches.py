"""Rules of the kernels that are launched while the one before them on the stream may still run. They cannot be seen in results
(the non-coherent path usually returns the right words), so the source is checked."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
KERNELS = os.path.join(ROOT, "mscclpp_b200", "csrc", "kernels")


def _definition(text, head):
    """The text from `head` to the end of its block, comments dropped."""
    text = re.sub(r"//[^\n]*", "", text)
    start = text.index(head)
    depth, i = 0, text.index("{", start)
    while True:
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        i += 1
        if depth == 0:
            return text[start:i]


def test_overlapped_kernels_read_nothing_through_the_non_coherent_path():
    """ld.global.nc is for data that nothing writes while the kernel runs. An overlapped kernel runs while the one before writes
    its operands, the residual, h and the rows' sums."""
    tp = open(os.path.join(KERNELS, "tp_fused.cu")).read()
    parts = [_definition(tp, "tpScaleRowsPartsKernel(const bf16* h"), _definition(tp, "struct ResidualSumsqStore {"),
             _definition(tp, "struct ResidualSumsqRows {")]
    parts += [re.sub(r"//[^\n]*", "", open(os.path.join(KERNELS, name)).read()) for name in ("gemm.cu", "gemm_sm100.cuh", "gemm2_sm100.cuh")]
    for text in parts:
        assert len(text) > 500
        assert not re.search(r"ld_input_v4|__ldg|\.nc\b|__restrict__", text)
