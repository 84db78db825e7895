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


def test_blocks_of_a_cluster_have_started_before_one_writes_to_another():
    """Shared memory of another block may be written once that block runs: being scheduled together does not say that it does. The
    first barrier of the cluster stands before the first such write, where the launch still waits for the kernel before it."""
    for name, head in (("tp_decode_local.cu", "tpDecodeLocalKernel(const"), ("gemm2_sm100.cuh", "void gemmCtaPair(")):
        text = _definition(open(os.path.join(KERNELS, name)).read(), head)
        met, wrote = text.index("cluster_sync_all()"), re.search(r"mapa_shared|shared::cluster", text).start()
        assert met < text.index("grid_dependency_wait()") and met < wrote, name


def test_no_binding_goes_on_to_another_kernel_after_an_error():
    """Which kernel a call takes is asked before the launch (tpDecodeLocalCovers), so that an error of the launch itself reaches the
    caller: none can be provoked without a fault."""
    folder = os.path.join(ROOT, "mscclpp_b200", "csrc", "bindings")
    for name in sorted(os.listdir(folder)):
        assert not re.search(r"[!=]=\s*cudaError", open(os.path.join(folder, name)).read()), name
    assert "tpDecodeLocalCovers(" in open(os.path.join(folder, "more.cpp")).read()
