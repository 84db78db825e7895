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
    parts += [re.sub(r"//[^\n]*", "", open(os.path.join(KERNELS, name)).read()) for name in ("gemm.cu", "gemm_sm100.cuh", "gemm2_sm100.cuh", "tp_decode_local.cu")]
    moe = open(os.path.join(KERNELS, "moe.cu")).read()
    # (the several-rank forms of the same source are launched after what they read: `kOne ? overlapped : not` is the one place they differ in)
    parts += [_definition(moe, head).replace("kOne ? ptx::ld_weak_v4(src + w0 + j * 32) : ptx::ld_input_v4(src + w0 + j * 32)", "")
              for head in ("moeDispatchKernel(MoeDispatchArgs a)", "moeCombineKernel(MoeCombineArgs a)")]
    parts.append(_definition(open(os.path.join(KERNELS, "collectives.cu")).read(), "allreduceLLKernel(CollArgs a)"))
    parts.append(_definition(open(os.path.join(KERNELS, "sp_fused.cu")).read(), "struct StoreGated {"))
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


def test_signals_between_blocks_of_a_cluster_have_its_scope():
    """An arrive on another block's barrier without a scope is one at CTA scope, which orders nothing between the two."""
    include = os.path.join(ROOT, "mscclpp_b200", "csrc", "include", "mscclpp")
    texts = [open(os.path.join(folder, name)).read() for top in (include, KERNELS) for folder, _, names in os.walk(top) for name in names
             if name.endswith((".cuh", ".cu", ".hpp"))]
    arrives = [m for text in texts for m in re.findall(r'"mbarrier\.arrive[^"]*shared::cluster[^"]*"', text)]
    assert arrives and all(re.search(r"\.(release|relaxed)\.cluster\.", a) for a in arrives), arrives
    # a relaxed one stands between the two fences of tensor memory
    core = re.sub(r"//[^\n]*", "", open(os.path.join(KERNELS, "gemm2_sm100.cuh")).read())
    assert re.search(r"mbarWaitFast<true>\(&st\.tmemEmpty.*?\n\s*if \(!ok\) break;\n\s*ptx::tcgen05_fence_after_sync\(\)", core)
    for name in ("tp_wave.cu", "tp_fused.cu", "gemm_sm100.cuh"):
        text = open(os.path.join(KERNELS, name)).read()
        assert len(re.findall(r"arriveEmpty\(\);", text)) == len(re.findall(
            r"tcgen05_fence_before_sync\(\);\s*__syncwarp\(\);\s*if \(lane == 0\) arriveEmpty\(\);", text)) > 0, name
