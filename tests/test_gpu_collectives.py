"""Native collective kernels against a plain PyTorch fp32 reference.

All ranks are emulated on ONE GPU: the kernels run every rank inside one launch
(gridDim.y = world), which exercises exactly the device code that runs across GPUs, minus NVLS.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu

DTYPES = [torch.bfloat16, torch.float16, torch.float32]


def _symm(world, nbytes=192 << 20):
    from mscclpp_b200 import SymmetricMemory

    return SymmetricMemory.emulated(world, nbytes=nbytes, timeout_ms=2000)


def _fill(symm, t, seed):
    """Per-rank N(0,1) data, returns the list of per-rank tensors (fp32 copies)."""
    ref = []
    for r in range(symm.world):
        g = torch.Generator(device="cuda").manual_seed(seed * 100 + r)
        x = torch.randn(t.shape, generator=g, device="cuda", dtype=torch.float32)
        view = symm.rank_view(t, r)
        if t.dtype in (torch.int32,):
            x = (x * 100).round()
        view.copy_(x.to(t.dtype))
        ref.append(view.to(torch.float32).clone())
    return ref


def _tol(dtype):
    return {torch.bfloat16: 2e-2, torch.float16: 4e-3, torch.float32: 1e-5}.get(dtype, 0)


@pytest.mark.parametrize("algo", ["packet", "allpair_packet", "packet128"])
@pytest.mark.parametrize("world", [2, 4, 8])
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("numel", [8, 40, 1024, 33000, 262144])
def test_allreduce_ll(world, dtype, numel, algo):
    from mscclpp_b200.ops import all_reduce
    from mscclpp_b200.ops.collectives import ll128_max_bytes

    if algo == "packet128" and numel * torch.empty((), dtype=dtype).element_size() > ll128_max_bytes(world):
        pytest.skip("beyond the range the LL128 scratch is sized for at this world size")
    symm = _symm(world)
    inp = symm.tensor((numel,), dtype)
    out = symm.tensor((numel,), dtype)
    for launch in range(3):  # consecutive launches alternate the LL scratch buffer
        ref = _fill(symm, inp, seed=launch + 1)
        expect = torch.stack(ref).sum(0)
        all_reduce(symm, inp, out, algo=algo, n_blocks=4)
        torch.cuda.synchronize()
        symm.check()
        for r in range(world):
            got = symm.rank_view(out, r).to(torch.float32)
            torch.testing.assert_close(got, expect.to(dtype).to(torch.float32), atol=_tol(dtype) * 4, rtol=_tol(dtype))
    symm.destroy()


@pytest.mark.parametrize("world", [2, 4, 8])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("numel", [4096, 262144 + 8, 3 << 20])
def test_allreduce_pipeline_buffers_outside_the_heap(world, dtype, numel):
    """Ordinary CUDA tensors (not heap memory): one kernel copies in, reduces through heap scratch and copies out.
    Row r of the [world, numel] tensors is emulated rank r's buffer; with 4 blocks the larger sizes take many rounds."""
    from mscclpp_b200.ops import all_reduce

    symm = _symm(world)
    for launch in range(2):
        g = torch.Generator(device="cuda").manual_seed(numel + launch)
        x = torch.randn((world, numel), generator=g, device="cuda").to(dtype)
        out = torch.full_like(x, float("nan"))
        assert not symm.contains(x)
        all_reduce(symm, x, out, algo="rsag_pipeline", n_blocks=4)
        torch.cuda.synchronize()
        symm.check()
        expect = x.float().sum(0).to(dtype).float()
        for r in range(world):
            torch.testing.assert_close(out[r].float(), expect, atol=_tol(dtype) * 4, rtol=_tol(dtype))
    symm.destroy()


@pytest.mark.parametrize("world,numel,n_blocks", [(1, 3, 1), (1, 100003, 2), (3, 1009, 2), (5, 70001, 3), (7, 40000, 0), (2, 5000003, 0), (4, 2100001, 0)])
@pytest.mark.parametrize("dtype", [torch.int32, torch.float16])
def test_allreduce_pipeline_ragged(world, numel, n_blocks, dtype):
    """Messages that end inside a 16-byte unit and inside a slice, ranks that fill no batch of sources, one round and many,
    in place and not. Integers are exact; fp16 sums in fp32 round once (2^-11 of the value) after `world` fp32 additions."""
    from mscclpp_b200.ops import all_reduce

    # (the rows of emulated ranks follow one another and start on 16-byte boundaries: only one rank can end inside a unit)
    stride = numel if world == 1 else (numel * dtype.itemsize + 15) // 16 * 16 // dtype.itemsize
    symm = _symm(world)
    g = torch.Generator(device="cuda").manual_seed(numel)
    x = torch.randn((world, stride), generator=g, device="cuda")
    x = (x * 1000).to(dtype) if not dtype.is_floating_point else x.to(dtype)
    expect = x.double().sum(0)
    bound = 0 if not dtype.is_floating_point else expect.abs() * 2.0 ** -11 + x.double().abs().sum(0) * world * 2.0 ** -23 + 2.0 ** -25
    for in_place in (False, True):
        src = x.clone()
        out = src if in_place else torch.zeros_like(src)
        all_reduce(symm, src, out, algo="rsag_pipeline", n_blocks=n_blocks)
        torch.cuda.synchronize()
        symm.check()
        assert bool(((out.double() - expect).abs() <= bound).all())
    symm.destroy()


@pytest.mark.parametrize("world", [2, 3, 4, 8])
@pytest.mark.parametrize("numel", [5, 4099, (1 << 18) + 3])
def test_allreduce_pipeline_parts_stored_or_fetched(world, numel):
    """Both ways for a reduced part to reach the other ranks, in turn on the same scratch, with slices that leave a part of a unit. (Whole numbers that
    fp32 sums exactly.)"""
    from mscclpp_b200 import native
    from mscclpp_b200.ops import collectives as C

    n = native()
    symm = _symm(world)
    scratch = C._pipeline_scratch(symm)
    x = torch.randint(-1000, 1000, (world, numel + (-numel) % 4), device="cuda").float()  # (rows begin at 16-byte boundaries)
    out = torch.empty_like(x)
    nbytes = numel * 4
    for fetch in (0, 1, -1, 0, 1):
        for blocks, slice_bytes in ((3, 32 * world), (8, 16 * world * 100)):
            out.fill_(-1.0)
            n.pipeline_allreduce(symm.heap, x.data_ptr(), out.data_ptr(), nbytes, n.DataType.float32, n.ReduceOp.SUM, scratch.data_ptr(), slice_bytes, blocks,
                                 512, torch.cuda.current_stream().cuda_stream, False, x.shape[1] * 4, scratch.numel(), fetch)
            symm.check()
            assert torch.equal(out[:, :numel], x.sum(0)[:numel].expand(world, -1)) and bool((out[:, numel:] == -1.0).all())
    symm.destroy()


def test_allreduce_pipeline_scratch_halves_stay_apart():
    """Peers may still fetch reduced parts of a launch when a rank copies in for the next one, which has other slices: what is
    copied in stays in the scratch's first half and what is reduced in its second, whatever the slices. A launch that is not told
    the scratch's size ends with a barrier instead."""
    from mscclpp_b200 import native
    from mscclpp_b200.ops import all_reduce
    from mscclpp_b200.ops import collectives as C

    world = 4
    symm = _symm(world)
    scratch = C._pipeline_scratch(symm)
    halves = [symm.rank_view(scratch, r).view(torch.float32).chunk(2) for r in range(world)]
    for first, second in halves:
        first.zero_(), second.zero_()
    for numel, n_blocks in ((37 << 10, 0), (8 << 20, 0), (1 << 20, 3), (3 << 20, 7), (5000, 0)):
        x = torch.ones(world, numel, device="cuda")
        out = torch.empty_like(x)
        all_reduce(symm, x, out, algo="rsag_pipeline", n_blocks=n_blocks)
        assert bool((out == world).all())
        for first, second in halves:
            assert bool((first == 1).any()) and not bool((first == world).any())
            assert bool((second == world).any()) and not bool((second == 1).any())
    n = native()
    for blocks, slice_bytes in ((5, 4096), (16, 64 << 10)):
        out.zero_()
        n.pipeline_allreduce(symm.heap, x.data_ptr(), out.data_ptr(), numel * 4, n.DataType.float32, n.ReduceOp.SUM, scratch.data_ptr(),
                             slice_bytes, blocks, 512, torch.cuda.current_stream().cuda_stream, False, numel * 4)
        assert bool((out == world).all())
    with pytest.raises(Exception):
        n.pipeline_allreduce(symm.heap, x.data_ptr(), out.data_ptr(), numel * 4, n.DataType.float32, n.ReduceOp.SUM, scratch.data_ptr(),
                             64 << 10, 16, 512, torch.cuda.current_stream().cuda_stream, False, numel * 4, 1 << 20)
    symm.check()
    symm.destroy()


@pytest.mark.parametrize("world", [2, 8])
def test_allreduce_ll_int_and_min(world):
    from mscclpp_b200.ops import all_reduce

    symm = _symm(world)
    inp = symm.tensor((5000,), torch.int32)
    out = symm.tensor((5000,), torch.int32)
    ref = _fill(symm, inp, seed=7)
    all_reduce(symm, inp, out, algo="packet", n_blocks=2)
    torch.cuda.synchronize()
    symm.check()
    assert torch.equal(symm.rank_view(out, world - 1).to(torch.float32), torch.stack(ref).sum(0))
    finp = symm.tensor((4096,), torch.bfloat16)
    fout = symm.tensor((4096,), torch.bfloat16)
    ref = _fill(symm, finp, seed=9)
    all_reduce(symm, finp, fout, op="min", algo="packet", n_blocks=2)
    torch.cuda.synchronize()
    symm.check()
    assert torch.equal(symm.rank_view(fout, 0).to(torch.float32), torch.stack(ref).min(0).values)
    symm.destroy()


@pytest.mark.parametrize("world", [2, 4, 8])
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("numel", [1024, 8 * 1000 * 8, 1 << 20])
def test_allreduce_two_shot(world, dtype, numel):
    from mscclpp_b200.ops import all_reduce

    symm = _symm(world)
    inp = symm.tensor((numel,), dtype)
    out = symm.tensor((numel,), dtype)
    for launch in range(2):
        ref = _fill(symm, inp, seed=launch + 11)
        expect = torch.stack(ref).sum(0)
        all_reduce(symm, inp, out, algo="rsag_zero_copy", n_blocks=8)
        torch.cuda.synchronize()
        symm.check()
        for r in range(world):
            got = symm.rank_view(out, r).to(torch.float32)
            torch.testing.assert_close(got, expect.to(dtype).to(torch.float32), atol=_tol(dtype) * 4, rtol=_tol(dtype))
    # in place
    ref = _fill(symm, inp, seed=99)
    all_reduce(symm, inp, None, algo="rsag_zero_copy", n_blocks=8)
    torch.cuda.synchronize()
    symm.check()
    expect = torch.stack(ref).sum(0).to(dtype).to(torch.float32)
    torch.testing.assert_close(symm.rank_view(inp, world - 1).to(torch.float32), expect, atol=_tol(dtype) * 4, rtol=_tol(dtype))
    symm.destroy()


@pytest.mark.parametrize("world", [2, 8])
def test_reduce_scatter_and_all_gather(world):
    from mscclpp_b200.ops import all_gather, reduce_scatter

    symm = _symm(world)
    per = 4096 * 3
    full = symm.tensor((world * per,), torch.bfloat16)
    part = symm.tensor((per,), torch.bfloat16)
    ref = _fill(symm, full, seed=21)
    reduce_scatter(symm, full, part, nvls=False, n_blocks=4)
    torch.cuda.synchronize()
    symm.check()
    total = torch.stack(ref).sum(0)
    for r in range(world):
        got = symm.rank_view(part, r).to(torch.float32)
        torch.testing.assert_close(got, total[r * per:(r + 1) * per].to(torch.bfloat16).to(torch.float32), atol=8e-2, rtol=2e-2)
    ref = _fill(symm, part, seed=23)
    all_gather(symm, part, full, nvls=False, n_blocks=4)
    torch.cuda.synchronize()
    symm.check()
    expect = torch.cat(ref)
    for r in range(world):
        assert torch.equal(symm.rank_view(full, r).to(torch.float32), expect)
    symm.destroy()


def _rmsnorm_ref(parts, residual, gamma, eps, dtype):
    h = torch.stack(parts).sum(0).to(dtype).to(torch.float32)
    if residual is not None:
        h = (h + residual).to(dtype).to(torch.float32)
    y = h * torch.rsqrt(h.pow(2).mean(-1, keepdim=True) + eps)
    if gamma is not None:
        y = y * gamma
    return y.to(dtype).to(torch.float32), h


@pytest.mark.parametrize("world", [2, 8])
@pytest.mark.parametrize("algo", ["packet", "rsag_zero_copy"])
@pytest.mark.parametrize("rows,hidden", [(1, 8192), (8, 8192), (24, 1024), (64, 4096)])
def test_allreduce_residual_rmsnorm(world, algo, rows, hidden):
    from mscclpp_b200.ops import all_reduce_rmsnorm

    if algo == "rsag_zero_copy" and rows < world:
        pytest.skip("row-sliced two-shot needs at least one row per rank")
    dtype = torch.bfloat16
    symm = _symm(world)
    inp = symm.tensor((rows, hidden), dtype)
    out = symm.tensor((rows, hidden), dtype)
    res_in = symm.tensor((rows, hidden), dtype)
    res_out = symm.tensor((rows, hidden), dtype)
    gamma = symm.tensor((hidden,), dtype)
    parts = _fill(symm, inp, seed=31)
    g = torch.Generator(device="cuda").manual_seed(5)
    residual = torch.randn((rows, hidden), generator=g, device="cuda").to(dtype)
    gam = (1 + 0.1 * torch.randn((hidden,), generator=g, device="cuda")).to(dtype)
    for r in range(world):
        symm.rank_view(res_in, r).copy_(residual)
        symm.rank_view(gamma, r).copy_(gam)
        symm.rank_view(out, r).zero_()
        symm.rank_view(res_out, r).zero_()
    all_reduce_rmsnorm(symm, inp, out, res_in, res_out, gamma, eps=1e-5, algo=algo, n_blocks=4)
    torch.cuda.synchronize()
    symm.check()
    y_ref, h_ref = _rmsnorm_ref(parts, residual.float(), gam.float(), 1e-5, dtype)
    for r in range(world):
        torch.testing.assert_close(symm.rank_view(res_out, r).float(), h_ref, atol=6e-2, rtol=2e-2)
        torch.testing.assert_close(symm.rank_view(out, r).float(), y_ref, atol=6e-2, rtol=2e-2)
    symm.destroy()


def test_bounded_wait_reports_timeout():
    """A rank that never shows up makes the others' waits expire with a status, not hang: here the
    'missing rank' is simulated by launching the LL kernel for world=2 data but with a heap whose
    second emulated rank sends to a different scratch epoch (we poison the epoch of rank 1)."""
    from mscclpp_b200 import SymmetricMemory
    from mscclpp_b200.ops import all_reduce

    symm = SymmetricMemory.emulated(2, nbytes=64 << 20, timeout_ms=50)
    inp = symm.tensor((1024,), torch.float32, zero=True)
    out = symm.tensor((1024,), torch.float32, zero=True)
    # desynchronise the launch epochs of the two emulated ranks: their packet flags will never match
    ctrl1 = symm.rank_view(symm_ctrl_epoch(symm), 1)
    ctrl1.fill_(1000)
    all_reduce(symm, inp, out, algo="packet", n_blocks=1)
    torch.cuda.synchronize()  # returns: the waits gave up after ~50 ms
    n = symm.heap.status()
    assert n.code != 0 and n.poisoned == 1
    with pytest.raises(Exception):
        symm.check()
    # the context is still usable afterwards
    assert float(torch.ones(4, device="cuda").sum()) == 4.0
    symm.destroy()


def symm_ctrl_epoch(symm):
    from mscclpp_b200 import tensor_from_pointer

    return tensor_from_pointer(symm.heap.local_base, (1,), torch.int32, symm.device, owner=symm)


@pytest.mark.parametrize("world", [1, 2, 8])
@pytest.mark.parametrize("tokens,hidden,k", [(1, 1024, 256), (5, 2048, 512), (8, 8192, 1024)])
def test_decode_layer_one_kernel(world, tokens, hidden, k):
    """Up to 8 tokens: weight-streaming slabs + one-shot packet allreduce + residual + RMSNorm in one launch, all ranks
    emulated on one GPU; three launches in a row alternate the packet scratch."""
    from mscclpp_b200 import SymmetricMemory
    from mscclpp_b200.parallel.tp_layer import RowParallelLinearNorm

    symm = SymmetricMemory.emulated(world, nbytes=256 << 20, timeout_ms=3000)
    layer = RowParallelLinearNorm(symm, out_features=hidden, k_shard=k, max_tokens=8)
    g = torch.Generator(device="cuda").manual_seed(tokens + hidden)
    ws = [(torch.randn((hidden, k), generator=g, device="cuda") * 0.05).to(torch.bfloat16) for _ in range(world)]
    gam = (1 + 0.1 * torch.randn((hidden,), generator=g, device="cuda")).to(torch.bfloat16)
    for r in range(world):
        symm.rank_view(layer.gamma, r).copy_(gam)
    ctas = max(1, 128 // world)
    for rep in range(3):
        xs = [torch.randn((tokens, k), generator=g, device="cuda").to(torch.bfloat16) for _ in range(world)]
        residual = torch.randn((tokens, hidden), generator=g, device="cuda").to(torch.bfloat16)
        for r in range(world):
            symm.rank_view(layer.residual_in, r)[:tokens].copy_(residual)
            symm.rank_view(layer.out, r).fill_(float("nan"))
            symm.rank_view(layer.residual_out, r).fill_(float("nan"))
        layer.forward_decode(xs[0], nvls=False, num_ctas=ctas, emulated_inputs=list(zip(xs, ws)))
        torch.cuda.synchronize()
        symm.check()
        acc = sum((x.float() @ w.float().t()).to(torch.bfloat16).float() for x, w in zip(xs, ws))
        h = (acc.to(torch.bfloat16).float() + residual.float()).to(torch.bfloat16).float()
        y = (h * torch.rsqrt(h.pow(2).mean(-1, keepdim=True) + layer.eps) * gam.float()).to(torch.bfloat16).float()
        for r in range(world):
            got_h = symm.rank_view(layer.residual_out, r)[:tokens].float()
            got_y = symm.rank_view(layer.out, r)[:tokens].float()
            assert (got_h - h).abs().max().item() <= 0.02 * h.abs().max().item() + 0.05, f"rank {r} rep {rep}"
            assert (got_y - y).abs().max().item() <= 0.1, f"rank {r} rep {rep}"
    symm.destroy()


@pytest.mark.parametrize("world", [1, 2, 4])
@pytest.mark.parametrize("mode", [0, 1, 3])
@pytest.mark.parametrize("tokens,hidden,k", [(1, 1024, 128), (8, 2048, 256), (128, 8192, 256), (300, 1024, 512), (1024, 2048, 128)])
def test_fused_tp_layer_one_kernel(world, mode, tokens, hidden, k):
    """GEMM + allreduce + residual + RMSNorm in one launch, all ranks emulated on one GPU."""
    from mscclpp_b200 import SymmetricMemory
    from mscclpp_b200.parallel.tp_layer import RowParallelLinearNorm

    symm = SymmetricMemory.emulated(world, nbytes=256 << 20, timeout_ms=3000)
    layer = RowParallelLinearNorm(symm, out_features=hidden, k_shard=k, max_tokens=tokens)
    g = torch.Generator(device="cuda").manual_seed(tokens + hidden)
    xs = [torch.randn((tokens, k), generator=g, device="cuda").to(torch.bfloat16) for _ in range(world)]
    ws = [(torch.randn((hidden, k), generator=g, device="cuda") * 0.05).to(torch.bfloat16) for _ in range(world)]
    residual = torch.randn((tokens, hidden), generator=g, device="cuda").to(torch.bfloat16)
    gam = (1 + 0.1 * torch.randn((hidden,), generator=g, device="cuda")).to(torch.bfloat16)
    for r in range(world):
        symm.rank_view(layer.residual_in, r)[:tokens].copy_(residual)
        symm.rank_view(layer.gamma, r).copy_(gam)
        symm.rank_view(layer.out, r).zero_()
        symm.rank_view(layer.residual_out, r).zero_()
    for rep in range(2):
        layer.forward_fused(xs[0], mode=mode, nvls=False, num_reducers=4, num_gemm_ctas=max(1, 24 // world),
                            emulated_inputs=list(zip(xs, ws)))
        torch.cuda.synchronize()
        symm.check()
    acc = sum((x.float() @ w.float().t()).to(torch.bfloat16).float() for x, w in zip(xs, ws))
    h = (acc.to(torch.bfloat16).float() + residual.float()).to(torch.bfloat16).float()
    y = (h * torch.rsqrt(h.pow(2).mean(-1, keepdim=True) + layer.eps) * gam.float()).to(torch.bfloat16).float()
    for r in range(world):
        got_h = symm.rank_view(layer.residual_out, r)[:tokens].float()
        got_y = symm.rank_view(layer.out, r)[:tokens].float()
        assert (got_h - h).abs().max().item() <= 0.02 * h.abs().max().item() + 0.05
        assert (got_y - y).abs().max().item() <= 0.1
    symm.destroy()


def test_fused_tp_layer_timeline_stamps():
    """The optional per-CTA time stamps of the fused kernel: ordered, and the reducer groups account for rows."""
    from mscclpp_b200 import SymmetricMemory
    from mscclpp_b200.parallel.tp_layer import RowParallelLinearNorm

    world, tokens, hidden, k = 2, 512, 2048, 128
    symm = SymmetricMemory.emulated(world, nbytes=128 << 20, timeout_ms=3000)
    layer = RowParallelLinearNorm(symm, out_features=hidden, k_shard=k, max_tokens=tokens)
    xs = [torch.randn((tokens, k), device="cuda").to(torch.bfloat16) for _ in range(world)]
    ws = [(torch.randn((hidden, k), device="cuda") * 0.05).to(torch.bfloat16) for _ in range(world)]
    gemm_ctas, reducers = 8, 4
    tl = torch.zeros((gemm_ctas + reducers, 16), dtype=torch.int64, device="cuda")
    layer.forward_fused(xs[0], mode=1, nvls=False, block_n=256, num_reducers=reducers, num_gemm_ctas=gemm_ctas,
                        emulated_inputs=list(zip(xs, ws)), timeline=tl)
    torch.cuda.synchronize()
    symm.check()
    t = tl.cpu()
    assert (t[:, 0] > 0).all()
    assert (t[:, 1] >= t[:, 0]).all() and (t[:, 2] >= t[:, 1]).all()
    assert int(t[:, 3].sum()) > 0  # first groups of the CTAs reduced rows
    assert (t[:, 8] + t[:, 9] + t[:, 10] <= t[:, 5]).all()  # the phases are parts of the time spent on rows
    assert (t[:gemm_ctas, 1] > t[:gemm_ctas, 0]).all()  # GEMM CTAs spent time in the matmul
    symm.destroy()


@pytest.mark.parametrize("world,rows_per_rank,k,n_cols,act", [(2, 256, 256, 256, "none"), (4, 128, 512, 512, "gelu"), (8, 128, 256, 256, "silu")])
def test_all_gather_gemm_one_kernel(world, rows_per_rank, k, n_cols, act):
    """All-gather -> GEMM in one launch (copier CTAs + gated tcgen05 GEMM), all ranks emulated on one GPU."""
    from mscclpp_b200 import SymmetricMemory
    from mscclpp_b200.parallel.sp_layer import all_gather_gemm

    symm = SymmetricMemory.emulated(world, nbytes=128 << 20, timeout_ms=3000)
    s_rows = world * rows_per_rank
    a_local = symm.tensor((rows_per_rank, k), torch.bfloat16)
    a_full = symm.tensor((s_rows, k), torch.bfloat16)
    out = symm.tensor((s_rows, n_cols), torch.bfloat16)
    g = torch.Generator(device="cuda").manual_seed(world * 100 + k)
    ws = [(torch.randn((n_cols, k), generator=g, device="cuda") * 0.05).to(torch.bfloat16) for _ in range(world)]
    for rep in range(2):
        shards = [torch.randn((rows_per_rank, k), generator=g, device="cuda").to(torch.bfloat16) for _ in range(world)]
        for r in range(world):
            symm.rank_view(a_local, r).copy_(shards[r])
            symm.rank_view(a_full, r).fill_(float("nan"))  # own rows are never copied there: must not be read
            symm.rank_view(out, r).zero_()
        all_gather_gemm(symm, a_local, a_full, ws, out, activation=act, block_n=256 if n_cols % 256 == 0 else 128, num_copiers=2,
                        num_gemm_ctas=max(1, 16 // world))
        torch.cuda.synchronize()
        symm.check()
        full = torch.cat(shards).float()
        for r in range(world):
            ref = full @ ws[r].float().t()
            if act == "gelu":
                ref = torch.nn.functional.gelu(ref, approximate="tanh")
            elif act == "silu":
                ref = torch.nn.functional.silu(ref)
            got = symm.rank_view(out, r).float()
            assert (got - ref).abs().max().item() <= 0.02 * ref.abs().max().item() + 0.02, (r, rep)
    symm.destroy()


# a shape for every form that one rank's product may take (gemm_plan_form), of widths that are no multiple of its tiles where it can be
@pytest.mark.parametrize("act", ["none", "gelu", "silu", "swiglu"])
@pytest.mark.parametrize("m,n,k,form", [(128, 1152, 256, (0, 64, 1)), (128, 640, 4096, (0, 64, 4)), (512, 3456, 256, (0, 128, 1)),
                                        (1408, 2944, 384, (0, 256, 1)), (640, 4224, 1280, (256, 256, 1)), (384, 3200, 1280, (128, 256, 1)),
                                        (256, 2688, 1536, (128, 128, 1))])
def test_all_gather_gemm_of_one_rank(act, m, n, k, form):
    """Nothing to gather: a plain product with its activation, against 64 bits. Activations of values up to +-100 and more, where the exponential
    overflows on one side."""
    from mscclpp_b200 import SymmetricMemory, native
    from mscclpp_b200.parallel.sp_layer import all_gather_gemm, interleave_gate_up

    assert native().gemm_plan_form(m, n, k) == form
    symm = SymmetricMemory.emulated(1, nbytes=256 << 20, timeout_ms=3000)
    g = torch.Generator(device="cuda").manual_seed(m + n)
    x, full = symm.tensor((m, k), torch.bfloat16), symm.tensor((m, k), torch.bfloat16)
    out = symm.tensor((m, n // 2 if act == "swiglu" else n), torch.bfloat16)
    x.copy_(torch.randn((m, k), generator=g, device="cuda"))
    w = (torch.randn((n, k), generator=g, device="cuda") * (30 / k ** 0.5)).to(torch.bfloat16)
    p = x.double() @ w.double().t()
    d = (x.double().abs() @ w.double().abs().t()) * k * 2.0 ** -24  # of the fp32 sum: at most K roundings of the products' magnitudes
    eps = 16 * 2.0 ** -23  # of the activation itself in fp32: exponential, reciprocal and products, a few units each
    if act == "none":
        ref, bound = p, d
    elif act == "silu":  # (its slope and GELU's are at most 1.13; an exponential's relative error grows with its argument)
        ref = torch.nn.functional.silu(p)
        bound = 1.13 * d + eps * (1 + p.abs()) * ref.abs()
    elif act == "gelu":
        ref = torch.nn.functional.gelu(p, approximate="tanh")
        bound = 1.13 * d + eps * (1 + p.abs() + p.abs() ** 3) * ref.abs()
    else:
        gate, up, dg, du = p[:, :n // 2], p[:, n // 2:], d[:, :n // 2], d[:, n // 2:]
        ref = torch.nn.functional.silu(gate) * up
        bound = 1.13 * dg * (up.abs() + du) + torch.nn.functional.silu(gate).abs() * du + eps * (1 + gate.abs()) * ref.abs()
        w = interleave_gate_up(w[:n // 2], w[n // 2:])
    bound = bound + ref.abs() * 2.0 ** -8 * 1.01 + 1e-37  # one rounding to bf16 (eight significant bits), or to zero below its range
    for _ in range(2):
        out.fill_(float("nan"))
        all_gather_gemm(symm, x, full, w, out, activation=act)
        torch.cuda.synchronize()
        symm.check()
        assert bool(((out.double() - ref).abs() <= bound).all())
    symm.destroy()


@pytest.mark.parametrize("world,rows_per_rank,k,ffn,block_n", [(2, 256, 256, 256, 256), (4, 128, 512, 128, 128), (2, 256, 128, 384, -1)])
def test_all_gather_gemm_swiglu(world, rows_per_rank, k, ffn, block_n):
    """All-gather -> GEMM over interleaved gate / up weights with the gated epilogue: out = silu(x Wg^T) * (x Wu^T), one
    launch, all ranks emulated on one GPU; against the fp32 composition."""
    from mscclpp_b200 import SymmetricMemory
    from mscclpp_b200.parallel.sp_layer import all_gather_gemm, interleave_gate_up

    symm = SymmetricMemory.emulated(world, nbytes=128 << 20, timeout_ms=3000)
    s_rows = world * rows_per_rank
    a_local = symm.tensor((rows_per_rank, k), torch.bfloat16)
    a_full = symm.tensor((s_rows, k), torch.bfloat16)
    out = symm.tensor((s_rows, ffn), torch.bfloat16)
    g = torch.Generator(device="cuda").manual_seed(world * 31 + ffn)
    wg = [(torch.randn((ffn, k), generator=g, device="cuda") * 0.05).to(torch.bfloat16) for _ in range(world)]
    wu = [(torch.randn((ffn, k), generator=g, device="cuda") * 0.05).to(torch.bfloat16) for _ in range(world)]
    ws = [interleave_gate_up(a, b) for a, b in zip(wg, wu)]
    for rep in range(2):
        shards = [torch.randn((rows_per_rank, k), generator=g, device="cuda").to(torch.bfloat16) for _ in range(world)]
        for r in range(world):
            symm.rank_view(a_local, r).copy_(shards[r])
            symm.rank_view(a_full, r).fill_(float("nan"))
            symm.rank_view(out, r).fill_(float("nan"))
        all_gather_gemm(symm, a_local, a_full, ws, out, activation="swiglu", block_n=block_n, num_copiers=2, num_gemm_ctas=max(2, 16 // world))
        torch.cuda.synchronize()
        symm.check()
        full = torch.cat(shards).float()
        for r in range(world):
            ref = torch.nn.functional.silu(full @ wg[r].float().t()) * (full @ wu[r].float().t())
            got = symm.rank_view(out, r).float()
            assert (got - ref).abs().max().item() <= 0.02 * ref.abs().max().item() + 0.02, (r, rep)
    symm.destroy()


@pytest.mark.parametrize("world,rows_per_rank,k,n_cols", [(2, 256, 128, 512), (4, 128, 256, 1024), (8, 128, 64, 256)])
def test_gemm_reduce_scatter_one_kernel(world, rows_per_rank, k, n_cols):
    """GEMM -> reduce-scatter in one launch: rank r ends with its row block of the summed product."""
    from mscclpp_b200 import SymmetricMemory
    from mscclpp_b200.parallel.sp_layer import gemm_reduce_scatter

    symm = SymmetricMemory.emulated(world, nbytes=128 << 20, timeout_ms=3000)
    s_rows = world * rows_per_rank
    partial = symm.tensor((s_rows, n_cols), torch.bfloat16)
    out = symm.tensor((rows_per_rank, n_cols), torch.bfloat16)
    g = torch.Generator(device="cuda").manual_seed(world * 10 + k)
    for rep in range(2):
        xs = [torch.randn((s_rows, k), generator=g, device="cuda").to(torch.bfloat16) for _ in range(world)]
        ws = [(torch.randn((n_cols, k), generator=g, device="cuda") * 0.05).to(torch.bfloat16) for _ in range(world)]
        for r in range(world):
            symm.rank_view(out, r).zero_()
        gemm_reduce_scatter(symm, xs, ws, partial, out, nvls=False, block_n=256 if n_cols % 256 == 0 else 128, num_reducers=3,
                            num_gemm_ctas=max(1, 16 // world))
        torch.cuda.synchronize()
        symm.check()
        total = sum((x.float() @ w.float().t()).to(torch.bfloat16).float() for x, w in zip(xs, ws))
        for r in range(world):
            ref = total[r * rows_per_rank:(r + 1) * rows_per_rank]
            got = symm.rank_view(out, r).float()
            assert (got - ref).abs().max().item() <= 0.02 * ref.abs().max().item() + 0.05, (r, rep)
    symm.destroy()


@pytest.mark.parametrize("rows,k,n_cols,act", [
    (128, 128, 128, "none"),      # one tile
    (256, 256, 512, "gelu"),      # one pair of SMs' tile in each direction
    (2304, 128, 256, "silu"),     # a band of 2048 rows and a last one of one tile, two-SM core
    (2176, 128, 384, "none"),     # the same on one-SM tiles
    (2304, 128, 512, "swiglu"),
])
def test_sequence_parallel_halves_on_one_rank(rows, k, n_cols, act):
    """One rank: no copiers, the band order, and the product stored where the reduce-scatter leaves it. Bounds: fp32
    accumulation (k * 2^-24 of the products' magnitudes, twice that through an activation of slope below 1.13 and the other
    factor of a gate), the activation's own error, one bf16 rounding."""
    from mscclpp_b200 import SymmetricMemory
    from mscclpp_b200.parallel.sp_layer import all_gather_gemm, gemm_reduce_scatter

    symm = SymmetricMemory.emulated(1, nbytes=64 << 20, timeout_ms=3000)
    g = torch.Generator(device="cuda").manual_seed(rows + n_cols)
    x = symm.tensor((rows, k), torch.bfloat16)
    x.copy_(torch.randn((rows, k), generator=g, device="cuda"))
    w = (torch.randn((n_cols, k), generator=g, device="cuda") * 0.1).to(torch.bfloat16)
    full = symm.tensor((rows, k), torch.bfloat16)
    out = symm.tensor((rows, n_cols // 2 if act == "swiglu" else n_cols), torch.bfloat16)
    back = symm.tensor((rows, n_cols), torch.bfloat16)
    partial = symm.tensor((rows, n_cols), torch.bfloat16)
    p = x.double() @ w.double().t()
    slack = (x.double().abs() @ w.double().abs().t()) * k * 2.0 ** -24
    ref, extra = p, slack
    if act == "gelu":
        ref = torch.nn.functional.gelu(p, approximate="tanh")
    elif act == "silu":
        ref = torch.nn.functional.silu(p)
    elif act == "swiglu":
        gate, up = (t.reshape(rows, -1) for t in p.view(rows, -1, 2, 32).unbind(2))
        sg, su = (t.reshape(rows, -1) for t in slack.view(rows, -1, 2, 32).unbind(2))
        ref = torch.nn.functional.silu(gate) * up
        extra = sg * up.abs() + su * gate.abs()
    for _ in range(2):
        out.fill_(float("nan"))
        back.fill_(float("nan"))
        all_gather_gemm(symm, x, full, w, out, activation=act)
        gemm_reduce_scatter(symm, x, w, partial, back)
        torch.cuda.synchronize()
        symm.check()
        assert bool(((out.double() - ref).abs() <= ref.abs() * (2.0 ** -8) + 2 * extra + 1e-6).all())
        assert bool(((back.double() - p).abs() <= p.abs() * 2.0 ** -8 + slack).all())
    symm.destroy()


@pytest.mark.parametrize("rows,k,n_cols", [(256, 128, 256), (384, 192, 128)])
def test_gemm_reduce_scatter_on_one_rank_with_reducers(rows, k, n_cols):
    """num_reducers on one rank: the product goes through `partial` and the reducers, to the same bits as without."""
    from mscclpp_b200 import SymmetricMemory
    from mscclpp_b200.parallel.sp_layer import gemm_reduce_scatter

    symm = SymmetricMemory.emulated(1, nbytes=64 << 20, timeout_ms=3000)
    g = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn((rows, k), generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn((n_cols, k), generator=g, device="cuda") * 0.1).to(torch.bfloat16)
    outs = [symm.tensor((rows, n_cols), torch.bfloat16) for _ in range(2)]
    partial = symm.tensor((rows, n_cols), torch.bfloat16)
    partial.fill_(float("nan"))
    gemm_reduce_scatter(symm, x, w, partial, outs[0])
    gemm_reduce_scatter(symm, x, w, partial, outs[1], num_reducers=2)
    torch.cuda.synchronize()
    symm.check()
    assert torch.equal(outs[0], outs[1]) and torch.equal(partial, outs[1])
    symm.destroy()


def _moe_reference(xs, idxs, wts, world, experts, f):
    """fp32 PyTorch model of dispatch -> expert function f(e, rows) -> combine, for all ranks."""
    ys = []
    for r in range(world):
        y = torch.zeros_like(xs[r], dtype=torch.float32)
        for k in range(idxs[r].shape[1]):
            e = idxs[r][:, k]
            valid = e >= 0
            contrib = torch.zeros_like(y)
            for ex in range(experts):
                m = valid & (e == ex)
                if m.any():
                    contrib[m] = f(ex, xs[r][m].float())
            y += wts[r][:, k:k + 1] * contrib
        ys.append(y)
    return ys


@pytest.mark.parametrize("world,experts,tokens,hidden,topk,fp8", [(2, 8, 200, 512, 2, False), (4, 16, 96, 1024, 2, True), (8, 64, 64, 4096, 2, False),
                                                                  (8, 64, 33, 1024, 4, True)])
def test_moe_dispatch_combine(world, experts, tokens, hidden, topk, fp8):
    """Dispatch pushes every (token, expert) pair into the hosting rank's expert-grouped buffer; combine pulls the expert
    outputs back. All ranks emulated on one GPU; checked against a plain PyTorch model of the same exchange."""
    from mscclpp_b200 import SymmetricMemory
    from mscclpp_b200.parallel.moe import ExpertParallelDispatcher, dequantize_rows

    symm = SymmetricMemory.emulated(world, nbytes=256 << 20, timeout_ms=3000)
    disp = ExpertParallelDispatcher(symm, num_experts=experts, hidden=hidden, max_tokens=tokens, topk=topk, fp8=fp8)
    el = experts // world
    g = torch.Generator(device="cuda").manual_seed(world * 1000 + tokens)
    for rep in range(2):
        xs = [torch.randn((tokens, hidden), generator=g, device="cuda").to(torch.bfloat16) for _ in range(world)]
        idxs = [torch.stack([torch.randperm(experts, generator=g, device="cuda")[:topk] for _ in range(tokens)]).to(torch.int32) for _ in range(world)]
        idxs[0][0, 0] = -1  # an unused slot
        wts = [torch.rand((tokens, topk), generator=g, device="cuda") for _ in range(world)]
        for r in range(world):
            x_s, idx_s, w_s = disp.stage(r, xs[r], idxs[r], wts[r])
        recv_x, counts, slot_map = disp.dispatch(x_s, idx_s, n_blocks=4)
        torch.cuda.synchronize()
        symm.check()
        # every destination holds exactly the rows routed to it, grouped by expert, tagged with their source
        for d in range(world):
            cnt = symm.rank_view(counts, d).cpu().tolist()
            expect_cnt = [sum(int((idxs[s] == d * el + j).sum()) for s in range(world)) for j in range(el)]
            assert cnt[:el] == expect_cnt and cnt[el] == sum(expect_cnt)
            rows = symm.rank_view(recv_x, d)[:cnt[el]]
            src = symm.rank_view(disp.recv_src, d)[:cnt[el]].cpu()
            got = dequantize_rows(rows, symm.rank_view(disp.recv_scales, d)[:cnt[el]]) if fp8 else rows.float()
            want = torch.stack([xs[int(v) >> 24][int(v) & 0xFFFFFF].float() for v in src.tolist()]) if cnt[el] else got
            tol = 0.07 * want.abs().max().item() if fp8 else 0.0
            assert (got - want).abs().max().item() <= tol
            # the expert of a row follows from its position
            bounds = [0]
            for c_ in expect_cnt:
                bounds.append(bounds[-1] + c_)
            for j in range(el):
                for v in src[bounds[j]:bounds[j + 1]].tolist():
                    s_, t_ = int(v) >> 24, int(v) & 0xFFFFFF
                    assert (idxs[s_][t_] == d * el + j).any()
        # experts: out = (e + 1) * 0.5 * row  (cheap, expert dependent)
        for d in range(world):
            cnt = symm.rank_view(counts, d).cpu().tolist()
            rows = symm.rank_view(recv_x, d)
            val = dequantize_rows(rows[:cnt[el]], symm.rank_view(disp.recv_scales, d)[:cnt[el]]) if fp8 else rows[:cnt[el]].float()
            out = symm.rank_view(disp.expert_out, d)
            start = 0
            for j in range(el):
                out[start:start + cnt[j]] = (val[start:start + cnt[j]] * (0.5 * (d * el + j + 1))).to(torch.bfloat16)
                start += cnt[j]
        y = disp.combine(idx_s, w_s, slot_map, n_blocks=4)
        torch.cuda.synchronize()
        symm.check()
        ref = _moe_reference(xs, idxs, wts, world, experts, lambda e, rows: (rows * (0.5 * (e + 1))).to(torch.bfloat16).float())
        for r in range(world):
            got = symm.rank_view(y, r).float()
            scale = ref[r].abs().max().item()
            assert (got - ref[r]).abs().max().item() <= (0.08 if fp8 else 0.02) * scale + 0.02, (r, rep)
    symm.destroy()


@pytest.mark.parametrize("tokens,hidden,experts,topk,fp8", [
    (1, 256, 8, 1, False),      # the smallest: one token, less than one piece of a row
    (33, 768, 16, 3, True),     # an odd number of 256-element steps in a row's last piece
    (149, 1280, 256, 8, False),  # one token more than thread blocks, all counters
    (148 * 32 + 5, 512, 64, 2, True),  # more tokens per block than one batch of destinations
    (700, 8192, 128, 5, False),  # the widest rows
])
def test_moe_one_rank(tokens, hidden, experts, topk, fp8):
    """One rank: rows grouped by expert in expert order, every pair's slot pointing at its row, and the weighted sum back.
    The result of identity experts is exact up to one bf16 rounding of an fp32 sum of `topk` terms."""
    from mscclpp_b200 import SymmetricMemory
    from mscclpp_b200.parallel.moe import ExpertParallelDispatcher, dequantize_rows

    symm = SymmetricMemory.emulated(1, nbytes=tokens * topk * hidden * 5 + tokens * hidden * 4 + (64 << 20), timeout_ms=3000)
    disp = ExpertParallelDispatcher(symm, num_experts=experts, hidden=hidden, max_tokens=tokens, topk=topk, capacity=tokens * topk, fp8=fp8,
                                    fp8_combine=fp8)
    g = torch.Generator(device="cuda").manual_seed(tokens)
    for _ in range(2):
        x = torch.randn((tokens, hidden), generator=g, device="cuda").to(torch.bfloat16)
        idx = torch.rand((tokens, experts), generator=g, device="cuda").topk(topk, dim=1).indices.to(torch.int32)
        idx[0, -1] = -1  # an unused slot
        weights = torch.rand((tokens, topk), generator=g, device="cuda")
        recv, counts, slots = disp.dispatch(x, idx)
        used = idx >= 0
        expect = torch.bincount(idx[used].long(), minlength=experts)
        assert torch.equal(counts.long().cpu(), torch.cat([expect, expect.sum(0, keepdim=True)]).cpu())
        first = torch.cumsum(expect, 0) - expect
        assert torch.equal(slots[used].sort().values.long(), torch.arange(int(used.sum()), device="cuda"))
        e = idx[used].long()
        assert bool(((slots[used] >= first[e]) & (slots[used] < first[e] + expect[e])).all())
        assert bool((slots[~used] == -1).all())
        token = torch.arange(tokens, device="cuda")[:, None].expand(-1, topk)[used]
        assert torch.equal(disp.recv_src[slots[used].long()].long(), token)
        rows = dequantize_rows(recv, disp.recv_scales) if fp8 else recv.float()
        got = rows[slots[used].long()]
        # e4m3 keeps three mantissa bits: half a unit in the last place is 2^-4 of the value, at least 2^-10 of the scaled range
        slack = x.float()[token].abs() / 16 + x.float()[token].abs().amax(1, keepdim=True) / 448 / 1024 if fp8 else torch.zeros_like(got)
        assert bool(((got - x.float()[token]).abs() <= slack * 1.001).all())
        if fp8:
            disp.expert_out_q, disp.expert_out_scales = disp.recv_x, disp.recv_scales
        y = disp.combine(idx, weights, slots, expert_out=None if fp8 else recv)
        ref = torch.zeros((tokens, hidden), dtype=torch.float64, device="cuda")
        ref.index_add_(0, token, rows[slots[used].long()].double() * weights[used].double()[:, None])
        bound = ref.abs() * 2.0 ** -8 + torch.zeros_like(ref).index_add_(
            0, token, rows[slots[used].long()].double().abs() * weights[used].double()[:, None]) * (topk + 1) * 2.0 ** -23
        assert bool(((y.double() - ref).abs() <= bound).all())
        symm.check()
    symm.destroy()


@pytest.mark.parametrize("tokens,topk,n_blocks", [(4096, 4, 0), (4097, 4, 0), (2048, 4, 0), (2049, 4, 0), (2, 2, 0), (1000, 8, 7)])
def test_moe_one_rank_counts(tokens, topk, n_blocks):
    """Either side of the line up to which every block of a one-rank dispatch counts all pairs; fewer tokens than blocks, few blocks;
    every token routed to the same experts, and ids that name no expert."""
    from mscclpp_b200 import SymmetricMemory
    from mscclpp_b200.parallel.moe import ExpertParallelDispatcher

    hidden, experts = 256, 24
    symm = SymmetricMemory.emulated(1, nbytes=tokens * topk * hidden * 5 + tokens * hidden * 4 + (64 << 20), timeout_ms=3000)
    disp = ExpertParallelDispatcher(symm, num_experts=experts, hidden=hidden, max_tokens=tokens, topk=topk, capacity=tokens * topk)
    g = torch.Generator(device="cuda").manual_seed(tokens)
    x = torch.randn((tokens, hidden), generator=g, device="cuda").to(torch.bfloat16)
    same = (torch.arange(topk, device="cuda", dtype=torch.int32) * 3).expand(tokens, -1).contiguous()
    holes = same.clone()
    holes[::3, 0] = -1
    holes[1::5, -1] = experts
    for idx in (same, holes):
        disp.recv_x.zero_()
        recv, counts, slots = disp.dispatch(x, idx, n_blocks=n_blocks)
        torch.cuda.synchronize()
        symm.check()
        used = (idx >= 0) & (idx < experts)
        expect = torch.bincount(idx[used].long(), minlength=experts)
        assert torch.equal(counts.long(), torch.cat([expect, expect.sum(0, keepdim=True)]))
        assert bool((slots[~used] == -1).all())
        assert torch.equal(slots[used].sort().values.long(), torch.arange(int(used.sum()), device="cuda"))
        first = torch.cumsum(expect, 0) - expect
        e = idx[used].long()
        assert bool(((slots[used] >= first[e]) & (slots[used] < first[e] + expect[e])).all())
        token = torch.arange(tokens, device="cuda")[:, None].expand(-1, topk)[used]
        assert torch.equal(recv[slots[used].long()], x[token])
    symm.destroy()


@pytest.mark.parametrize("tokens,topk", [(3, 2), (1000, 8), (4096, 2), (1100, 8)])
@pytest.mark.parametrize("fp8", [False, True])
def test_moe_one_rank_chain(tokens, topk, fp8):
    """Dispatch and combine of one batch right behind those of another: each launch overlaps the one before it, which may still read or
    write the received rows, the slots and the counts. Without waiting, eagerly and from a graph, the same bits as one by one. (1100 x 8:
    the dispatch that does not overlap, between combines that do.)"""
    from mscclpp_b200 import SymmetricMemory
    from mscclpp_b200.parallel.moe import ExpertParallelDispatcher

    hidden, experts = 2048, 64
    symm = SymmetricMemory.emulated(1, nbytes=tokens * topk * hidden * 8 + tokens * hidden * 12 + (64 << 20), timeout_ms=3000)
    disp = ExpertParallelDispatcher(symm, num_experts=experts, hidden=hidden, max_tokens=tokens, topk=topk, capacity=tokens * topk, fp8=fp8, fp8_combine=fp8)
    if fp8:
        disp.expert_out_q, disp.expert_out_scales = disp.recv_x, disp.recv_scales
    else:
        disp.expert_out = disp.recv_x
    g = torch.Generator(device="cuda").manual_seed(tokens)
    batches = []
    for _ in range(3):
        x = torch.randn((tokens, hidden), generator=g, device="cuda").to(torch.bfloat16)
        idx = torch.rand((tokens, experts), generator=g, device="cuda").topk(topk, dim=1).indices.to(torch.int32)
        batches.append((x, idx, torch.rand((tokens, topk), generator=g, device="cuda"), symm.tensor((tokens, hidden), torch.bfloat16)))

    def run(each=lambda: None):
        for x, idx, weights, y in batches:
            slots = disp.dispatch(x, idx)[2]
            each()
            disp.combine(idx, weights, slots, out=y)
            each()

    def results():
        torch.cuda.synchronize()
        symm.check()
        got = [y.clone() for *_, y in batches] + [disp.recv_counts.clone()]
        for *_, y in batches:
            y.fill_(float("nan"))
        disp.recv_counts.zero_()
        torch.cuda.synchronize()
        return got

    run(torch.cuda.synchronize)
    expect = results()
    assert all(bool(torch.isfinite(e).all()) for e in expect)
    for _ in range(5):
        run()
        assert all(torch.equal(a, b) for a, b in zip(results(), expect))
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(side):
        with torch.cuda.graph(graph, stream=side):
            run()
    torch.cuda.current_stream().wait_stream(side)
    for _ in range(5):
        graph.replay()
        assert all(torch.equal(a, b) for a, b in zip(results(), expect))
    del graph
    symm.destroy()


@pytest.mark.parametrize("offset", [0, 8])
@pytest.mark.parametrize("tokens,hidden,topk", [(3, 256, 1), (70, 768, 3), (160, 2304, 8)])
def test_moe_dispatch_fp8_rows_at_eight_byte_offsets(tokens, hidden, topk, offset):
    """Quantised rows are stored in 16-byte words where the receive buffer allows it and in 8-byte words where it does not. Either
    way they are the bytes and scales of the stand-alone quantiser, and the bytes around the buffer stay as they are."""
    from mscclpp_b200 import SymmetricMemory, native
    from mscclpp_b200.parallel.moe import ExpertParallelDispatcher

    n, experts, rows = native(), 16, tokens * topk
    symm = SymmetricMemory.emulated(1, nbytes=rows * hidden * 8 + tokens * hidden * 4 + (64 << 20), timeout_ms=3000)
    disp = ExpertParallelDispatcher(symm, num_experts=experts, hidden=hidden, max_tokens=tokens, topk=topk, capacity=rows + 1, fp8=True)
    whole = disp.recv_x.view(-1)
    whole.fill_(0xA5)
    disp.recv_x, disp.capacity = whole[offset:offset + rows * hidden].view(rows, hidden), rows
    assert disp.recv_x.data_ptr() % 16 == offset
    g = torch.Generator(device="cuda").manual_seed(tokens)
    x = torch.randn((tokens, hidden), generator=g, device="cuda").to(torch.bfloat16)
    idx = torch.rand((tokens, experts), generator=g, device="cuda").topk(topk, dim=1).indices.to(torch.int32)
    recv, _, slots = disp.dispatch(x, idx)
    q = torch.empty((tokens, hidden), dtype=torch.uint8, device="cuda")
    scales = torch.empty((tokens, hidden // 128), dtype=torch.float32, device="cuda")
    n.moe_quantize_rows(x.data_ptr(), q.data_ptr(), scales.data_ptr(), tokens, hidden, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    symm.check()
    for k in range(topk):
        assert torch.equal(recv[slots[:, k].long()], q)
        assert torch.equal(disp.recv_scales[slots[:, k].long()], scales)
    assert bool((whole[:offset] == 0xA5).all()) and bool((whole[offset + rows * hidden:] == 0xA5).all())
    symm.destroy()


@pytest.mark.parametrize("tokens,hidden,topk", [(5, 256, 1), (19, 768, 2), (21, 2304, 3), (40, 8192, 5), (17, 1280, 8), (300, 2048, 8)])
@pytest.mark.parametrize("fp8", [False, True])
def test_moe_combine_piece_sizes(tokens, hidden, topk, fp8):
    """The combine takes longer or shorter pieces of the rows, and of more or fewer rows together, by how many warps the launch
    has: from one thread block to 148, with ragged last pieces. Each element is the same fp32 sum in the same order in all of
    them; its distance from the 64-bit sum is bounded by topk + 1 fp32 roundings and one of bf16."""
    from mscclpp_b200 import SymmetricMemory
    from mscclpp_b200.parallel.moe import ExpertParallelDispatcher, dequantize_rows

    experts = 16
    symm = SymmetricMemory.emulated(1, nbytes=tokens * topk * hidden * 8 + tokens * hidden * 4 + (64 << 20), timeout_ms=3000)
    disp = ExpertParallelDispatcher(symm, num_experts=experts, hidden=hidden, max_tokens=tokens, topk=topk, capacity=tokens * topk,
                                    fp8_combine=fp8)
    g = torch.Generator(device="cuda").manual_seed(tokens + hidden)
    x = torch.randn((tokens, hidden), generator=g, device="cuda").to(torch.bfloat16)
    idx = torch.rand((tokens, experts), generator=g, device="cuda").topk(topk, dim=1).indices.to(torch.int32)
    idx[tokens // 2, topk // 2] = -1  # an unused slot
    weights = torch.rand((tokens, topk), generator=g, device="cuda")
    _, _, slots = disp.dispatch(x, idx)
    rows = tokens * topk
    disp.expert_out.copy_(torch.randn((rows, hidden), generator=g, device="cuda"))
    if fp8:
        disp.quantize_expert_out(rows)
    values = dequantize_rows(disp.expert_out_q, disp.expert_out_scales) if fp8 else disp.expert_out.float()
    w = torch.where(idx >= 0, weights, torch.zeros_like(weights)).double()
    terms = values.double()[slots.clamp(min=0).long()] * w[:, :, None]
    ref, bound = terms.sum(1), terms.sum(1).abs() * 2.0 ** -8 + terms.abs().sum(1) * (topk + 2) * 2.0 ** -23
    first = None
    for n_blocks in (1, 2, 6, 30, 148):
        disp.y.fill_(float("nan"))
        y = disp.combine(idx, weights, slots, n_blocks=n_blocks)
        symm.check()
        assert bool(((y.double() - ref).abs() <= bound).all())
        first = y.clone() if first is None else first
        assert torch.equal(y, first)
    symm.destroy()


@pytest.mark.parametrize("world,experts,tokens,hidden,topk", [(2, 8, 120, 512, 2), (8, 64, 48, 4096, 2), (4, 16, 64, 1024, 4)])
def test_moe_combine_fp8_payload(world, experts, tokens, hidden, topk):
    """Combine with e4m3 expert outputs (1 x 128 scales): the stand-alone quantiser against a PyTorch model of it, then the
    combined rows against the fp32 weighted sum of the bf16 expert outputs (tolerance of the e4m3 rounding)."""
    from mscclpp_b200 import SymmetricMemory
    from mscclpp_b200.parallel.moe import ExpertParallelDispatcher, dequantize_rows

    symm = SymmetricMemory.emulated(world, nbytes=256 << 20, timeout_ms=3000)
    disp = ExpertParallelDispatcher(symm, num_experts=experts, hidden=hidden, max_tokens=tokens, topk=topk, fp8_combine=True)
    el = experts // world
    g = torch.Generator(device="cuda").manual_seed(world * 77 + tokens)
    for rep in range(2):
        xs = [torch.randn((tokens, hidden), generator=g, device="cuda").to(torch.bfloat16) for _ in range(world)]
        idxs = [torch.stack([torch.randperm(experts, generator=g, device="cuda")[:topk] for _ in range(tokens)]).to(torch.int32) for _ in range(world)]
        wts = [torch.rand((tokens, topk), generator=g, device="cuda") for _ in range(world)]
        for r in range(world):
            x_s, idx_s, w_s = disp.stage(r, xs[r], idxs[r], wts[r])
        recv_x, counts, slot_map = disp.dispatch(x_s, idx_s, n_blocks=4)
        torch.cuda.synchronize()
        symm.check()
        for d in range(world):
            cnt = symm.rank_view(counts, d).cpu().tolist()
            rows = symm.rank_view(recv_x, d)
            out = symm.rank_view(disp.expert_out, d)
            start = 0
            for j in range(el):
                out[start:start + cnt[j]] = (rows[start:start + cnt[j]].float() * (0.5 * (d * el + j + 1))).to(torch.bfloat16)
                start += cnt[j]
            disp.quantize_expert_out(cnt[el], rank=d)
            torch.cuda.synchronize()
            # the quantiser: scale = amax / 448 per 128 elements, values within one e4m3 step of the input
            val = out[:cnt[el]].float()
            scales = symm.rank_view(disp.expert_out_scales, d)[:cnt[el]]
            want_scale = val.view(cnt[el], -1, 128).abs().amax(-1) / 448.0
            want_scale = torch.where(want_scale > 0, want_scale, torch.ones_like(want_scale))
            assert torch.allclose(scales, want_scale, rtol=1e-5, atol=0)
            back = dequantize_rows(symm.rank_view(disp.expert_out_q, d)[:cnt[el]], scales)
            assert (back - val).abs().max().item() <= 0.07 * val.abs().max().item()
        y = disp.combine(idx_s, w_s, slot_map, n_blocks=4)
        torch.cuda.synchronize()
        symm.check()
        ref = _moe_reference(xs, idxs, wts, world, experts, lambda e, rows: (rows * (0.5 * (e + 1))).to(torch.bfloat16).float())
        for r in range(world):
            got = symm.rank_view(y, r).float()
            assert (got - ref[r]).abs().max().item() <= 0.08 * ref[r].abs().max().item() + 0.02, (r, rep)
    symm.destroy()


def test_moe_dispatch_reports_small_receive_buffer():
    """A receive buffer that cannot hold the routed rows is reported as an error; nothing is written out of bounds."""
    from mscclpp_b200 import SymmetricMemory, native
    from mscclpp_b200.parallel.moe import ExpertParallelDispatcher

    symm = SymmetricMemory.emulated(2, nbytes=64 << 20, timeout_ms=1000)
    disp = ExpertParallelDispatcher(symm, num_experts=4, hidden=256, max_tokens=64, topk=2, capacity=16)
    x = torch.ones((64, 256), dtype=torch.bfloat16, device="cuda")
    idx = torch.tensor([[0, 1]] * 64, dtype=torch.int32, device="cuda")  # everything goes to rank 0
    for r in range(2):
        x_s, idx_s, _ = disp.stage(r, x, idx)
    disp.dispatch(x_s, idx_s, n_blocks=2)
    torch.cuda.synchronize()
    with pytest.raises(native().Error):
        symm.check()
    assert int(symm.rank_view(disp.slot_map, 0).max()) == -1
    symm.heap.reset_status()
    symm.destroy()


@pytest.mark.parametrize("world,rows_per_rank", [(2, 256), (4, 512)])
def test_two_sm_core_in_fused_kernels(world, rows_per_rank):
    """The fused kernels on the two-SM GEMM core (256 x 256 tiles on CTA pairs, clusters of two): all-gather -> GEMM,
    GEMM -> reduce-scatter and the fused TP layer, all ranks emulated on one GPU."""
    from mscclpp_b200 import SymmetricMemory
    from mscclpp_b200.parallel.sp_layer import all_gather_gemm, gemm_reduce_scatter
    from mscclpp_b200.parallel.tp_layer import RowParallelLinearNorm

    symm = SymmetricMemory.emulated(world, nbytes=256 << 20, timeout_ms=3000)
    s_rows, k, n_cols = world * rows_per_rank, 256, 512
    g = torch.Generator(device="cuda").manual_seed(world + rows_per_rank)
    ctas = max(2, (24 // world) & ~1)
    # all-gather -> GEMM
    a_local = symm.tensor((rows_per_rank, k), torch.bfloat16)
    a_full = symm.tensor((s_rows, k), torch.bfloat16)
    out = symm.tensor((s_rows, n_cols), torch.bfloat16)
    ws = [(torch.randn((n_cols, k), generator=g, device="cuda") * 0.05).to(torch.bfloat16) for _ in range(world)]
    shards = [torch.randn((rows_per_rank, k), generator=g, device="cuda").to(torch.bfloat16) for _ in range(world)]
    for rep in range(2):
        for r in range(world):
            symm.rank_view(a_local, r).copy_(shards[r])
            symm.rank_view(out, r).zero_()
        all_gather_gemm(symm, a_local, a_full, ws, out, block_n=0, num_copiers=2, num_gemm_ctas=ctas)
        torch.cuda.synchronize()
        symm.check()
    full = torch.cat(shards).float()
    for r in range(world):
        ref = full @ ws[r].float().t()
        assert (symm.rank_view(out, r).float() - ref).abs().max().item() <= 0.02 * ref.abs().max().item() + 0.02
    # GEMM -> reduce-scatter
    partial = symm.tensor((s_rows, n_cols), torch.bfloat16)
    out_rs = symm.tensor((rows_per_rank, n_cols), torch.bfloat16)
    xs = [torch.randn((s_rows, k), generator=g, device="cuda").to(torch.bfloat16) for _ in range(world)]
    for rep in range(2):
        gemm_reduce_scatter(symm, xs, ws, partial, out_rs, nvls=False, block_n=0, num_reducers=2, num_gemm_ctas=ctas)
        torch.cuda.synchronize()
        symm.check()
    total = sum((x.float() @ w.float().t()).to(torch.bfloat16).float() for x, w in zip(xs, ws))
    for r in range(world):
        ref = total[r * rows_per_rank:(r + 1) * rows_per_rank]
        assert (symm.rank_view(out_rs, r).float() - ref).abs().max().item() <= 0.02 * ref.abs().max().item() + 0.05
    # fused TP layer (GEMM + allreduce + residual + RMSNorm)
    tokens = 512
    layer = RowParallelLinearNorm(symm, out_features=n_cols, k_shard=k, max_tokens=tokens)
    xt = [torch.randn((tokens, k), generator=g, device="cuda").to(torch.bfloat16) for _ in range(world)]
    residual = torch.randn((tokens, n_cols), generator=g, device="cuda").to(torch.bfloat16)
    for r in range(world):
        symm.rank_view(layer.residual_in, r)[:tokens].copy_(residual)
        symm.rank_view(layer.gamma, r).fill_(1.0)
    for mode in (0, 1):
        for rep in range(2):
            layer.forward_fused(xt[0], mode=mode, nvls=False, block_n=-1, num_reducers=2, num_gemm_ctas=ctas, emulated_inputs=list(zip(xt, ws)))
            torch.cuda.synchronize()
            symm.check()
        acc = sum((x.float() @ w.float().t()).to(torch.bfloat16).float() for x, w in zip(xt, ws))
        h = (acc.to(torch.bfloat16).float() + residual.float()).to(torch.bfloat16).float()
        y = (h * torch.rsqrt(h.pow(2).mean(-1, keepdim=True) + layer.eps)).to(torch.bfloat16).float()
        for r in range(world):
            assert (symm.rank_view(layer.residual_out, r)[:tokens].float() - h).abs().max().item() <= 0.02 * h.abs().max().item() + 0.05
            assert (symm.rank_view(layer.out, r)[:tokens].float() - y).abs().max().item() <= 0.1
    symm.destroy()


@pytest.mark.parametrize("m,n,k", [(256, 256, 64), (777, 512, 256), (2048, 1024, 512)])
def test_two_sm_gemm(m, n, k):
    from mscclpp_b200.ops.gemm import gemm_bf16

    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    a = torch.randn((m, k), generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn((n, k), generator=g, device="cuda") * 0.05).to(torch.bfloat16)
    d = gemm_bf16(a, w, two_sm=True)
    torch.cuda.synchronize()
    ref = a.float() @ w.float().t()
    assert (d.float() - ref).abs().max().item() <= 0.01 * ref.abs().max().item() + 0.01


@pytest.mark.parametrize("world,rows,hidden,with_residual", [(2, 100, 1024, True), (4, 64, 8192, True), (8, 333, 4096, False)])
def test_row_owner_allreduce_rmsnorm(world, rows, hidden, with_residual):
    """Standalone allreduce + residual + RMSNorm on the fused kernel's reducer (row owners, whole rows in registers)."""
    from mscclpp_b200 import SymmetricMemory, native

    n = native()
    symm = SymmetricMemory.emulated(world, nbytes=128 << 20, timeout_ms=3000)
    partial = symm.tensor((rows, hidden), torch.bfloat16)
    res_in = symm.tensor((rows, hidden), torch.bfloat16)
    res_out = symm.tensor((rows, hidden), torch.bfloat16)
    out = symm.tensor((rows, hidden), torch.bfloat16)
    gamma = symm.tensor((hidden,), torch.bfloat16)
    rinv = symm.tensor((rows,), torch.float32)
    g = torch.Generator(device="cuda").manual_seed(rows)
    parts = [torch.randn((rows, hidden), generator=g, device="cuda").to(torch.bfloat16) for _ in range(world)]
    residual = torch.randn((rows, hidden), generator=g, device="cuda").to(torch.bfloat16)
    gam = (1 + 0.1 * torch.randn((hidden,), generator=g, device="cuda")).to(torch.bfloat16)
    for r in range(world):
        symm.rank_view(partial, r).copy_(parts[r])
        symm.rank_view(res_in, r).copy_(residual)
        symm.rank_view(gamma, r).copy_(gam)
    mode = 1 if with_residual else 0
    for rep in range(2):
        for r in range(world):
            symm.rank_view(out, r).zero_()
        n.tp_reduce_norm(symm.heap, partial.data_ptr(), res_in.data_ptr() if with_residual else 0, res_out.data_ptr() if with_residual else 0,
                         out.data_ptr(), gamma.data_ptr(), rinv.data_ptr(), rows, hidden, 1e-5, 4, 0, mode, False,
                         torch.cuda.current_stream().cuda_stream)
        if mode == 1:
            for r in range(world):
                n.tp_scale_rows(symm.rank_view(res_out, r).data_ptr(), symm.rank_view(rinv, r).data_ptr(), gamma.data_ptr(),
                                symm.rank_view(out, r).data_ptr(), rows, hidden, torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        symm.check()
    acc = sum(p.float() for p in parts).to(torch.bfloat16).float()
    h = (acc + residual.float()).to(torch.bfloat16).float() if with_residual else acc
    y = (h * torch.rsqrt(h.pow(2).mean(-1, keepdim=True) + 1e-5) * gam.float()).to(torch.bfloat16).float()
    for r in range(world):
        assert (symm.rank_view(out, r).float() - y).abs().max().item() <= 0.1
        if with_residual:
            assert (symm.rank_view(res_out, r).float() - h).abs().max().item() <= 0.02 * h.abs().max().item() + 0.05
    symm.destroy()


@pytest.mark.parametrize("world", [2, 8])
@pytest.mark.parametrize("dtype", [torch.float8_e4m3fn, torch.float8_e5m2])
@pytest.mark.parametrize("algo", ["packet", "rsag_zero_copy"])
def test_fp8_allreduce_accumulates_in_fp32(world, dtype, algo):
    """FP8 inputs are summed in fp32 and rounded once: the result equals round(fp32 sum) and its error is never
    larger than that of summing in fp8 step by step (the property the reference checks in test_fp8_accum.py)."""
    from mscclpp_b200.ops import all_reduce

    symm = _symm(world)
    numel = 16384
    inp = symm.tensor((numel,), dtype)
    out = symm.tensor((numel,), dtype)
    vals = []
    for r in range(world):
        g = torch.Generator(device="cuda").manual_seed(900 + r)
        x = (torch.randn(numel, generator=g, device="cuda") * 0.5).to(dtype)
        symm.rank_view(inp, r).copy_(x)
        vals.append(x.float())
    all_reduce(symm, inp, out, algo=algo, n_blocks=4)
    torch.cuda.synchronize()
    symm.check()
    exact = torch.stack(vals).sum(0)
    oracle = exact.to(dtype).float()          # one rounding of the fp32 sum
    stepwise = vals[0].clone()
    for v in vals[1:]:
        stepwise = (stepwise + v).to(dtype).float()   # what accumulating in fp8 would give
    for r in range(world):
        got = symm.rank_view(out, r).float()
        assert torch.equal(got, oracle), (r, (got - oracle).abs().max().item())
    assert (oracle - exact).abs().mean().item() <= (stepwise - exact).abs().mean().item() + 1e-9
    symm.destroy()


@pytest.mark.parametrize("world", [2, 4, 8])
def test_broadcast_and_all_to_all(world):
    """Native broadcast (root streams into every rank) and all-to-all (peer stores), all ranks emulated on one GPU."""
    from mscclpp_b200.ops import all_to_all, broadcast

    symm = _symm(world)
    per = 4096
    src = symm.tensor((world * per,), torch.float32)
    dst = symm.tensor((world * per,), torch.float32)
    for r in range(world):
        symm.rank_view(src, r).copy_(torch.arange(world * per, device="cuda", dtype=torch.float32) + 100000 * r)
    for root in (0, world - 1):
        for r in range(world):
            symm.rank_view(dst, r).zero_()
        broadcast(symm, src, dst, root=root, nvls=False, n_blocks=4)
        torch.cuda.synchronize()
        symm.check()
        want = symm.rank_view(src, root)
        for r in range(world):
            assert torch.equal(symm.rank_view(dst, r), want)
    for r in range(world):
        symm.rank_view(dst, r).zero_()
    all_to_all(symm, src, dst, n_blocks=4)
    torch.cuda.synchronize()
    symm.check()
    for r in range(world):
        want = torch.cat([symm.rank_view(src, p)[r * per:(r + 1) * per] for p in range(world)])
        assert torch.equal(symm.rank_view(dst, r), want)
    symm.destroy()
