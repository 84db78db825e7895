"""tcgen05/TMEM bf16 GEMM against a PyTorch fp32 reference."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k,block_n", [
    (128, 256, 64, 256),
    (128, 256, 1024, 256),
    (256, 512, 128, 128),
    (1, 8192, 1024, 64),
    (8, 8192, 1024, 64),
    (200, 1024, 512, 128),
    (2048, 8192, 1024, 256),
    (777, 768, 320, 64),
    (4096, 4096, 512, 256),   # several bands of the L2-friendly tile order
    (2100, 2048, 192, 128),   # row tail inside the last band
])
def test_gemm_matches_fp32_reference(m, n, k, block_n):
    from mscclpp_b200.ops import gemm_bf16

    g = torch.Generator(device="cuda").manual_seed(m * 7 + n)
    a = torch.randn((m, k), generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn((n, k), generator=g, device="cuda") * 0.05).to(torch.bfloat16)
    out = torch.full((m, n), float("nan"), device="cuda", dtype=torch.bfloat16)
    gemm_bf16(a, w, out, block_n=block_n)
    torch.cuda.synchronize()
    ref = a.float() @ w.float().t()
    err = (out.float() - ref).abs().max().item()
    scale = ref.abs().max().item()
    assert err <= 1e-2 * scale + 1e-2, f"max err {err} (scale {scale})"


def test_gemm_auto_tile_and_repeat():
    from mscclpp_b200.ops import gemm_bf16

    a = torch.randn((512, 1024), device="cuda").to(torch.bfloat16)
    w = (torch.randn((2048, 1024), device="cuda") * 0.02).to(torch.bfloat16)
    ref = (a.float() @ w.float().t())
    for _ in range(3):
        out = gemm_bf16(a, w)
        torch.cuda.synchronize()
        assert (out.float() - ref).abs().max().item() <= 1e-2 * ref.abs().max().item() + 1e-2


@pytest.mark.parametrize("m,n,k", [(512, 512, 256), (4096, 8192, 1024), (1000, 1024, 512)])
def test_gemm_two_sm_tiles(m, n, k):
    from mscclpp_b200.ops import gemm_bf16

    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    a = torch.randn((m, k), generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn((n, k), generator=g, device="cuda") * 0.05).to(torch.bfloat16)
    out = torch.full((m, n), float("nan"), device="cuda", dtype=torch.bfloat16)
    gemm_bf16(a, w, out, two_sm=True)
    torch.cuda.synchronize()
    ref = a.float() @ w.float().t()
    assert (out.float() - ref).abs().max().item() <= 1e-2 * ref.abs().max().item() + 1e-2


def test_gemm_form_on_this_gpu():
    """The device says how many clusters of four it holds; a whole B200 holds as many as the costs were fitted with."""
    from mscclpp_b200 import native

    n = native()
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("not a whole B200")
    for m in (9, 33, 80, 200, 645, 1500):
        for nn in (512, 704, 1408, 2048, 4096):
            for k in (512, 2048, 4992, 8192):
                assert n.gemm_plan_form(m, nn, k) == n.gemm_plan_form(m, nn, k, 148, 34)


# (rows per pair of SMs or 0, columns, CTAs that share a tile)
FORMS = [(0, 64, 1), (0, 64, 4), (0, 128, 1), (0, 256, 1), (256, 256, 1), (128, 256, 1), (128, 128, 1)]


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("m,n,k", [
    (1, 64, 256),        # one row, one block of columns
    (129, 320, 320),     # one row and one block of columns more than tiles have; an odd number of k blocks
    (77, 192, 576),      # (and of parts of the reduction)
    (128, 256, 4096),    # the ring of stages many times round
    (2000, 4160, 192),   # several tiles per SM or pair
])
def test_gemm_forms(form, m, n, k):
    from mscclpp_b200 import native

    if k // 64 < form[2]:
        pytest.skip("more parts than k blocks")
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    a = torch.randn((m, k), generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn((n, k), generator=g, device="cuda") * 0.05).to(torch.bfloat16)
    buf = torch.full((m * n + 4096,), 7.0, device="cuda", dtype=torch.bfloat16)  # what lies behind the result stays as it is
    out = buf[:m * n].view(m, n)
    ref = a.double() @ w.double().t()
    # one rounding to bf16 (eight significant bits: half a unit in the last place is at most 2^-8 of the value) of an fp32 sum,
    # whose own error is at most K roundings of the sum of the products' magnitudes
    bound = ref.abs() * 2.0 ** -8 * 1.01 + (a.double().abs() @ w.double().abs().t()) * k * 2.0 ** -24
    for rep in range(2):
        out.fill_(float("nan"))
        native().gemm_bf16_form(a.data_ptr(), w.data_ptr(), out.data_ptr(), m, n, k, n, torch.cuda.current_stream().cuda_stream, *form)
        torch.cuda.synchronize()
        assert bool(((out.double() - ref).abs() <= bound).all())
    assert bool((buf[m * n:] == 7.0).all())


@pytest.mark.parametrize("one_kernel", [True, False])
@pytest.mark.parametrize("tokens,hidden,k,two_sm", [(200, 1024, 256, False), (1024, 2048, 512, True), (777, 512, 128, False),
                                                    (1, 8192, 1024, False), (2048, 8192, 1024, True), (1333, 2048, 256, True)])
def test_single_gpu_layer_gemm_epilogue_residual_sumsq(tokens, hidden, k, two_sm, one_kernel):
    """One GPU: GEMM whose epilogue adds the residual and accumulates the rows' sums of squares; the normalisation either
    in the same launch (rows handed to the epilogue warps block by block) or as a second, local pass."""
    import os

    from mscclpp_b200 import SymmetricMemory
    from mscclpp_b200.parallel.tp_layer import RowParallelLinearNorm

    symm = SymmetricMemory.emulated(1, nbytes=512 << 20, timeout_ms=3000)
    layer = RowParallelLinearNorm(symm, out_features=hidden, k_shard=k, max_tokens=tokens)
    g = torch.Generator(device="cuda").manual_seed(tokens)
    x = torch.randn((tokens, k), generator=g, device="cuda").to(torch.bfloat16)
    residual = torch.randn((tokens, hidden), generator=g, device="cuda").to(torch.bfloat16)
    layer.gamma.copy_((1 + 0.1 * torch.randn((hidden,), generator=g, device="cuda")).to(torch.bfloat16))
    for rep in range(2):
        layer.out.fill_(float("nan"))
        out, res = layer.forward_local(x, residual, two_sm=two_sm, one_kernel=one_kernel)
        torch.cuda.synchronize()
    h = ((x.float() @ layer.weight.float().t()).to(torch.bfloat16).float() + residual.float()).to(torch.bfloat16).float()
    y = (h * torch.rsqrt(h.pow(2).mean(-1, keepdim=True) + layer.eps) * layer.gamma.float()).to(torch.bfloat16).float()
    assert (res.float() - h).abs().max().item() <= 0.02 * h.abs().max().item() + 0.05
    assert (out.float() - y).abs().max().item() <= 0.1
    symm.destroy()


@pytest.mark.parametrize("tokens", [1, 63, 129, 700])
@pytest.mark.parametrize("hidden,k,tile", [
    (1024, 320, (128, 128)),   # (an odd number of k blocks)
    (1024, 320, (128, 256)),
    (5120, 256, (128, 256)),   # several tiles per pair of SMs
    (1152, 576, (0, 0)),       # the tile that the shape gets: N is a multiple of 128 only
    (1088, 320, (0, 0)),       # ... of 64 only
])
def test_single_gpu_layer_gemm_tiles_of_128_rows(tokens, hidden, k, tile):
    """The product with its epilogue in tiles of 128 rows on pairs of SMs, and where the width leaves no choice: h, and the sums of
    squares that the scale pass makes 1/rms of."""
    from mscclpp_b200 import native

    g = torch.Generator(device="cuda").manual_seed(tokens + hidden)
    x = torch.randn((tokens, k), generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn((hidden, k), generator=g, device="cuda") * 0.05).to(torch.bfloat16)
    residual = torch.randn((tokens, hidden), generator=g, device="cuda").to(torch.bfloat16)
    buf = torch.full((tokens * hidden + 4096,), 7.0, device="cuda", dtype=torch.bfloat16)
    h = buf[:tokens * hidden].view(tokens, hidden)
    sums = torch.full((hidden // 64 * tokens + 64,), -1.0, device="cuda")
    product = x.double() @ w.double().t()
    ref = product + residual.double()
    # the product is rounded to bf16 and the sum again: 2^-8 of either value; the fp32 sum's own error as in test_gemm_forms
    bound = (product.abs() + ref.abs()) * 2.0 ** -8 * 1.01 + (x.double().abs() @ w.double().abs().t()) * k * 2.0 ** -24
    for _ in range(2):
        h.fill_(float("nan"))
        parts = native().gemm_residual_sumsq(x.data_ptr(), w.data_ptr(), residual.data_ptr(), h.data_ptr(), sums.data_ptr(), tokens, hidden, k,
                                             tile[1], False, torch.cuda.current_stream().cuda_stream, tile[0] or -1)
        torch.cuda.synchronize()
        assert bool(((h.double() - ref).abs() <= bound).all())
        total = sums[:parts * tokens].view(parts, tokens).double().sum(0)
        want = h.double().square().sum(1)
        assert bool(((total - want).abs() <= want * hidden * 2.0 ** -24).all())
    assert bool((buf[tokens * hidden:] == 7.0).all()) and bool((sums[parts * tokens:] == -1.0).all())


@pytest.mark.parametrize("tokens,hidden,k", [
    (256, 256, 64),      # one tile, one block of the reduction
    (257, 2048, 192),    # a row block with one row, warps without rows
    (1333, 2048, 256),   # rows beyond M inside a box
    (2305, 8192, 128),   # several tiles per pair of SMs, a band of 2048 rows and a rest
    (1000, 4096, 2048),
])
@pytest.mark.parametrize("with_residual", [True, False])
def test_single_gpu_layer_on_pairs_of_sms(tokens, hidden, k, with_residual):
    """The two-launch layer on two-SM tiles: residual boxes by bulk loads, h by bulk stores, sums of squares per lane, then
    the scale pass. Bounds: fp32 accumulation (k * 2^-24 of the products' magnitudes), one bf16 rounding before and one
    after the residual is added, one of the output."""
    from mscclpp_b200 import SymmetricMemory, native
    from mscclpp_b200.parallel.tp_layer import RowParallelLinearNorm

    n = native()
    symm = SymmetricMemory.emulated(1, nbytes=256 << 20, timeout_ms=3000)
    layer = RowParallelLinearNorm(symm, out_features=hidden, k_shard=k, max_tokens=tokens)
    g = torch.Generator(device="cuda").manual_seed(tokens + k)
    layer.gamma.copy_((1 + 0.1 * torch.randn((hidden,), generator=g, device="cuda")).to(torch.bfloat16))
    parts = torch.full((tokens * hidden // 128,), float("nan"), device="cuda")
    for _ in range(2):
        x = torch.randn((tokens, k), generator=g, device="cuda").to(torch.bfloat16)
        residual = torch.randn((tokens, hidden), generator=g, device="cuda").to(torch.bfloat16)
        layer.out.fill_(float("nan"))
        layer.residual_out.fill_(float("nan"))
        if with_residual:
            out, res = layer.forward_local(x, residual, two_sm=True, one_kernel=False)
        else:
            out, res = layer.out, layer.residual_out
            s = torch.cuda.current_stream().cuda_stream
            num = n.gemm_residual_sumsq(x.data_ptr(), layer.weight.data_ptr(), 0, res.data_ptr(), parts.data_ptr(), tokens, hidden, k, 256, True, s)
            n.tp_scale_rows_from_sumsq(res.data_ptr(), parts.data_ptr(), num, layer.gamma.data_ptr(), out.data_ptr(), tokens, hidden, layer.eps, s)
        torch.cuda.synchronize()
        p = x.double() @ layer.weight.double().t()
        h = p + residual.double() if with_residual else p
        slack = (x.double().abs() @ layer.weight.double().abs().t()) * k * 2.0 ** -24 + p.abs() * 2.0 ** -8 + h.abs() * 2.0 ** -8
        assert bool(((res.double() - h).abs() <= slack).all())
        y = res.double() * torch.rsqrt(res.double().square().mean(-1, keepdim=True) + layer.eps) * layer.gamma.double()
        assert bool(((out.double() - y).abs() <= y.abs() * 2.0 ** -8).all())
    symm.destroy()


@pytest.mark.parametrize("tokens,hidden,k", [
    (256, 256, 64),      # one tile
    (257, 2048, 192),    # a row block with one row
    (2305, 8192, 128),   # several waves, and row blocks that straddle two of them
    (1999, 6400, 1024),  # 25 tiles per row block; rows beyond M inside a scale warp's sixteen
    (8192, 2048, 1088),
])
def test_single_gpu_layer_in_waves(tokens, hidden, k):
    """The one-launch layer that keeps h on chip: with and without residual and gamma, twice in a row (the counters it leaves are
    those it needs). Bounds as for the two-launch form above."""
    from mscclpp_b200 import SymmetricMemory, native

    n = native()
    symm = SymmetricMemory.emulated(1, nbytes=64 << 20, timeout_ms=3000)
    g = torch.Generator(device="cuda").manual_seed(tokens + k)
    w = (0.05 * torch.randn((hidden, k), generator=g, device="cuda")).to(torch.bfloat16)
    gamma = (1 + 0.1 * torch.randn((hidden,), generator=g, device="cuda")).to(torch.bfloat16)
    parts = torch.full(((tokens + 255) // 256 * 256 * hidden // 128,), float("nan"), device="cuda")
    counters = torch.zeros((n.tp_layer_wave_counter_words(tokens),), dtype=torch.int32, device="cuda")
    for residual, gam in ((True, gamma), (True, None), (False, gamma), (True, gamma)):
        x = torch.randn((tokens, k), generator=g, device="cuda").to(torch.bfloat16)
        r = torch.randn((tokens, hidden), generator=g, device="cuda").to(torch.bfloat16)
        out, res = (torch.full((tokens, hidden), float("nan"), device="cuda", dtype=torch.bfloat16) for _ in range(2))
        n.tp_layer_wave(symm.heap, x.data_ptr(), w.data_ptr(), r.data_ptr() if residual else 0, res.data_ptr(), out.data_ptr(),
                        0 if gam is None else gam.data_ptr(), parts.data_ptr(), counters.data_ptr(), tokens, hidden, k, 1e-5,
                        torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        symm.check()
        assert not bool(counters.any())
        p = x.double() @ w.double().t()
        h = p + r.double() if residual else p
        slack = (x.double().abs() @ w.double().abs().t()) * k * 2.0 ** -24 + p.abs() * 2.0 ** -8 + h.abs() * 2.0 ** -8
        assert bool(((res.double() - h).abs() <= slack).all())
        y = res.double() * torch.rsqrt(res.double().square().mean(-1, keepdim=True) + 1e-5) * (1.0 if gam is None else gam.double())
        assert bool(((out.double() - y).abs() <= y.abs() * 2.0 ** -8).all())
    with pytest.raises(Exception):  # a row block has to fit two waves
        n.tp_layer_wave(symm.heap, x.data_ptr(), w.data_ptr(), 0, res.data_ptr(), out.data_ptr(), 0, parts.data_ptr(), counters.data_ptr(), 256,
                        256 * 149, 64, 1e-5, torch.cuda.current_stream().cuda_stream)
    symm.destroy()


def test_single_gpu_layer_default_forms_in_a_chain():
    """forward_local as it is called, no form forced: long prompts in one launch between shorter ones in two, all reading what the
    launch before wrote; pieces of the rows with an offset; without waiting the same bits as one by one. Against fp64 at the end."""
    from mscclpp_b200 import SymmetricMemory, native
    from mscclpp_b200.parallel.tp_layer import RowParallelLinearNorm

    size, short, long = 2048, 1280, 28 * 256 + 37  # 8 tiles a row block: 40 tiles, 232 tiles
    total = short + long
    assert native().tp_layer_wave_fits(8192) and not RowParallelLinearNorm._wave_form(short, size, size)
    assert RowParallelLinearNorm._wave_form(long, size, size) and RowParallelLinearNorm._wave_form(total, size, size)
    symm = SymmetricMemory.emulated(1, nbytes=3 * total * size * 8 + (64 << 20), timeout_ms=3000)
    layers = [RowParallelLinearNorm(symm, out_features=size, k_shard=size, max_tokens=total, seed=i) for i in range(3)]
    g = torch.Generator(device="cuda").manual_seed(11)
    for layer in layers:
        layer.out.zero_()
        layer.residual_out.zero_()
        layer.residual_in.copy_(torch.randn((total, size), generator=g, device="cuda"))
    layers[1].residual_in, layers[2].residual_in = layers[0].residual_out, layers[1].residual_out
    x = torch.randn((total, size), generator=g, device="cuda").to(torch.bfloat16)

    def step(i, rows, src):
        return lambda: layers[i].forward_local(src[rows], row_offset=rows.start)

    first, rest, every = slice(0, short), slice(short, total), slice(0, total)
    chain = [step(0, first, x), step(0, rest, x), step(1, every, layers[0].out), step(2, rest, layers[1].out), step(2, first, layers[1].out)]
    _same_without_waiting(chain, [t for layer in layers for t in (layer.out, layer.residual_out)])
    symm.check()
    assert not any(bool(layer._wave_counters.any()) for layer in layers)
    for launch in chain:
        launch()
    torch.cuda.synchronize()
    rows = torch.randint(0, total, (300,), generator=g, device="cuda")
    src, residual = x, layers[0].residual_in
    for layer in layers:
        p = src[rows].double() @ layer.weight.double().t()
        h, got = p + residual[rows].double(), layer.residual_out[rows].double()
        slack = (src[rows].double().abs() @ layer.weight.double().abs().t()) * size * 2.0 ** -24 + p.abs() * 2.0 ** -8 + h.abs() * 2.0 ** -8
        assert bool(((got - h).abs() <= slack).all())
        y = got * torch.rsqrt(got.square().mean(-1, keepdim=True) + layer.eps)
        assert bool(((layer.out[rows].double() - y).abs() <= y.abs() * 2.0 ** -8).all())
        src, residual = layer.out, layer.residual_out
    symm.destroy()


def test_single_gpu_layer_in_waves_from_host_memory():
    """forward_from_host in pieces that are long prompts themselves (row offsets into the parts and the counters)."""
    from mscclpp_b200 import SymmetricMemory
    from mscclpp_b200.parallel.tp_layer import RowParallelLinearNorm

    tokens, hidden, k = 2 * 1792 + 5, 8192, 1024  # 7 row blocks x 32 tiles in each of two pieces, a piece of five rows behind them
    assert RowParallelLinearNorm._wave_form(1792, hidden, k)
    symm = SymmetricMemory.emulated(1, nbytes=tokens * hidden * 8 + (64 << 20), timeout_ms=3000)
    layer = RowParallelLinearNorm(symm, out_features=hidden, k_shard=k, max_tokens=tokens)
    layer.residual_in.normal_()
    x = torch.randn((tokens, k)).to(torch.bfloat16).pin_memory()
    layer.forward_from_host(x, chunks=3)
    torch.cuda.synchronize()
    got = layer.out.clone(), layer.residual_out.clone()
    layer.out.zero_()
    layer.residual_out.zero_()
    layer.forward_local(x.cuda(), one_kernel=False)
    torch.cuda.synchronize()
    symm.check()
    assert torch.equal(got[1], layer.residual_out)
    # two orders of the rows' sums: 1/rms to fp32 rounding, `out` to one bf16 rounding
    assert bool(((got[0].double() - layer.out.double()).abs() <= layer.out.double().abs() * 2.0 ** -7).all())
    symm.destroy()


def test_single_gpu_layer_in_waves_gives_up():
    """A row block that is never complete (its counter starts below zero): the waits for it run out, the launch ends, the status says
    so, the counters are zero again and the next launch is right. One tile per pair of SMs, so that nothing is in flight when
    the waits run out."""
    from mscclpp_b200 import SymmetricMemory, native

    n = native()
    tokens, hidden, k = 1024, 1024, 128
    x, w, r = (torch.randn(s, device="cuda").to(torch.bfloat16) for s in ((tokens, k), (hidden, k), (tokens, hidden)))
    parts = torch.empty((tokens * hidden // 128,), device="cuda")
    counters = torch.zeros((n.tp_layer_wave_counter_words(tokens),), dtype=torch.int32, device="cuda")

    def launch(symm):
        out, h = torch.zeros_like(r), torch.zeros_like(r)
        n.tp_layer_wave(symm.heap, x.data_ptr(), w.data_ptr(), r.data_ptr(), h.data_ptr(), out.data_ptr(), 0, parts.data_ptr(), counters.data_ptr(),
                        tokens, hidden, k, 1e-5, torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        return out, h

    symm = SymmetricMemory.emulated(1, nbytes=64 << 20, timeout_ms=50)
    counters[1 + 3] = -1  # 128-row block 3
    launch(symm)
    with pytest.raises(Exception):
        symm.check()
    assert not bool(counters.any())
    symm.destroy()
    symm = SymmetricMemory.emulated(1, nbytes=64 << 20, timeout_ms=3000)
    out, h = launch(symm)
    symm.check()
    p = x.double() @ w.double().t()
    assert bool(((h.double() - p - r.double()).abs() <= (x.double().abs() @ w.double().abs().t()) * k * 2.0 ** -24 + p.abs() * 2.0 ** -8 + h.double().abs() * 2.0 ** -7).all())
    assert bool(torch.isfinite(out).all())
    symm.destroy()


@pytest.mark.parametrize("rows,n,parts", [(1, 8, 1), (3, 72, 2), (445, 1000, 5), (444 * 32 + 7, 256, 4), (900, 8192, 64), (37, 16392, 128)])
def test_scale_pass_sizes(rows, n, parts):
    """out = h * rsqrt(sum of the row's parts / n + eps) * gamma at the edges of the pass: rows of less than a warp's words,
    of several batches per thread, more rows than resident blocks take at once. One bf16 rounding of an fp32 product."""
    from mscclpp_b200 import native

    nat = native()
    g = torch.Generator(device="cuda").manual_seed(rows + n)
    h = torch.randn((rows, n), generator=g, device="cuda").to(torch.bfloat16)
    table = torch.rand((parts, rows), generator=g, device="cuda") * n
    gamma = (1 + 0.1 * torch.randn((n,), generator=g, device="cuda")).to(torch.bfloat16)
    out = torch.full((rows, n), float("nan"), device="cuda", dtype=torch.bfloat16)
    for gam in (gamma, None):
        nat.tp_scale_rows_from_sumsq(h.data_ptr(), table.data_ptr(), parts, 0 if gam is None else gam.data_ptr(), out.data_ptr(), rows, n, 1e-5,
                                     torch.cuda.current_stream().cuda_stream)
        y = h.double() * torch.rsqrt(table.double().sum(0) / n + 1e-5)[:, None] * (1.0 if gam is None else gam.double())
        assert bool(((out.double() - y).abs() <= y.abs() * (2.0 ** -8)).all())


def _same_without_waiting(launches, outputs):
    """Runs `launches` with a synchronisation after each, then without one between them, eagerly and replayed from a CUDA
    graph: the contents of `outputs` have to be the same bits every time."""
    def run(each=lambda: None):
        for launch in launches:
            launch()
            each()

    def results():
        torch.cuda.synchronize()
        got = [o.clone() for o in outputs]
        for o in outputs:
            o.fill_(float("nan"))
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


@pytest.mark.parametrize("tokens,two_sm", [(100, False), (333, False), (1000, False), (333, True), (2305, True)])
def test_chained_layers_wait_for_one_another(tokens, two_sm):
    """Launches that overlap the one before them, back to back: a GEMM that reads what the scale pass just before it writes
    (x) and what the GEMM before that wrote (its residual), and a second pass over the same layer, whose GEMM overwrites the
    sums and h that the first scale pass reads."""
    from mscclpp_b200 import SymmetricMemory
    from mscclpp_b200.parallel.tp_layer import RowParallelLinearNorm

    hidden = 1024
    symm = SymmetricMemory.emulated(1, nbytes=256 << 20, timeout_ms=3000)
    layers = [RowParallelLinearNorm(symm, out_features=hidden, k_shard=hidden, max_tokens=tokens, seed=i) for i in range(4)]
    g = torch.Generator(device="cuda").manual_seed(tokens)
    x = torch.randn((tokens, hidden), generator=g, device="cuda").to(torch.bfloat16)
    other = torch.randn((tokens, hidden), generator=g, device="cuda").to(torch.bfloat16)
    first = torch.randn((tokens, hidden), generator=g, device="cuda").to(torch.bfloat16)
    for i, layer in enumerate(layers):
        layer.residual_in = first if i == 0 else layers[i - 1].residual_out

    def step(i, a):
        return lambda: layers[i].forward_local(a, two_sm=two_sm, one_kernel=False)

    chain = [step(i, x if i == 0 else layers[i - 1].out[:tokens]) for i in range(4)]
    _same_without_waiting(chain, [t for layer in layers for t in (layer.out, layer.residual_out)])
    _same_without_waiting([step(0, other), step(0, x), step(1, layers[0].out[:tokens]), step(0, other), step(2, layers[0].out[:tokens])],
                          [t for layer in layers[:3] for t in (layer.out, layer.residual_out)])
    symm.destroy()


@pytest.mark.parametrize("m,two_sm", [(100, False), (777, False), (777, True), (2304, True)])
def test_chained_gemms_wait_for_one_another(m, two_sm):
    """Each product is the A operand of the next one, or its residual; every second buffer is written again while the launch
    before may still read it. A copy (a node that is no kernel) stands in the middle."""
    from mscclpp_b200 import native
    from mscclpp_b200.ops import gemm_bf16

    n, size = native(), 512
    g = torch.Generator(device="cuda").manual_seed(m)
    w = (torch.randn((size, size), generator=g, device="cuda") * size ** -0.5).to(torch.bfloat16)
    x = torch.randn((m, size), generator=g, device="cuda").to(torch.bfloat16)
    bufs = [torch.full((m, size), float("nan"), device="cuda", dtype=torch.bfloat16) for _ in range(4)]
    parts = [torch.full((size // (128 if two_sm else 64), m), float("nan"), device="cuda") for _ in range(2)]

    def product(a, d):
        return lambda: gemm_bf16(a, w, d, two_sm=two_sm)

    def added(a, residual, h, sums):
        def launch():
            num = n.gemm_residual_sumsq(a.data_ptr(), w.data_ptr(), residual.data_ptr(), h.data_ptr(), sums.data_ptr(), m, size, size, 128,
                                        two_sm, torch.cuda.current_stream().cuda_stream)
            assert num == sums.shape[0]
        return launch

    _same_without_waiting([product(x, bufs[0]), product(bufs[0], bufs[1]), product(bufs[1], bufs[0]), lambda: bufs[2].copy_(bufs[0]),
                           product(bufs[2], bufs[1]), product(bufs[1], bufs[3])], bufs)
    _same_without_waiting([added(x, x, bufs[0], parts[0]), added(x, bufs[0], bufs[1], parts[1]), added(bufs[1], bufs[1], bufs[2], parts[0]),
                           added(x, bufs[2], bufs[0], parts[1]), added(bufs[0], bufs[0], bufs[3], parts[0])], bufs + parts)


@pytest.mark.parametrize("tokens,hidden,k", [
    (1, 8, 256),        # one block, eight columns
    (2, 1032, 256),     # the last block has eight columns of what others have
    (3, 1032, 512),     # pairs of blocks, the odd one out without columns
    (8, 5120, 2560),
    (5, 18944, 3072),   # the widest slab, whose tiles go six times around the ring
    (4, 18952, 256),    # wider: the cooperative form
])
def test_decode_layer_one_gpu(tokens, hidden, k):
    """The layer for a few tokens on one rank: with and without residual and gamma, launches back to back (the count they leave is
    the one they need). Bounds: fp32 accumulation, one bf16 rounding before and one after the residual, one of the output."""
    from mscclpp_b200 import SymmetricMemory, native
    from mscclpp_b200.parallel.tp_layer import RowParallelLinearNorm

    n = native()
    symm = SymmetricMemory.emulated(1, nbytes=64 << 20, timeout_ms=3000)
    layer = RowParallelLinearNorm(symm, out_features=hidden, k_shard=k, max_tokens=tokens, init_std=0.05)
    g = torch.Generator(device="cuda").manual_seed(tokens + hidden)
    layer.gamma.copy_((1 + 0.1 * torch.randn((hidden,), generator=g, device="cuda")).to(torch.bfloat16))
    for plain in (False, True, False):
        x = torch.randn((tokens, k), generator=g, device="cuda").to(torch.bfloat16)
        residual = torch.randn((tokens, hidden), generator=g, device="cuda").to(torch.bfloat16)
        layer.out.fill_(float("nan"))
        layer.residual_out.fill_(float("nan"))
        if plain:
            n.tp_decode(symm.heap, [x.data_ptr()], [layer.weight.data_ptr()], 0, layer.residual_out.data_ptr(), layer.out.data_ptr(), 0, tokens, hidden,
                        k, layer.eps, False, 0, torch.cuda.current_stream().cuda_stream, 0, layer._decode_ws.data_ptr())
        else:
            for _ in range(3):
                layer.forward_decode(x, residual)
        torch.cuda.synchronize()
        symm.check()
        p = x.double() @ layer.weight.double().t()
        h = p if plain else p + residual.double()
        res, out = layer.residual_out[:tokens].double(), layer.out[:tokens].double()
        slack = (x.double().abs() @ layer.weight.double().abs().t()) * k * 2.0 ** -24 + p.abs() * 2.0 ** -8 + h.abs() * 2.0 ** -8
        assert bool(((res - h).abs() <= slack).all())
        y = res * torch.rsqrt(res.square().mean(-1, keepdim=True) + layer.eps) * (1.0 if plain else layer.gamma.double())
        assert bool(((out - y).abs() <= y.abs() * 2.0 ** -8).all())
    symm.destroy()


@pytest.mark.parametrize("tokens,hidden,k", [(1, 8192, 1024), (8, 5120, 2560), (3, 1032, 256), (5, 2048, 768), (2, 18944, 3072)])
def test_decode_layer_one_gpu_sums_in_the_order_of_the_cooperative_form(tokens, hidden, k):
    """h = product + residual is the same bits as from the launch that several ranks take (768 and 256: the last tiles leave two of the
    four slices of the reduction without work)."""
    from mscclpp_b200 import SymmetricMemory, native
    from mscclpp_b200.parallel.tp_layer import RowParallelLinearNorm

    symm = SymmetricMemory.emulated(1, nbytes=64 << 20, timeout_ms=3000)
    layer = RowParallelLinearNorm(symm, out_features=hidden, k_shard=k, max_tokens=tokens)
    g = torch.Generator(device="cuda").manual_seed(hidden + k)
    x = torch.randn((tokens, k), generator=g, device="cuda").to(torch.bfloat16)
    residual = torch.randn((tokens, hidden), generator=g, device="cuda").to(torch.bfloat16)
    h = layer.forward_decode(x, residual)[1].clone()
    native().tp_decode(symm.heap, [x.data_ptr()], [layer.weight.data_ptr()], layer.residual_in.data_ptr(), layer.residual_out.data_ptr(),
                       layer.out.data_ptr(), layer.gamma.data_ptr(), tokens, hidden, k, layer.eps, False, 0,
                       torch.cuda.current_stream().cuda_stream, 0, 0)
    torch.cuda.synchronize()
    symm.check()
    assert torch.equal(h, layer.residual_out[:tokens])
    symm.destroy()


@pytest.mark.parametrize("tokens", [1, 8])
def test_chained_decode_layers_wait_for_one_another(tokens):
    """Decode launches overlap the one before them and prefetch their operands under it: activations that the layer before
    writes, a residual that it writes, and weights that a copy right before writes."""
    from mscclpp_b200 import SymmetricMemory
    from mscclpp_b200.parallel.tp_layer import RowParallelLinearNorm

    hidden = 2048
    symm = SymmetricMemory.emulated(1, nbytes=64 << 20, timeout_ms=3000)
    layers = [RowParallelLinearNorm(symm, out_features=hidden, k_shard=hidden, max_tokens=tokens, seed=i) for i in range(3)]
    weights = [layer.weight.clone() for layer in layers]
    g = torch.Generator(device="cuda").manual_seed(tokens)
    x, first = (torch.randn((tokens, hidden), generator=g, device="cuda").to(torch.bfloat16) for _ in range(2))
    layers[0].residual_in.copy_(first)
    layers[1].residual_in, layers[2].residual_in = layers[0].residual_out, layers[1].residual_out
    chain = [lambda: layers[0].weight.copy_(weights[1]), lambda: layers[0].forward_decode(x), lambda: layers[0].weight.copy_(weights[0]),
             lambda: layers[0].forward_decode(x), lambda: layers[1].forward_decode(layers[0].out), lambda: layers[2].forward_decode(layers[1].out)]
    _same_without_waiting(chain, [t for layer in layers for t in (layer.out, layer.residual_out)])
    symm.check()
    symm.destroy()
