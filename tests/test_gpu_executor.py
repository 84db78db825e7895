"""GPU plan interpreter against the numpy plan interpreter on identical plans and inputs.
All ranks of a plan are emulated on one GPU in one cooperative launch."""
import json
import os

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

NP2TORCH = {np.float32: torch.float32, np.float16: torch.float16, np.int32: torch.int32}


def _run_both(plan_json, world, in_elems, out_elems, np_dtype, inplace, launches=2, packet_type="LL16"):
    from mscclpp_b200 import SymmetricMemory, native
    from mscclpp_b200.language.interpreter import PlanInterpreter

    n = native()
    symm = SymmetricMemory.emulated(world, nbytes=128 << 20, timeout_ms=3000)
    tdtype = NP2TORCH[np_dtype]
    t_in = symm.tensor((in_elems,), tdtype)
    t_out = t_in if inplace else symm.tensor((out_elems,), tdtype)
    executor = n.Executor(symm.heap)
    plans = [n.ExecutionPlan.from_string(plan_json, r) for r in range(world)]
    interp = PlanInterpreter(plan_json)
    dt = {np.float32: n.DataType.float32, np.float16: n.DataType.float16, np.int32: n.DataType.int32}[np_dtype]
    for launch in range(launches):
        rng = np.random.default_rng(100 + launch)
        if np_dtype == np.int32:
            ins = [rng.integers(-1000, 1000, size=in_elems).astype(np_dtype) for _ in range(world)]
        else:
            ins = [rng.uniform(-1, 1, size=in_elems).astype(np_dtype) for _ in range(world)]
        outs = [np.zeros(out_elems, dtype=np_dtype) for _ in range(world)]
        for r in range(world):
            symm.rank_view(t_in, r).copy_(torch.from_numpy(ins[r]))
            if not inplace:
                symm.rank_view(t_out, r).zero_()
        expect = interp.run([a.copy() for a in ins], None if inplace else outs)
        executor.execute(0, t_in.data_ptr(), t_out.data_ptr(), in_elems * ins[0].itemsize, out_elems * ins[0].itemsize, dt,
                         plans[0], torch.cuda.current_stream().cuda_stream, getattr(n.PacketType, packet_type))
        torch.cuda.synchronize()
        symm.check()
        for r in range(world):
            got = symm.rank_view(t_out, r).cpu().numpy()
            if np_dtype == np.int32:
                np.testing.assert_array_equal(got, expect[r])
            else:
                np.testing.assert_allclose(got.astype(np.float32), expect[r].astype(np.float32), rtol=2e-3, atol=2e-3,
                                           err_msg=f"rank {r} of {world}, launch {launch}, {in_elems} elements, packets {packet_type}")
    team = executor.last_team()
    executor.reset()
    symm.destroy()
    return team


@pytest.mark.parametrize("world", [2, 4, 8])
@pytest.mark.parametrize("algo", ["allreduce_allpairs", "allreduce_allpairs_packet", "allreduce_nvls"])
@pytest.mark.parametrize("instances", [1, 2])
def test_allreduce_plans(world, algo, instances):
    from mscclpp_b200.default_algos import single_node

    plan = single_node.build(algo, world, instances=instances).to_json()
    elems = 4 * world * instances * 64
    _run_both(plan, world, elems, elems, np.float32, inplace=True)
    _run_both(plan, world, elems, elems, np.float16, inplace=True)


@pytest.mark.parametrize("world", [2, 8])
@pytest.mark.parametrize("packet_type", ["LL8", "LL16"])
def test_packet_plans_with_both_packet_formats(world, packet_type):
    """The same LL plan through 8-byte and 16-byte packets, a small and a larger message. (Sizes divide evenly into the
    plan's chunks: with a remainder the plan format maps unequal input chunks onto scratch chunks of other sizes, in
    the reference as well, and neighbouring ranges then overlap.)"""
    from mscclpp_b200.default_algos import single_node

    plan = single_node.build("allreduce_allpairs_packet", world).to_json()
    for elems in (4 * world * 16, 4 * world * 1024):
        _run_both(plan, world, elems, elems, np.float32, inplace=True, packet_type=packet_type)


@pytest.mark.parametrize("nodes,gpus", [(2, 2), (2, 4)])
def test_port_channel_plans_go_through_the_host_proxy(nodes, gpus):
    """The hierarchical multi-node plans talk to the GPUs of other nodes through port channels: the interpreter kernel
    queues requests in the executor's FIFO and the executor's proxy thread moves the packets with the copy engines.
    Here the 'nodes' are groups of emulated ranks on one GPU, which exercises exactly that path."""
    from mscclpp_b200.default_algos import allreduce_multi_nodes, reducescatter_multi_nodes
    from mscclpp_b200.language.collectives import AllReduce, ReduceScatter
    from mscclpp_b200.language.utils import AlgoSpec

    w = nodes * gpus

    def spec(name, coll):
        return AlgoSpec(name=name, collective=coll, nranks_per_node=gpus, world_size=w, in_place=True, instances=1, protocol="LL",
                        auto_sync=False, num_threads_per_block=1024, reuse_resources=True, use_double_scratch_buffer=True)

    plan = allreduce_multi_nodes(spec("ar_mn_gpu", AllReduce(w, 1, True))).to_json()
    assert '"port"' in plan
    elems = w * nodes * 64
    _run_both(plan, w, elems, elems, np.float32, inplace=True, launches=3)
    plan = reducescatter_multi_nodes(spec("rs_mn_gpu", ReduceScatter(w, 1, True))).to_json()
    assert '"port"' in plan


def test_plan_with_more_blocks_than_the_gpu_can_hold_is_refused():
    """Thread blocks of a plan wait on one another, so all of them (times the emulated ranks) must be resident at once;
    a launch that cannot be is refused with a message that names the plan and the numbers, before anything runs."""
    from mscclpp_b200 import SymmetricMemory, native
    from mscclpp_b200.default_algos import single_node

    n = native()
    world = 8
    plan_json = single_node.build("allreduce_allpairs", world, instances=32).to_json()  # 32 blocks of 1024 threads per rank
    blocks = max(len(g["threadblocks"]) for g in json.loads(plan_json)["gpus"])
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    if blocks * world <= sms:
        pytest.skip("this plan fits the GPU even with all ranks emulated")
    symm = SymmetricMemory.emulated(world, nbytes=128 << 20, timeout_ms=1000)
    elems = 4 * world * 32 * 64
    t = symm.tensor((elems,), torch.float32, zero=True)
    ex = n.Executor(symm.heap)
    with pytest.raises(Exception, match="resident at the same time"):
        ex.execute(0, t.data_ptr(), t.data_ptr(), elems * 4, elems * 4, n.DataType.float32, n.ExecutionPlan.from_string(plan_json, 0), 0)
    ex.reset()
    symm.destroy()


@pytest.mark.parametrize("world", [2, 8])
def test_allgather_reducescatter_alltoall_plans(world):
    from mscclpp_b200.default_algos import single_node

    per = 256
    _run_both(single_node.build("reducescatter_allpairs", world).to_json(), world, world * per, per, np.float32, inplace=False)
    _run_both(single_node.build("alltoall_allpairs", world).to_json(), world, world * per, world * per, np.int32, inplace=False)
    _run_both(single_node.build("allgather_allpairs", world, in_place=False).to_json(), world, per, world * per, np.int32, inplace=False)


def test_reduction_operands_that_begin_off_a_word_are_refused():
    """Refused before anything is launched: a heap buffer that begins four bytes into a word, chunks that do (buffer_alignment 4), a pipeline unit that is no
    multiple of 16. Chunks of less than a word still run."""
    from mscclpp_b200 import SymmetricMemory, native
    from mscclpp_b200.default_algos.single_node import make_spec
    from mscclpp_b200.language.collectives import AllReduce
    from mscclpp_b200.language.loop import LoopIterationContext
    from mscclpp_b200.language.program import CollectiveProgram
    from mscclpp_b200.language.rank import Rank

    def plan(name, alignment, unit=0):
        prog = CollectiveProgram.from_spec(make_spec(name, AllReduce(2, 2, True), 2, buffer_alignment=alignment))
        with prog:
            loop = LoopIterationContext(unit=unit, num_chunks=1) if unit else None
            if loop:
                loop.__enter__()
            for r in range(2):
                inp = Rank(r).get_input_buffer()
                Rank(r).reduce(inp[1:2], [inp[2:3]], tb=0)
            if loop:
                loop.__exit__(None, None, None)
        return n.ExecutionPlan.from_string(prog.to_json(), 0)

    n = native()
    symm = SymmetricMemory.emulated(2, nbytes=64 << 20, timeout_ms=1000)
    t = symm.tensor((1024,), torch.float32, zero=True)
    ex = n.Executor(symm.heap)
    run = lambda p, offset, nbytes: ex.execute(0, t.data_ptr() + offset, t.data_ptr() + offset, nbytes, nbytes, n.DataType.float32, p, 0)
    for p, offset, nbytes in ((plan("aligned", 16), 4, 1024), (plan("words", 4), 0, 1024 + 16), (plan("units", 16, unit=24), 0, 1024)):
        with pytest.raises(Exception, match="multiple of 16 bytes"):
            run(p, offset, nbytes)
    for r in range(2):
        symm.rank_view(t, r).copy_(torch.arange(1024) + 1024.0 * r)
    run(plan("words", 4), 0, 48)  # four chunks of three elements
    run(plan("units_of_words", 16, unit=32), 0, 1024)
    torch.cuda.synchronize()
    symm.check()
    for r in range(2):
        want = torch.arange(1024) + 1024.0 * r
        want[3:6] += want[6:9].clone()
        want[64:128] += want[128:192].clone()
        assert torch.equal(symm.rank_view(t, r).cpu(), want)
    ex.reset()
    symm.destroy()


def test_malformed_plan_is_rejected():
    from mscclpp_b200 import native
    from mscclpp_b200.default_algos import single_node

    n = native()
    plan = json.loads(single_node.build("allreduce_allpairs", 2).to_json())
    plan["gpus"][0]["threadblocks"][0]["ops"].append({"name": "frobnicate"})
    from mscclpp_b200 import SymmetricMemory

    symm = SymmetricMemory.emulated(2, nbytes=64 << 20, timeout_ms=1000)
    t = symm.tensor((1024,), torch.float32, zero=True)
    ex = n.Executor(symm.heap)
    with pytest.raises(Exception):
        ex.execute(0, t.data_ptr(), t.data_ptr(), 4096, 4096, n.DataType.float32, n.ExecutionPlan.from_string(json.dumps(plan), 0), 0)
    ex.reset()
    symm.destroy()


def test_tracer_records_executor_operations(tmp_path):
    """With the tracer on, every thread block of a plan leaves ENTRY/EXIT pairs that convert to a Chrome trace."""
    from mscclpp_b200 import SymmetricMemory, native
    from mscclpp_b200.default_algos import single_node
    from mscclpp_b200.utils.npkit_trace import convert_npkit_dump_to_trace

    n = native()
    world = 2
    plan_json = single_node.build("allreduce_allpairs", world).to_json()
    symm = SymmetricMemory.emulated(world, nbytes=64 << 20, timeout_ms=3000)
    t = symm.tensor((4096,), torch.float32)
    for r in range(world):
        symm.rank_view(t, r).fill_(r + 1.0)
    n.npkit.init(0)
    try:
        assert n.npkit.enabled()
        executor = n.Executor(symm.heap)
        plan = n.ExecutionPlan.from_string(plan_json, 0)
        executor.execute(0, t.data_ptr(), t.data_ptr(), t.numel() * 4, t.numel() * 4, n.DataType.float32, plan,
                         torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        symm.check()
        assert bool((symm.rank_view(t, 1) == 3.0).all().item())
        n.npkit.dump(str(tmp_path))
    finally:
        n.npkit.shutdown()
    assert not n.npkit.enabled()
    files = sorted(os.listdir(tmp_path))
    assert any(f.startswith("gpu_events_rank_0_buf_") for f in files) and "gpu_time_sync_rank_0" in files
    trace = json.loads(open(convert_npkit_dump_to_trace(str(tmp_path), str(tmp_path / "out"))).read())["traceEvents"]
    slices = [e for e in trace if e["ph"] == "X"]
    assert slices and all(e["dur"] >= 0 for e in slices)
    assert {"EXECUTOR_OP_SIGNAL", "EXECUTOR_OP_WAIT"} & {e["name"] for e in slices} or any("EXECUTOR_OP" in e["name"] for e in slices)
    executor.reset()
    symm.destroy()


def test_tracer_names_thread_blocks_that_several_ctas_run(tmp_path):
    """Two thread blocks on each of two ranks, run by four CTAs each or more: a buffer per thread block of the plan, each with all of its operations,
    one after the other."""
    from mscclpp_b200 import SymmetricMemory, native
    from mscclpp_b200.utils.npkit_trace import convert_npkit_dump_to_trace

    n = native()
    plan_json = _plan_of_large_operations("barrier")
    names = [[op["name"] for op in tb["ops"]] for gpu in json.loads(plan_json)["gpus"] for tb in gpu["threadblocks"]]
    assert len(names) == 4
    symm = SymmetricMemory.emulated(2, nbytes=64 << 20, timeout_ms=3000)
    t = symm.tensor((1 << 19,), torch.float32, zero=True)
    executor = n.Executor(symm.heap)
    plan = n.ExecutionPlan.from_string(plan_json, 0)
    n.npkit.init(0)
    try:
        executor.execute(0, t.data_ptr(), t.data_ptr(), t.numel() * 4, t.numel() * 4, n.DataType.float32, plan, torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        symm.check()
        assert executor.last_team() >= 4
        n.npkit.dump(str(tmp_path))
    finally:
        n.npkit.shutdown()
    prefix = "gpu_events_rank_0_buf_"
    written = {int(f[len(prefix):]) for f in os.listdir(tmp_path) if f.startswith(prefix) and os.path.getsize(tmp_path / f) > 0}
    assert written == {0, 1, 2, 3}
    for b in range(4):
        events = np.fromfile(tmp_path / f"{prefix}{b}", dtype=np.uint64).reshape(-1, 2)
        assert len(events) == 2 * len(names[b]) and (np.diff(events[:, 1].astype(np.int64)) >= 0).all()
    trace = json.loads(open(convert_npkit_dump_to_trace(str(tmp_path), str(tmp_path / "out"))).read())["traceEvents"]
    assert sum(e["ph"] == "X" for e in trace) == sum(len(ops) for ops in names)
    executor.reset()
    symm.destroy()


def test_guard_bands_around_executor_buffers(monkeypatch):
    """With MSCCLPP_EXECUTOR_CANARY=1 the executor's scratch sits between two bands of 0xA5 on every rank. A correct plan
    leaves them alone (a packet plan writes its scratch from every peer, up to the last byte); a byte written just past
    the scratch is found by check_canaries() and again reported by reset(), which still returns the buffers."""
    from mscclpp_b200 import SymmetricMemory, native
    from mscclpp_b200._core.symm import tensor_from_pointer
    from mscclpp_b200.default_algos import single_node

    monkeypatch.setenv("MSCCLPP_EXECUTOR_CANARY", "1")
    n = native()
    world = 4
    symm = SymmetricMemory.emulated(world, nbytes=64 << 20, timeout_ms=3000)
    elems = 4 * world * 256
    t = symm.tensor((elems,), torch.float32)
    for r in range(world):
        symm.rank_view(t, r).fill_(r + 1.0)
    executor = n.Executor(symm.heap)
    assert executor.check_canaries() == 0  # nothing allocated yet
    plan = n.ExecutionPlan.from_string(single_node.build("allreduce_allpairs_packet", world).to_json(), 0)
    for _ in range(3):
        executor.execute(0, t.data_ptr(), t.data_ptr(), elems * 4, elems * 4, n.DataType.float32, plan,
                         torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    symm.check()
    regions = executor.canary_regions()
    assert len(regions) == 2 * world and all(nbytes == 256 for _, _, nbytes in regions)
    assert executor.check_canaries() == len(regions)

    label, address, nbytes = next(r for r in regions if "/scratch/back" in r[0] and r[0].endswith("rank 2"))
    band = tensor_from_pointer(address, (nbytes,), torch.uint8, t.device)
    assert bool((band == 0xA5).all().item())
    band[3] = 0
    torch.cuda.synchronize()
    with pytest.raises(Exception, match="guard band .*scratch/back/rank 2.*first at byte 3"):
        executor.check_canaries()
    free_before = symm.heap.bytes_free() if hasattr(symm.heap, "bytes_free") else None
    with pytest.raises(Exception, match="guard band"):
        executor.reset()
    if free_before is not None:
        assert symm.heap.bytes_free() > free_before  # the buffers went back to the heap all the same
    assert executor.canary_regions() == []
    symm.destroy()


@pytest.mark.parametrize("world", [2, 3, 4, 5, 6, 7, 8])
def test_reductions_of_every_number_of_sources(world):
    """The interpreter requests a reduction's sources in groups of four, two and one: every remainder of that split."""
    from mscclpp_b200.default_algos import single_node

    for per in (8, 1040):
        _run_both(single_node.build("reducescatter_allpairs", world).to_json(), world, world * per, per, np.float16, inplace=False)
        _run_both(single_node.build("reducescatter_allpairs", world).to_json(), world, world * per, per, np.int32, inplace=False)


# elements of a chunk, fp16; the words do not divide by their threads. team: the CTAs that run each thread block of the reduction
@pytest.mark.parametrize("world,instances,per,team", [(2, 1, 32768 + 8, 1), (2, 1, 65536 + 24, 1), (2, 1, 131072 + 1032, 8), (2, 1, 262144 + 1032, 8),
                                                      (3, 2, 262144 + 16, 8), (4, 5, 5 * 131072 + 80, 4), (8, 1, 65536 + 16, 8), (8, 8, 65536 + 64, 1),
                                                      (8, 8, 524288 + 64, 2)])
def test_thread_blocks_of_several_ctas(world, instances, per, team):
    from mscclpp_b200.default_algos import single_node

    build = lambda name: single_node.build(name, world, instances=instances, in_place=False).to_json()
    teams = [_run_both(build("reducescatter_allpairs"), world, world * per, per, np.float16, inplace=False),
             _run_both(build("alltoall_allpairs"), world, world * per, world * per, np.float16, inplace=False),
             _run_both(build("allgather_allpairs"), world, per, world * per, np.float16, inplace=False),
             _run_both(single_node.build("allreduce_nvls", world, instances=instances).to_json(), world, world * per, world * per, np.float16, inplace=True)]
    assert teams[0] == team


def _plan_of_large_operations(kind):
    """Two ranks: what a thread block does once (barrier, semaphore, request to the host proxy) between the operations that its CTAs
    share, a pipeline, and sizes that leave a part of a word."""
    from mscclpp_b200.default_algos.single_node import make_spec
    from mscclpp_b200.language.channel import MemoryChannel, PortChannel
    from mscclpp_b200.language.collectives import AllReduce
    from mscclpp_b200.language.loop import LoopIterationContext
    from mscclpp_b200.language.program import CollectiveProgram
    from mscclpp_b200.language.rank import Buffer, Rank, Semaphore

    prog = CollectiveProgram.from_spec(make_spec(f"large_{kind}", AllReduce(2, 2, True), 2, buffer_alignment=4 if kind == "tail" else 16))
    with prog:
        scratch = [Buffer(r, 2) for r in range(2)]
        inputs = [Rank(r).get_input_buffer() for r in range(2)]
        if kind in ("port", "tail"):
            chan = [(PortChannel if kind == "port" else MemoryChannel)(1 - r, r) for r in range(2)]
            for r in range(2):
                chan[r].put(scratch[1 - r][0:1], inputs[r][0:1], tb=0)
                chan[r].signal(tb=0)
            for r in range(2):
                chan[r].wait(tb=0)
                Rank(r).reduce(scratch[r][0:1], [inputs[r][0:1]], tb=0)
            for r in range(2):
                Rank(r).copy(inputs[r][0:1], scratch[r][0:1], tb=0)
            return prog.to_json()
        for r in range(2):
            rank, inp, s = Rank(r), inputs[r], scratch[r]
            if kind == "barrier":
                for tb in range(2):
                    rank.copy(s[tb:tb + 1], inp[tb:tb + 1], tb=tb)
                rank.barrier([0, 1])
                for tb in range(2):
                    rank.reduce(inp[2 + tb:3 + tb], [s[1 - tb:2 - tb]], tb=tb)
                rank.barrier([0, 1])
                for tb in range(2):
                    rank.copy(inp[tb:tb + 1], inp[3 - tb:4 - tb], tb=tb)
            else:
                sem = Semaphore(r, 0)
                loop = LoopIterationContext(unit=512 << 10, num_chunks=1) if kind == "pipeline" else None
                if loop is not None:
                    loop.__enter__()
                rank.copy(s[0:1], inp[0:1], tb=0)
                sem.release(tb=0)
                sem.acquire(tb=1)
                rank.reduce(inp[2:3], [s[0:1]], tb=1)
                if loop is not None:
                    loop.__exit__(None, None, None)
    return prog.to_json()


@pytest.mark.parametrize("kind,per", [("barrier", (512 << 10) + 48), ("semaphore", (512 << 10) + 48), ("pipeline", (1536 << 10) + 80), ("port", (512 << 10) + 48),
                                      ("tail", (512 << 10) + 4)])
def test_what_a_thread_block_of_several_ctas_does_once(kind, per):
    assert _run_both(_plan_of_large_operations(kind), 2, per, per, np.int32, inplace=True, launches=3) == 8  # (four chunks of `per` bytes, int32)


@pytest.mark.parametrize("setting,team", [("1", 1), ("2", 2), ("", 8)])
def test_how_many_ctas_share_a_thread_block_can_be_limited(monkeypatch, setting, team):
    from mscclpp_b200.default_algos import single_node

    monkeypatch.setenv("MSCCLPP_EXECUTOR_TEAM", setting)
    per = 262144 + 1032
    assert _run_both(single_node.build("reducescatter_allpairs", 2, in_place=False).to_json(), 2, 2 * per, per, np.float16, inplace=False) == team


def test_a_wait_that_runs_out_ends_every_cta_of_a_thread_block():
    """The signals that the first wait is for are left out of the plan. The error is reported, nobody has reduced anything, and the
    complete plan works afterwards."""
    from mscclpp_b200 import SymmetricMemory, native
    from mscclpp_b200.default_algos import single_node

    n = native()
    plan = json.loads(single_node.build("reducescatter_allpairs", 2, in_place=False).to_json())
    complete = n.ExecutionPlan.from_string(json.dumps(plan), 0)
    plan["name"] += "_without_signals"
    for gpu in plan["gpus"]:
        for tb in gpu["threadblocks"]:
            assert tb["ops"][0]["name"] == "rlxsignal"
            tb["ops"] = tb["ops"][1:]
    lacking = n.ExecutionPlan.from_string(json.dumps(plan), 0)
    symm = SymmetricMemory.emulated(2, nbytes=64 << 20, timeout_ms=300)
    per = 1 << 18  # two sources of 1 MB: eight CTAs
    t_in, t_out = symm.tensor((2 * per,), torch.float32), symm.tensor((per,), torch.float32)
    ins = [torch.arange(2 * per, device="cuda", dtype=torch.float32) * (r + 1) for r in range(2)]
    for r in range(2):
        symm.rank_view(t_in, r).copy_(ins[r])
        symm.rank_view(t_out, r).fill_(-1.0)
    executor = n.Executor(symm.heap)

    def run(loaded):
        executor.execute(0, t_in.data_ptr(), t_out.data_ptr(), 8 * per, 4 * per, n.DataType.float32, loaded, torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()

    run(lacking)
    assert executor.last_team() == 8
    with pytest.raises(Exception, match="gave up"):
        symm.check()
    for r in range(2):
        assert bool((symm.rank_view(t_out, r) == -1.0).all())
    symm.heap.reset_status()
    run(complete)
    symm.check()
    for r in range(2):
        assert torch.equal(symm.rank_view(t_out, r), (ins[0] + ins[1])[r * per:(r + 1) * per])
    executor.reset()
    symm.destroy()


def _packets_then_reduction(kind):
    """Two ranks, one thread block each: a packet operation of fewer packets than threads, then a reduction of other
    chunks, which the DSL puts directly behind it (their chunks do not overlap)."""
    from mscclpp_b200.default_algos.single_node import make_spec
    from mscclpp_b200.language.channel import MemoryChannel
    from mscclpp_b200.language.collectives import AllReduce
    from mscclpp_b200.language.program import CollectiveProgram
    from mscclpp_b200.language.rank import Buffer, Rank

    prog = CollectiveProgram.from_spec(make_spec(f"packets_then_reduction_{kind}", AllReduce(2, 2, True), 2, protocol="LL"))
    with prog:
        scratch = [Buffer(r, 4) for r in range(2)]
        chan = [MemoryChannel(1 - r, r) for r in range(2)]
        for r in range(2):
            chan[r].put_packets(scratch[1 - r][0:1], Rank(r).get_input_buffer()[0:1], tb=0)
        for r in range(2):
            inp = Rank(r).get_input_buffer()
            if kind == "unpack":
                Rank(r).unpack_packets(inp[1:2], scratch[r][0:1], tb=0)
            elif kind == "reduce":
                Rank(r).reduce(inp[1:2], [scratch[r][0:1]], tb=0, packet=True)
            else:
                chan[r].read_put_packets(scratch[1 - r][1:2], scratch[r][0:1], tb=0)
            Rank(r).reduce(inp[2:3], [inp[3:4]], tb=0)
    return json.loads(prog.to_json())


@pytest.mark.parametrize("kind", ["unpack", "reduce", "forward"])
@pytest.mark.parametrize("packet_type", ["LL8", "LL16"])
def test_packets_that_never_come_end_the_block_before_a_reduction(monkeypatch, kind, packet_type):
    """The peers' puts are left out of the plan, so the wait for packets runs out in the threads that have one. The error is
    reported, the reduction behind it has run in no thread (its destination and everything else are as before, the guard bands
    intact), and the complete plan works afterwards."""
    from mscclpp_b200 import SymmetricMemory, native

    monkeypatch.setenv("MSCCLPP_EXECUTOR_CANARY", "1")
    n = native()
    plan = _packets_then_reduction(kind)
    complete = n.ExecutionPlan.from_string(json.dumps(plan), 0)
    plan["name"] += "_without_puts"  # (an executor knows a plan by its name)
    for gpu in plan["gpus"]:
        for tb in gpu["threadblocks"]:
            names = [op["name"] for op in tb["ops"]]
            assert names[0] == "ppkt" and names[-1] == "re" and len(names) == 3
            tb["ops"] = tb["ops"][1:]
    symm = SymmetricMemory.emulated(2, nbytes=64 << 20, timeout_ms=300)
    per = 128  # elements of a chunk: at most 128 packets, 1024 threads
    t = symm.tensor((4 * per,), torch.float32)
    before = [torch.arange(4 * per, device="cuda", dtype=torch.float32) + 1000 * r for r in range(2)]
    executor = n.Executor(symm.heap)

    def run(loaded):
        for r in range(2):
            symm.rank_view(t, r).copy_(before[r])
        executor.execute(0, t.data_ptr(), t.data_ptr(), 16 * per, 16 * per, n.DataType.float32, loaded,
                         torch.cuda.current_stream().cuda_stream, getattr(n.PacketType, packet_type))
        torch.cuda.synchronize()

    lacking = n.ExecutionPlan.from_string(json.dumps(plan), 0)
    run(lacking)
    with pytest.raises(Exception, match="gave up"):
        symm.check()
    assert executor.check_canaries() > 0
    for r in range(2):
        assert torch.equal(symm.rank_view(t, r), before[r])
    symm.heap.reset_status()
    run(complete)
    symm.check()
    for r in range(2):
        expect = before[r].view(4, per).clone()
        if kind != "forward":
            expect[1] = before[1 - r][:per] + (expect[1] if kind == "reduce" else 0)
        expect[2] += expect[3]
        assert torch.equal(symm.rank_view(t, r).view(4, per), expect)
    executor.reset()
    symm.destroy()
