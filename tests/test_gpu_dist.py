"""Expert-parallel path on two GPUs: every rank routes all tokens, computes its half of the
256 experts, NCCL sums the bf16 partial outputs.  Skipped on boxes with fewer than two GPUs
(the CPU form of the same plan runs in tests/test_dist_cpu.py over gloo)."""
import os
import socket

import pytest
import torch
import torch.multiprocessing as mp

pytestmark = pytest.mark.gpu


def _free_port():
    s = socket.socket()
    s.bind(("127.0.0.1", 0))
    p = s.getsockname()[1]
    s.close()
    return p


def _worker(rank, world, port, T, q):
    import sys
    from pathlib import Path
    root = Path(__file__).resolve().parent.parent
    sys.path.insert(0, str(root))
    sys.path.insert(0, str(root / "tests"))
    import torch.distributed as dist
    import __graft_entry__ as entry
    entry.load_package()
    from fp8_moe_dev_b200 import gen
    from fp8_moe_dev_b200.dist import ShardedMoe, token_range
    os.environ["MASTER_ADDR"] = "127.0.0.1"
    os.environ["MASTER_PORT"] = str(port)
    os.environ["NCCL_NVLS_ENABLE"] = "0"
    torch.cuda.set_device(rank)
    dist.init_process_group("nccl", rank=rank, world_size=world, device_id=torch.device("cuda", rank))
    try:
        logits, bias = gen.make_routing(T, seed=11)
        hidden, hscale = gen.make_hidden(T, seed=12)
        dev = [x.cuda() for x in (logits, bias, hidden, hscale)]
        moe = ShardedMoe(T)
        E = moe.num_local_experts
        w = gen.make_shard(moe.local_expert_offset, E, device="cuda", out_device="cuda")
        out = torch.empty(T, 7168, dtype=torch.bfloat16, device="cuda")
        partial = torch.empty_like(out)
        moe.layer.run(*dev, *w, moe.local_expert_offset, 2.5, partial)
        moe.layer.check()
        full = moe.run(*dev, *w, 2.5, out, mode="all_reduce").clone()
        moe.layer.check()
        # the same sum done by hand: gather the partial outputs and add them in rank order
        parts = [torch.empty_like(partial) for _ in range(world)]
        dist.all_gather(parts, partial)
        want = parts[0].clone()
        for p in parts[1:]:
            want += p
        ok_sum = torch.equal(full, want)
        scat = moe.run(*dev, *w, 2.5, out, mode="reduce_scatter")
        lo, hi = token_range(rank, world, T)
        ok_scatter = torch.equal(scat[:hi - lo], want[lo:hi])
        nonzero = bool(full.float().abs().sum() > 0)
        # combine + reduce-scatter fused into one step over peer memory, three calls in a row
        # (both parities of the receive buffer and its reuse); with two ranks the fp32 sum of
        # two bf16 rows rounded once equals the bf16 sum, so the results must be identical
        ok_fused = True
        for _ in range(3):
            torch.cuda.synchronize()
            dist.barrier()
            got = moe.run(*dev, *w, 2.5, out, mode="fused")
            moe.layer.check()
            ok_fused = ok_fused and got.shape[0] == (T + world - 1) // world and torch.equal(got[:hi - lo], want[lo:hi])
        # host-resident inputs: every rank copies its token slice, NVLink all-gathers the rest
        if T % world == 0:
            pin = [x.pin_memory() for x in (logits, hidden, hscale)]
            host_out = torch.zeros(T, 7168, dtype=torch.bfloat16).pin_memory()
            for mode in ("fused", "reduce_scatter"):
                host_out.zero_()
                dist.barrier()
                moe.run_host(pin[0], dev[1], pin[1], pin[2], *w, 2.5, host_out, mode=mode)
                moe.layer.check()
                ok_fused = ok_fused and torch.equal(host_out[lo:hi], want[lo:hi].cpu())
            # the same kept two deep in flight over two output buffers
            outs = [torch.zeros(T, 7168, dtype=torch.bfloat16).pin_memory() for _ in range(2)]
            tickets = []
            for i in range(4):
                if i >= 2:
                    moe.host_wait(tickets[i - 2])
                    ok_fused = ok_fused and torch.equal(outs[i % 2][lo:hi], want[lo:hi].cpu())
                    outs[i % 2].zero_()
                tickets.append(moe.run_host_async(pin[0], dev[1], pin[1], pin[2], *w, 2.5, outs[i % 2], mode="fused"))
            for i in (2, 3):
                moe.host_wait(tickets[i])
                ok_fused = ok_fused and torch.equal(outs[i % 2][lo:hi], want[lo:hi].cpu())
            moe.layer.check()
            # the same with the inputs replicated by NCCL all-gathers instead of peer copies
            moe_n = ShardedMoe(T)
            moe_n.copy_engine_gather = False
            host_out.zero_()
            dist.barrier()
            moe_n.run_host(pin[0], dev[1], pin[1], pin[2], *w, 2.5, host_out, mode="fused")
            moe_n.layer.check()
            ok_fused = ok_fused and torch.equal(host_out[lo:hi], want[lo:hi].cpu())
        # strided expert placement: other owners, same pairs; the summed output agrees up to the
        # rounding of the partial outputs, and the ranks' row counts add up to the same total
        rows_c = torch.tensor([int(moe.layer.read("pair_count", T).sum())], device="cuda")
        moe_s = ShardedMoe(T, placement="strided")
        ws = gen.make_experts(moe_s.expert_ids, device="cuda", out_device="cuda")
        got_s = moe_s.run(*dev, *ws, 2.5, out, mode="fused")
        moe_s.layer.check()
        rows_s = torch.tensor([int(moe_s.layer.read("pair_count", T).sum())], device="cuda")
        dist.all_reduce(rows_c)
        dist.all_reduce(rows_s)
        a, b = got_s[:hi - lo].float(), want[lo:hi].float()
        rel = float((a - b).norm() / (b.norm() + 1e-30))
        ok_fused = ok_fused and int(rows_c) == int(rows_s) and rel < 1e-2
        # experts placed by measured load
        import fp8_moe_dev_b200 as pkg2
        loads = pkg2.expert_loads(dev[0], dev[1], 2.5)
        moe_b = ShardedMoe(T, placement="balanced", loads=loads)
        wb = gen.make_experts(moe_b.expert_ids, device="cuda", out_device="cuda")
        got_b = moe_b.run(*dev, *wb, 2.5, out, mode="fused")
        moe_b.layer.check()
        rows_b = torch.tensor([int(moe_b.layer.read("pair_count", T).sum())], device="cuda")
        mine_b = int(rows_b)
        dist.all_reduce(rows_b)
        a = got_b[:hi - lo].float()
        rel = float((a - b).norm() / (b.norm() + 1e-30))
        ok_fused = ok_fused and int(rows_b) == int(rows_c) and rel < 1e-2 and abs(mine_b - int(rows_b) / world) <= 0.06 * int(rows_b) + 8
        q.put((rank, ok_sum, ok_scatter and ok_fused, nonzero))
    finally:
        dist.destroy_process_group()


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs two GPUs")
@pytest.mark.parametrize("T", [96, 33])
def test_two_gpu_expert_parallel_sum(T):
    world = 2
    ctx = mp.get_context("spawn")
    q = ctx.Queue()
    port = _free_port()
    procs = [ctx.Process(target=_worker, args=(r, world, port, T, q)) for r in range(world)]
    for p in procs:
        p.start()
    for p in procs:
        p.join(600)
        assert p.exitcode == 0
    res = sorted(q.get(timeout=10) for _ in range(world))
    assert res == [(0, True, True, True), (1, True, True, True)], res


def _worker_varying_t(rank, world, port, q):
    """One ShardedMoe sized for 96 tokens, fused calls with T = 96, 33, 96, 40, 96, 12 and no barrier or
    host synchronisation between them; the ranks are skewed against each other by device-side sleeps, so
    that one rank's push of the next epoch overlaps the other's reduce of the current one."""
    import sys
    from pathlib import Path
    root = Path(__file__).resolve().parent.parent
    sys.path.insert(0, str(root))
    sys.path.insert(0, str(root / "tests"))
    import torch.distributed as dist
    import __graft_entry__ as entry
    entry.load_package()
    from fp8_moe_dev_b200 import gen
    from fp8_moe_dev_b200.dist import ShardedMoe, token_range
    os.environ["MASTER_ADDR"] = "127.0.0.1"
    os.environ["MASTER_PORT"] = str(port)
    os.environ["NCCL_NVLS_ENABLE"] = "0"
    torch.cuda.set_device(rank)
    dist.init_process_group("nccl", rank=rank, world_size=world, device_id=torch.device("cuda", rank))
    try:
        Tmax = 96
        seq = [96, 33, 96, 40, 96, 12]   # all above 8 tokens: both forms then run the same staged chain
        moe = ShardedMoe(Tmax)
        w = gen.make_shard(moe.local_expert_offset, moe.num_local_experts, device="cuda", out_device="cuda")
        cases, want = {}, {}
        for T in sorted(set(seq)):
            logits, bias = gen.make_routing(T, seed=100 + T)
            hidden, hscale = gen.make_hidden(T, seed=200 + T)
            cases[T] = [x.cuda() for x in (logits, bias, hidden, hscale)]
            out = torch.empty(T, 7168, dtype=torch.bfloat16, device="cuda")
            lo, hi = token_range(rank, world, T)
            want[T] = moe.run(*cases[T], *w, 2.5, out, mode="reduce_scatter")[:hi - lo].clone()
        torch.cuda.synchronize()
        dist.barrier()
        got = []
        for i, T in enumerate(seq):
            if (i + rank) % 2 == 0:
                torch.cuda._sleep(3_000_000)      # about 2 ms: lets the other rank run ahead
            scat = torch.empty((T + world - 1) // world, 7168, dtype=torch.bfloat16, device="cuda")
            moe.run_fused(*cases[T], *w, 2.5, scatter_out=scat)
            got.append(scat)
        moe.layer.check()
        ok = True
        for T, g in zip(seq, got):
            lo, hi = token_range(rank, world, T)
            ok = ok and torch.equal(g[:hi - lo], want[T])
        q.put((rank, ok))
    finally:
        dist.destroy_process_group()


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs two GPUs")
def test_two_gpu_fused_exchange_with_varying_batch_sizes():
    world = 2
    ctx = mp.get_context("spawn")
    q = ctx.Queue()
    port = _free_port()
    procs = [ctx.Process(target=_worker_varying_t, args=(r, world, port, q)) for r in range(world)]
    for p in procs:
        p.start()
    for p in procs:
        p.join(600)
        assert p.exitcode == 0
    res = sorted(q.get(timeout=10) for _ in range(world))
    assert res == [(0, True), (1, True)], res
