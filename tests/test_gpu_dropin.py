"""The drop-in `run(...)`, whose handles the caller never sees: what it may not remember from one call to the next."""
import threading

import pytest
import torch

import helpers as hp
from helpers import H, RSF

pytestmark = pytest.mark.gpu


def _fresh(pkg, dev, weights, T):
    """The result of a handle that has seen no other tensors."""
    layer = pkg.MoeLayer(T, 32, 0)
    try:
        out = torch.empty(T, H, dtype=torch.bfloat16, device="cuda")
        layer.run(*dev, *weights, 0, RSF, out)
        layer.check()
        return out.view(torch.int16)
    finally:
        layer.close()


# decode kernel; the smallest and a middle batch of the four-stage GEMMs; the three-stage ones
@pytest.mark.parametrize("T", [4, 9, 40, 300])
def test_other_scales_at_the_same_addresses_are_seen(pkg, T):
    dev = [x.cuda() for x in hp.cpu_inputs(T, seed=7000 + T)]
    w1, s1, w2, s2 = hp.gpu_shard(0, 32)
    a, b = s1.clone(), s2.clone()
    out = torch.empty(T, H, dtype=torch.bfloat16, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(T)
    for _ in range(3):
        pkg.run(*dev, w1, a, w2, b, 0, RSF, out)
        got = out.view(torch.int16).clone()
        assert torch.equal(got, _fresh(pkg, dev, (w1, a.clone(), w2, b.clone()), T))
        a.mul_(torch.rand(a.shape, generator=g, device="cuda") + 0.5)
        b.mul_(torch.rand(b.shape, generator=g, device="cuda") + 0.5)


# split-K (decode kernel off), both rings of the expert GEMMs, other shapes down to one K block
@pytest.mark.parametrize("T,E,hidden,inter,decode", [(3, 32, H, 2048, False), (9, 32, H, 2048, True), (65, 64, H, 2048, True),
                                                     (40, 32, 8192, 256, True), (40, 32, 256, 8192, True), (17, 32, 256, 128, True)])
def test_scales_in_place_change_nothing(pkg, T, E, hidden, inter, decode):
    from fp8_moe_dev_b200 import gen
    layer = pkg.MoeLayer(T, E, 0, hidden=hidden, intermediate=inter)
    layer.set_decode_kernel(decode)
    try:
        logits, bias = gen.make_routing(T, seed=7100 + T)
        hid, scale = gen.make_hidden(T, seed=7101 + T, hidden=hidden)
        weights = gen.make_shard(0, E, device="cuda", out_device="cuda", hidden=hidden, inter=inter)
        outs = []
        for on in (False, True, False):
            layer.set_scales_in_place(on)
            out = torch.zeros(T, hidden, dtype=torch.bfloat16, device="cuda")
            layer.run(logits.cuda(), bias.cuda(), hid.cuda(), scale.cuda(), *weights, 0, RSF, out)
            layer.check()
            outs.append(out.view(torch.int16))
        assert torch.count_nonzero(outs[0]) > 0
        assert torch.equal(outs[1], outs[0]) and torch.equal(outs[2], outs[0])
    finally:
        layer.close()


def test_overlapping_calls_from_threads_and_streams(pkg):
    """Calls of several batch sizes on two threads, each with a stream of its own and one made outside torch, none of
    them ordered by the caller: every result is the one of a call alone."""
    cases = {}
    for T in (3, 40, 300):
        dev = [x.cuda() for x in hp.cpu_inputs(T, seed=7200 + T)]
        weights = hp.gpu_shard(0, 32)
        cases[T] = (dev, weights, _fresh(pkg, dev, weights, T))
    torch.cuda.synchronize()
    own = [torch.cuda.Stream() for _ in range(2)]
    assert all(s.stream_id & 1 for s in own) and torch.cuda.default_stream().stream_id == 0
    foreign = torch.cuda.ExternalStream(own[1].cuda_stream)
    assert foreign.stream_id != 0 and foreign.stream_id & 1 == 0
    wrong = []

    def work(streams):
        outs = []
        for k in range(30):
            for T, (dev, weights, want) in cases.items():
                with torch.cuda.stream(streams[k % len(streams)]):
                    out = torch.empty(T, H, dtype=torch.bfloat16, device="cuda")
                    pkg.run(*dev, *weights, 0, RSF, out)
                outs.append((out, want))
        torch.cuda.synchronize()
        wrong.extend(not torch.equal(out.view(torch.int16), want) for out, want in outs)

    threads = [threading.Thread(target=work, args=(s,)) for s in ([own[0], torch.cuda.default_stream()], [foreign])]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(wrong) == 180 and not any(wrong)
