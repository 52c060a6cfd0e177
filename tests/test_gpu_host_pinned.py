"""run_host with pinned buffers, which the kernels reach in place, against the copying form (pageable buffers)
and the device-resident call: the same bits in every row, those of tokens without a local expert among them."""
import ctypes as C

import pytest
import torch

import helpers as hp
from helpers import RSF

pytestmark = pytest.mark.gpu


def _in_block(x, shift):
    """`x` in pinned memory, `shift` bytes behind the start of its allocation, with bytes on either side."""
    block = torch.zeros(shift + x.numel() * x.element_size() + 64, dtype=torch.uint8).pin_memory()
    part = block[shift:shift + x.numel() * x.element_size()].view(x.dtype).view(x.shape)
    part.copy_(x)
    return part


# batches on both sides of the decode kernel's limit (8), of the rule that writes empty rows aside (256 tokens, 64
# experts) and of its other shape; logits and scales 4 bytes off a 16-byte boundary take the word-wise fetch
@pytest.mark.parametrize("T,E,hidden,inter,shift", [
    (1, 32, 7168, 2048, 0), (8, 32, 7168, 2048, 4), (9, 32, 7168, 2048, 0), (255, 32, 7168, 2048, 4),
    (256, 32, 7168, 2048, 0), (257, 64, 7168, 2048, 4), (300, 128, 7168, 2048, 0), (3, 32, 1024, 512, 0),
    (400, 32, 1024, 512, 4), (300, 32, 8192, 256, 0)])
def test_pinned_buffers_in_place(pkg, T, E, hidden, inter, shift):
    from fp8_moe_dev_b200 import gen
    layer = pkg.MoeLayer(512, E, 0, hidden=hidden, intermediate=inter)
    try:
        logits, bias = gen.make_routing(T, seed=50 + T)
        hid, scale = gen.make_hidden(T, seed=60 + T, hidden=hidden)
        weights = gen.make_shard(0, E, device="cuda", out_device="cuda", hidden=hidden, inter=inter)
        bias = bias.cuda()
        want = torch.empty(T, hidden, dtype=torch.bfloat16, device="cuda")
        layer.run(logits.cuda(), bias, hid.cuda(), scale.cuda(), *weights, 0, RSF, want)
        layer.check()
        want = want.cpu().view(torch.int16)
        pageable = torch.full((T, hidden), 7.0, dtype=torch.bfloat16)
        layer.run_host(logits, bias, hid, scale, *weights, 0, RSF, pageable)
        assert torch.equal(pageable.view(torch.int16), want)
        src = [_in_block(logits, shift), _in_block(hid, 16), _in_block(scale, shift)]
        for _ in range(2):
            out = _in_block(torch.full((T, hidden), 7.0, dtype=torch.bfloat16), 32)
            layer.run_host(src[0], bias, src[1], src[2], *weights, 0, RSF, out)
            assert torch.equal(out.view(torch.int16), want)
        layer.check()
    finally:
        layer.close()


def test_output_over_an_input_is_taken(pkg):
    """An output that shares memory with the activations: the inputs are read before the first row is written."""
    T = 300
    layer = pkg.MoeLayer(512, 32, 0)
    try:
        inputs = hp.cpu_inputs(T, seed=77)
        weights = hp.gpu_shard(0, 32)
        want = hp.run_layer(layer, inputs, weights, 0).cpu()
        block = torch.zeros(T * 7168 * 2, dtype=torch.uint8).pin_memory()
        hid = block[:T * 7168].view(torch.float8_e4m3fn).view(T, 7168)
        hid.copy_(inputs[2])
        out = block.view(torch.bfloat16).view(T, 7168)
        layer.run_host(inputs[0].pin_memory(), inputs[1].cuda(), hid, inputs[3].pin_memory(), *weights, 0, RSF, out)
        assert torch.equal(out.view(torch.int16), want.view(torch.int16))
    finally:
        layer.close()


@pytest.mark.parametrize("T,which", [(4, "logits"), (40, "logits"), (40, "scale"), (300, "both")])
def test_floats_off_their_boundary_are_copied(pkg, T, which):
    """Pinned logits or scales at any byte address: taken as before, through the copies, which take any address."""
    layer = pkg.MoeLayer(512, 32, 0)
    try:
        inputs = hp.cpu_inputs(T, seed=80 + T)
        weights = hp.gpu_shard(0, 32)
        want = hp.run_layer(layer, inputs, weights, 0).cpu()
        bias, out = inputs[1].cuda(), torch.empty(T, 7168, dtype=torch.bfloat16).pin_memory()
        for off in (1, 2, 3, 4, 6):
            blocks = []
            for x, moved in ((inputs[0], which != "scale"), (inputs[3], which != "logits")):
                at = off if moved else 0
                block = torch.zeros(x.numel() * 4 + 16, dtype=torch.uint8).pin_memory()
                block[at:at + x.numel() * 4].copy_(x.reshape(-1).view(torch.uint8))
                blocks.append((block, block.data_ptr() + at))
            hidden = inputs[2].pin_memory()
            a = pkg._lib.Args(blocks[0][1], bias.data_ptr(), hidden.data_ptr(), blocks[1][1], *(w.data_ptr() for w in weights),
                              0, RSF, out.data_ptr(), T)
            out.fill_(7.0)
            rc = layer._lib.moe_fp8_b200_run_host(layer._h, C.byref(a), C.c_void_p(torch.cuda.current_stream().cuda_stream))
            assert rc == 0, layer._lib.moe_fp8_b200_last_error(layer._h)
            assert layer.host_path() == ("in place" if off == 4 else "copies")
            assert torch.equal(out.view(torch.int16), want.view(torch.int16))
        layer.check()
    finally:
        layer.close()


# both sides of the rules: 128 experts copy above 1024 tokens; 256 experts never; empty rows leave aside from 256
# tokens on up to 64 experts
@pytest.mark.parametrize("T,E,path", [(8, 32, "in place"), (256, 64, "in place"), (1024, 128, "in place"), (1025, 128, "copies"),
                                      (1025, 256, "in place"), (2048, 32, "in place")])
def test_which_path_a_pinned_call_takes(pkg, T, E, path):
    """... and that new contents of the same pinned buffers are seen."""
    layer = pkg.MoeLayer(T, E, 0)
    try:
        weights = hp.gpu_shard(0, E)
        src = [None if i == 1 else x.pin_memory() for i, x in enumerate(hp.cpu_inputs(T, seed=90))]
        out = torch.empty(T, 7168, dtype=torch.bfloat16).pin_memory()
        assert layer.host_path() is None
        for seed in (91, 92):
            inputs = hp.cpu_inputs(T, seed=seed)
            want = hp.run_layer(layer, inputs, weights, 0).cpu()
            for i in (0, 2, 3):
                src[i].copy_(inputs[i])
            layer.run_host(src[0], inputs[1].cuda(), src[2], src[3], *weights, 0, RSF, out)
            assert layer.host_path() == path
            assert torch.equal(out.view(torch.int16), want.view(torch.int16))
        layer.run_host(inputs[0], inputs[1].cuda(), inputs[2], inputs[3], *weights, 0, RSF, torch.empty_like(want))
        assert layer.host_path() == "copies"      # pageable
    finally:
        layer.close()


@pytest.mark.parametrize("T", [5, 255, 256, 700])
def test_no_token_has_an_expert_here(pkg, T):
    """Every selected expert lies outside the shard: no tile, no row; the output is zeros, written aside from 256
    tokens on."""
    layer = pkg.MoeLayer(700, 32, 0)
    try:
        logits, bias, hid, scale = hp.cpu_inputs(T, seed=95)
        logits = logits - 8.0
        logits[:, 64:72] += 16.0
        weights = hp.gpu_shard(0, 32)
        out = torch.full((T, 7168), 7.0, dtype=torch.bfloat16).pin_memory()
        layer.run_host(logits.pin_memory(), (bias * 0).cuda(), hid.pin_memory(), scale.pin_memory(), *weights, 0, RSF, out)
        assert layer.host_path() == "in place" and torch.count_nonzero(out) == 0
        assert layer.read("expert_count", 32).sum() == 0
        layer.check()
    finally:
        layer.close()
