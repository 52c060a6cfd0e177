"""run_host with pinned buffers, which the kernels reach in place, against the copying form (pageable buffers)
and the device-resident call: the same bits in every row, those of tokens without a local expert among them."""
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
