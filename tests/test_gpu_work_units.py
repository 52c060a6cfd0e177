"""The kernels that draw their work: the expert GEMMs at the edges of their 128-row tiles, as one launch and cut
between the two GEMMs, and the decode kernel where its rows are handed from phase to phase."""
import numpy as np
import pytest
import torch

import helpers as hp
from helpers import H, RSF

pytestmark = pytest.mark.gpu

OFFSET = 96   # the shard's routing group is the fourth


def _inputs(rows_a, rows_b, T, seed):
    """`rows_a` tokens whose only expert in this shard is its third one, `rows_b` whose only one is its 18th; the rest
    have none.  The other seven picks lie in groups outside the shard."""
    rng = np.random.Generator(np.random.PCG64(seed))
    logits = rng.standard_normal((T, 256)).astype(np.float32) * 0.05 - 6.0
    away = [0, 1, 32, 33, 64, 65, 66, 160, 161]
    order = rng.permutation(T)
    for i, t in enumerate(order):
        local = [OFFSET + 2] if i < rows_a else [OFFSET + 17] if i < rows_a + rows_b else []
        picks = away[:7] + local if local else away[:6] + away[7:]
        logits[t, picks] += 8.0
    bias = torch.zeros(256, dtype=torch.bfloat16)
    _, _, hidden, hscale = hp.cpu_inputs(T, seed)
    return torch.from_numpy(logits), bias, hidden, hscale


# one row; the last row of a 64-row stage and one more; one row less than a tile, a tile, one more; two tiles and one
# row.  T <= 64 runs the four-stage form, more the three-stage one.
@pytest.mark.parametrize("rows_a,rows_b,T", [(1, 0, 9), (63, 1, 64), (64, 0, 64), (64, 1, 65), (65, 3, 90), (127, 0, 127),
                                             (128, 5, 140), (129, 128, 300), (257, 31, 300)])
def test_expert_gemms_at_tile_edges(pkg, oracle, rows_a, rows_b, T):
    layer = pkg.MoeLayer(T, 32, 0)
    cut = pkg.MoeLayer(T, 32, 0)
    cut.set_stage_timing(True)   # the two GEMMs as launches of their own
    try:
        inputs = _inputs(rows_a, rows_b, T, 700 + T + rows_a)
        weights = hp.gpu_shard(OFFSET, 32)
        for _ in range(2):       # the second run finds the counters as the first left them
            got = hp.run_layer(layer, inputs, weights, OFFSET)
        counts = layer.read("expert_count", 32)
        assert counts[2] == rows_a and counts[17] == rows_b and counts.sum() == rows_a + rows_b
        assert torch.equal(got.view(torch.int16), hp.run_layer(cut, inputs, weights, OFFSET).view(torch.int16))
        w1, s1, w2, s2 = weights
        ref, rows = oracle.layer(inputs[0].numpy(), hp.np_u16(inputs[1]), hp.np_u8(inputs[2]), inputs[3].numpy(),
                                 hp.np_u8(w1), s1.cpu().numpy(), hp.np_u8(w2), s2.cpu().numpy(), OFFSET, RSF)
        assert rows == rows_a + rows_b
        out, want = got.float().cpu().numpy(), oracle.bf16_decode(ref)
        # a sum in another order moves single e4m3 codes of the activations (2^-4 of a value each): 2e-2 over a row
        assert hp.error_stats(out, want)["rel_l2"] < 2e-2
        routed = np.abs(want).max(axis=1) > 0
        assert routed.sum() == rows and np.all(out[~routed] == 0)
        worst = (np.linalg.norm(out - want, axis=1)[routed] / np.linalg.norm(want, axis=1)[routed]).max()
        assert worst < 4e-2, worst   # every single row is there
    finally:
        layer.close()
        cut.close()


@pytest.mark.parametrize("rows_a,rows_b,T", [(1, 1, 2), (4, 1, 5), (8, 0, 8), (3, 5, 8)])
def test_decode_rows_between_the_phases(pkg, rows_a, rows_b, T):
    """Up to all eight rows on one expert, against the staged chain; then a row that is not a number: its own output
    is not a number either, the others are as before, no wait runs out and the next call is clean."""
    dec, chain = pkg.MoeLayer(16, 32, 0), pkg.MoeLayer(16, 32, 0)
    chain.set_decode_kernel(False)
    try:
        inputs = _inputs(rows_a, rows_b, T, 900 + T + rows_a)
        weights = hp.gpu_shard(OFFSET, 32)
        want = hp.run_layer(chain, inputs, weights, OFFSET).float().cpu().numpy()
        first = hp.run_layer(dec, inputs, weights, OFFSET)
        assert hp.error_stats(first.float().cpu().numpy(), want)["rel_l2"] < 5e-3
        broken = [x.clone() for x in inputs]
        broken[3][5, 0] = float("nan")
        out = hp.run_layer(dec, broken, weights, OFFSET)
        assert torch.isnan(out[0].float()).all()
        assert torch.equal(out[1:].view(torch.int16), first[1:].view(torch.int16))
        again = hp.run_layer(dec, inputs, weights, OFFSET)
        assert torch.equal(again.view(torch.int16), first.view(torch.int16))
    finally:
        dec.close()
        chain.close()
