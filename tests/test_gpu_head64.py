"""dQ, dK, dV (and dBias of one S row) at head dim 64, at the edges of the kernel's tiles, rings and walks.

Q has three buffers, dO and K two, V one; one dQ accumulator, so that from two kv tiles on the partial sums of a whole (row, head)
pair go through the scratch area of its CTA, and those of the pairs left over after full rounds of the 148 SMs to an accumulator.
"""
import pytest
import torch

from oracle import evo_ref
from _util import assert_parity, oracle_on_rounded, run_layer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,S,N,H,bias_type", [
    (1, 3, 64, 2, torch.float32),        # one tile, six pairs
    (1, 160, 128, 2, torch.float32),     # one tile, 320 whole pairs: three segments, of one step each, a CTA
    (1, 5, 136, 2, torch.float32),       # two tiles, by segments; the second of eight rows
    (1, 75, 192, 4, torch.bfloat16),     # two tiles, 296 whole and four left over; half a tile of q rows missing
    (1, 74, 256, 4, torch.float32),      # ... 296 whole: the scratch area is used again by the next pair
    (1, 40, 264, 4, torch.bfloat16),     # three tiles, 148 whole and twelve left over
    (1, 37, 520, 4, torch.float32),      # five tiles, 148 whole
    (2, 1, 264, 2, torch.float32),       # one row: dBias from fragments, fp32 ...
    (38, 1, 200, 8, torch.bfloat16),     # ... and bf16, with whole pairs and segments
    (38, 1, 136, 8, torch.float32),
])
def test_head64(B, S, N, H, bias_type):
    q, k, v, mask, bias, d_o = evo_ref.make_inputs(B, S, N, H, 64, 0.5, 1.0, "bernoulli0.9", seed=N + S)
    got = run_layer(q, k, v, mask, bias, d_o, bias_type=bias_type)
    assert_parity(oracle_on_rounded(q, k, v, mask, bias, d_o), got, dbias_type=bias_type, tag=f"B={B} S={S} N={N} H={H}")
