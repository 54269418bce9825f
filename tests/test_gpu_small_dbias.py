"""dBias of small problems, which the dQ/dK/dV kernel adds up in memory instead of leaving it to the dBias kernel: up to seven steps
(pairs of tiles) for the fullest of 148 CTAs, in a backward that is one call, at D <= 32 where (row, head) pairs are taken whole, at D = 64 also where
they are dealt by kv tiles.  With one step a CTA and a bf16 result the warp
that adds the last row to its part of a tile converts it, otherwise a kernel behind does."""
import pytest
import torch

from oracle import evo_ref
from _util import assert_parity, oracle_on_rounded, run_layer

pytestmark = pytest.mark.gpu

CASES = [
    # (B, S, N, H): one step a CTA, parts of 32 x 32 empty, ragged and full; one row more than a CTA has
    (1, 2, 8, 1), (2, 17, 40, 2), (1, 37, 64, 4), (1, 74, 120, 2), (2, 3, 128, 24),
    (1, 75, 104, 2),        # 150 pairs of one tile: two steps
    (1, 100, 72, 8),        # six
    (1, 518, 64, 2),        # seven, 518 rows to a sum
    (1, 65, 128, 16),       # eight: the dBias kernel
    (2, 2, 136, 3),         # two tiles, by segments
    (1, 45, 200, 3),        # ... whole
    (1, 2, 840, 3),         # seven tiles by segments, one step short of the line
    (1, 3, 904, 2),         # eight tiles: over it
]


@pytest.mark.parametrize("bias_type", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("D", [16, 32, 64])
@pytest.mark.parametrize("B,S,N,H", CASES)
def test_small_dbias(B, S, N, H, D, bias_type):
    q, k, v, mask, bias, d_o = evo_ref.make_inputs(B, S, N, H, D, 0.5, 1.0, "bernoulli0.9", seed=N + S + D)
    ref = oracle_on_rounded(q, k, v, mask, bias, d_o)
    for _ in range(2):                  # (counters and sums start anew with every call)
        got = run_layer(q, k, v, mask, bias, d_o, bias_type=bias_type)
        assert_parity(ref, got, dbias_type=bias_type, tag=f"B={B} S={S} N={N} H={H} D={D}")
