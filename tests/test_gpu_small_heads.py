"""dQ, dK, dV (and dBias of one S row) at head dims 16 and 32, at the edges of the kernel's tiles, halves and walks.

A tile is 128 kv rows by two halves of 64 q columns.  A CTA takes (row, head) pairs whole as far as they fill rounds of the 148 SMs,
and the pairs left over by single kv tiles ("segments").  dQ of a whole pair stays in tensor memory for up to four tiles and goes
through a scratch area from five on; segments add theirs to an accumulator.
"""
import pytest
import torch

from oracle import evo_ref
from _util import assert_parity, oracle_on_rounded, run_layer

pytestmark = pytest.mark.gpu

SIZES = [8, 64, 72, 128, 136, 192, 200, 256, 384, 392, 456, 512, 520, 648]


# 4 and 12 pairs: whole with one tile, by segments with more.
@pytest.mark.parametrize("S", [1, 3])
@pytest.mark.parametrize("N", SIZES)
@pytest.mark.parametrize("D,bias_type", [(16, torch.float32), (32, torch.bfloat16), (32, torch.float32)])
def test_tiles_and_halves(D, bias_type, N, S):
    q, k, v, mask, bias, d_o = evo_ref.make_inputs(2, S, N, 2, D, 0.5, 1.0, "bernoulli0.9", seed=N + S)
    got = run_layer(q, k, v, mask, bias, d_o, bias_type=bias_type)
    assert_parity(oracle_on_rounded(q, k, v, mask, bias, d_o), got, dbias_type=bias_type, tag=f"N={N} S={S} D={D}")


@pytest.mark.parametrize("S,N,D", [
    (37, 392, 16), (37, 512, 32),       # 148 pairs of four tiles: as many dQ accumulators as there are, in use at once
    (74, 456, 16), (74, 512, 32),       # ... 296 pairs: and again by the next pair
    (74, 384, 32),                      # three tiles: the accumulators of a pair begin where those before it ended
    (37, 648, 32), (74, 520, 16),       # six and five tiles: through scratch
])
def test_whole_pairs(S, N, D):
    q, k, v, mask, bias, d_o = evo_ref.make_inputs(1, S, N, 4, D, 0.5, 1.0, "bernoulli0.9", seed=N + S)
    got = run_layer(q, k, v, mask, bias, d_o)
    assert_parity(oracle_on_rounded(q, k, v, mask, bias, d_o), got, tag=f"N={N} S={S} D={D}")


# H = 4.  The pairs past the last full round are dealt by segments if that ends sooner.
@pytest.mark.parametrize("S,N", [
    (80, 120),      # one tile: it never does; 320 whole pairs
    (40, 264),      # 148 whole + 36 segments, three tiles
    (80, 264),      # 296 whole + 72
    (59, 264),      # 148 whole + 264: up to two segments a CTA, of different pairs
    (75, 392),      # 296 whole + 16, four tiles
    (40, 520),      # 148 whole, through scratch, + 60
    (59, 520),      # 148 whole, through scratch, + 440: up to three segments a CTA
])
def test_pairs_left_over_after_full_rounds(S, N):
    q, k, v, mask, bias, d_o = evo_ref.make_inputs(1, S, N, 4, 32, 0.5, 1.0, "tail0to32", seed=N)
    got = run_layer(q, k, v, mask, bias, d_o)
    assert_parity(oracle_on_rounded(q, k, v, mask, bias, d_o), got, tag=f"N={N} S={S}")


# One S row: the kernel also writes dBias, from fragments.
@pytest.mark.parametrize("D,bias_type", [(16, torch.float32), (16, torch.bfloat16), (32, torch.float32), (32, torch.bfloat16)])
@pytest.mark.parametrize("B,N,H", [
    (38, 104, 8),      # 304 pairs of one tile, taken whole
    (8, 512, 16),      # 128 pairs of four tiles, whole: dQ stays in tensor memory
    (8, 640, 16),      # ... of five: dQ through scratch
    (150, 200, 1),     # 148 whole, then the segments of two pairs
    (38, 392, 8),      # 296 whole, then the segments of eight
])
def test_one_row(B, N, H, D, bias_type):
    q, k, v, mask, bias, d_o = evo_ref.make_inputs(B, 1, N, H, D, 0.5, 1.0, "bernoulli0.9", seed=B + N)
    got = run_layer(q, k, v, mask, bias, d_o, bias_type=bias_type)
    assert_parity(oracle_on_rounded(q, k, v, mask, bias, d_o), got, dbias_type=bias_type, tag=f"B={B} N={N} H={H} D={D}")
