"""Edges of the forward's item streams (D <= 64): rows taken in groups that share bias tiles, with groups
cut short at the end of a batch; separate items per stream, with streams that run out; ragged last tiles.
Tolerance: the operator's parity bar (tests/_util.py)."""
import pytest

from oracle import evo_ref
from _util import assert_parity, oracle_on_rounded, run_layer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,S,N,H,D", [
    (2, 40, 264, 3, 32),     # 40 = 13 groups of three rows + one row, in each of two batches
    (2, 41, 264, 3, 64),     # groups of two rows, the last with one
    (1, 75, 128, 4, 16),     # one kv tile per item
    (50, 1, 136, 3, 32),     # one row per batch: separate items, 300 of them on 148 SMs
    (40, 1, 264, 2, 64),
    (1, 3, 1000, 8, 32),     # eight ragged tiles, fewer items than streams
])
def test_forward_streams(B, S, N, H, D):
    q, k, v, mask, bias, d_o = evo_ref.make_inputs(B, S, N, H, D, 1.0, 1.0, "bernoulli0.9", seed=B + S + N)
    got = run_layer(q, k, v, mask, bias, d_o)
    ref = oracle_on_rounded(q, k, v, mask, bias, d_o)
    assert_parity(ref, got, tag=f"B={B} S={S} H={H} N={N} D={D}")
