"""Edges of how the kernels cut a problem into items.  Forward streams (D <= 64): rows taken in groups that share bias tiles, with groups
cut short at the end of a batch; separate items per stream, with streams that run out; ragged last tiles.
Tolerance: the operator's parity bar (tests/_util.py)."""
import pytest
import torch

from oracle import evo_ref
from _util import assert_parity, bf16_round, oracle_on_rounded, run_layer

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


# D = 96 and 128: pairs of q tiles, or (one tile per row) items dealt to two streams
@pytest.mark.parametrize("B,S,N,H,D", [
    (1, 37, 392, 5, 128),    # four tiles, several pairs per CTA
    (2, 25, 264, 3, 96),     # three tiles: every second pair lacks its second
    (1, 101, 128, 3, 128),   # 303 items for 296 streams: some without a second
    (2, 1, 8, 3, 96),        # fewer items than SMs
])
def test_forward_wide(B, S, N, H, D):
    q, k, v, mask, bias, d_o = evo_ref.make_inputs(B, S, N, H, D, 1.0, 1.0, "bernoulli0.9", seed=3 * S + N)
    got = run_layer(q, k, v, mask, bias, d_o)
    ref = oracle_on_rounded(q, k, v, mask, bias, d_o)
    assert_parity(ref, got, tag=f"B={B} S={S} H={H} N={N} D={D}")


# dQ/dK/dV kernel: whole items (every kv tile of a row and head in one CTA) where (rows x heads) fill the 148
# SMs, single segments where they do not; dQ of whole items stays in tensor memory for one tile at D = 64 and 128
# and up to four at D <= 32, with more it goes through scratch
@pytest.mark.parametrize("bias_type", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("B,S,N,H,D", [
    (1, 49, 264, 3, 32),     # whole, three ragged tiles, in tensor memory
    (1, 49, 520, 3, 32),     # ... five, through scratch
    (1, 37, 328, 4, 64),     # ... three
    (1, 37, 264, 4, 128),
    (1, 74, 200, 2, 96),     # two tiles
    (1, 150, 136, 2, 32),    # ... and two items per CTA, then the segments of four
    (1, 74, 200, 2, 64),
    (1, 160, 72, 2, 16),     # one tile
    (1, 150, 104, 2, 128),   # one tile
    (1, 5, 520, 3, 32),      # segments
    (1, 5, 520, 3, 64),
    (1, 3, 392, 5, 96),
])
def test_backward_items(B, S, N, H, D, bias_type):
    q, k, v, mask, bias, d_o = evo_ref.make_inputs(B, S, N, H, D, 1.0, 1.0, "bernoulli0.9", seed=7 * S + N)
    got = run_layer(q, k, v, mask, bias, d_o, bias_type=bias_type)
    ref = oracle_on_rounded(q, k, v, mask, bias, d_o)
    assert_parity(ref, got, dbias_type=bias_type, tag=f"B={B} S={S} H={H} N={N} D={D}")


# ... and pairs of a row and a head past the last full round of the 148 SMs, dealt by segments after the whole ones
@pytest.mark.parametrize("bias_type", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("B,S,N,H,D", [
    (1, 50, 200, 3, 32),     # 150: scratch and accumulator of whole rows do not fit, so all by segments
    (1, 101, 136, 3, 64),    # 296 + 7; dQ of the whole ones goes through scratch
    (1, 50, 264, 3, 32),     # 150: all by segments, three a CTA
    (1, 99, 264, 3, 32),     # 296 + 1; three tiles in tensor memory
    (1, 50, 392, 3, 64),     # 150: all by segments
    (1, 99, 392, 3, 64),     # 296 + 1; dQ of the whole ones goes through scratch
    (2, 38, 520, 4, 16),     # 296 + 8; through scratch
    (1, 20, 200, 16, 32),    # 296 + 24: the first of the rest lies in the middle of a row
    (1, 19, 264, 8, 64),     # 152: all by segments
    (1, 38, 264, 4, 128),    # D = 128: all of them by segments
    (150, 1, 200, 1, 64),    # 148 + 2 of one row: the same kernel also writes dBias
])
def test_backward_rest(B, S, N, H, D, bias_type):
    q, k, v, mask, bias, d_o = evo_ref.make_inputs(B, S, N, H, D, 1.0, 1.0, "bernoulli0.9", seed=7 * S + N)
    got = run_layer(q, k, v, mask, bias, d_o, bias_type=bias_type)
    ref = oracle_on_rounded(q, k, v, mask, bias, d_o)
    assert_parity(ref, got, dbias_type=bias_type, tag=f"B={B} S={S} H={H} N={N} D={D}")


# dBias over many S rows of inputs of order one passes the flat 2e-2 of the other tests (from S = 300 on at D = 128): its entries
# are of order 50 there.  What it is off by comes from the forward, whose O, and through it delta = rowsum(dO o O) in all of a
# row's dS, has P rounded to bf16.  A P is off by a uniform error of at most 2^-8 of it, so delta by a standard deviation of at
# most 2^-8 / sqrt(3) |P o dP|, and dBias by that times P, added up over the rows: six times it bounds 40,000 entries.  Beside
# it 1e-4 of each dS for what goes with its size (LSE and delta in 16 bits, the cubic exp2 at D = 32).
@pytest.mark.parametrize("S,D", [(300, 128), (1024, 128), (1024, 96), (1024, 64), (1024, 32)])
def test_dbias_over_many_rows(S, D):
    N, H = 104, 2
    q, k, v, mask, bias, d_o = evo_ref.make_inputs(1, S, N, H, D, 1.0, 1.0, "bernoulli0.9", seed=7 * S + N)
    got = run_layer(q, k, v, mask, bias, d_o)
    ref = oracle_on_rounded(q, k, v, mask, bias, d_o)
    assert_parity(ref, got, names=("o", "dq", "dk", "dv"), tag=f"S={S} D={D}")
    assert evo_ref.rel_l2_err(ref["dbias"], got["dbias"]) <= 1e-3
    q, k, v, mask, bias, d_o = bf16_round(q, k, v, mask, bias, d_o)
    logits = torch.einsum("bsihd,bsjhd->bshij", q, k) / D ** 0.5 + bias + mask
    p, dp = torch.softmax(logits, -1), torch.einsum("bsihd,bsjhd->bshij", d_o, v)
    var = (p * dp).square().sum(-1, keepdim=True) * (2.0 ** -16 / 3)
    ds = p * (dp - (p * dp).sum(-1, keepdim=True))
    bound = 6 * (p.square() * var).sum(1).sqrt() + 1e-4 * ds.abs().sum(1) + 1e-4
    off = (got["dbias"][:, 0] - ref["dbias"][:, 0]).abs() / bound
    assert off.max() <= 1, off.max()


# ... in the smallest workspace that is accepted, whose dQ area has no room for N rounded up to 32 rows per pair
@pytest.mark.parametrize("B,S,N,H,D", [
    (1, 5, 264, 3, 32),      # fewer pairs than SMs: segments
    (1, 5, 200, 3, 64),
    (1, 50, 264, 6, 32),     # 296 + 4; the whole ones need no scratch
    (1, 50, 520, 6, 32),     # ... and do
    (1, 49, 520, 3, 32),     # 147 pairs, whole but for the room: segments
    (1, 75, 264, 4, 64),     # 296 + 4 through scratch
    (1, 37, 264, 4, 128),    # D = 128, three tiles: 148 pairs, whole but for the room
    (1, 37, 104, 4, 96),     # ... one tile: whole
])
@pytest.mark.parametrize("gated", [False, True])
def test_backward_smallest_workspace(B, S, N, H, D, gated):
    import _evoattn
    inputs = evo_ref.make_inputs(B, S, N, H, D, 1.0, 1.0, "bernoulli0.9", seed=S + N)
    q, k, v, mask, bias, d_o = (t.cuda().to(torch.bfloat16) for t in inputs)
    dims, st = _evoattn.EvoDims(B, S, N, H, D), torch.cuda.current_stream().cuda_stream
    o, og, resid = (torch.empty_like(q) for _ in range(3))
    lse = torch.empty((B, S, H, N), device="cuda")
    gate = torch.randn_like(q) if gated else None
    _evoattn.fwd_gated(dims, None, q, k, v, bias, mask, gate, o, og if gated else None, resid, lse, 0.0, st)
    full = _evoattn.bwd_gated_workspace_bytes(dims) if gated else _evoattn.bwd_workspace_bytes(dims)
    dh = 32 if D <= 32 else 64 if D <= 64 else 128
    least = full - (-N % 32) * B * S * H * dh * 4 // 256 * 256
    both = _evoattn.BWD_PHASE_DBIAS | _evoattn.BWD_PHASE_DQKV

    def run(size, *phases):
        out = [torch.full_like(q, float("nan")) for _ in range(3)]
        d_gate = torch.full_like(q, float("nan")) if gated else None
        dbias = torch.full((B, H, N, N), float("nan"), device="cuda")
        ws = torch.full((size + 4096,), 0x7f, dtype=torch.uint8, device="cuda")
        for ph in phases:
            _evoattn.bwd_gated(dims, None, q, k, v, bias, mask, gate, o, resid, lse, d_o, *out, d_gate, dbias, ws[:size], 0.0,
                               ph, 0, st)
        _evoattn.device_status()
        assert (ws[size:] == 0x7f).all()          # nothing past the end
        return out + [dbias] + ([d_gate] if gated else [])

    ref = run(full, both)
    for phases in ((both,), (_evoattn.BWD_PHASE_DBIAS, _evoattn.BWD_PHASE_DQKV)):
        got = run(least, *phases)
        for name, a, b in zip(("dq", "dk", "dv", "dbias", "dgate"), ref, got):
            # dQ: the same fp32 partial sums in another order, then bf16; dBias: fp32 sums over slices in any order
            tol = {"dq": 2.0 ** -7, "dbias": 1e-5}.get(name, 0.0) * a.float().abs().max().item()
            assert (a.float() - b.float()).abs().max().item() <= tol, name
    with pytest.raises(_evoattn.EvoAttnError) as e:
        run(least - 256, both)
    assert e.value.code == -4
