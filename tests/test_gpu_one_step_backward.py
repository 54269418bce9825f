"""The backward of one S row of one tile, at most one (batch, head) pair a CTA and D <= 64: one kernel, whose drain warps form the terms that
the prep kernel otherwise writes.  148 pairs are the last that take it on 148 SMs."""
import pytest
import torch

from oracle import evo_ref
from _util import assert_parity, oracle_on_rounded, run_layer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bias_type", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("D", [16, 32, 64])
@pytest.mark.parametrize("B,N,H", [(1, 8, 1), (3, 40, 2), (37, 120, 4), (37, 128, 4), (149, 128, 1)])
def test_parity(B, N, H, D, bias_type):
    q, k, v, mask, bias, d_o = evo_ref.make_inputs(B, 1, N, H, D, 0.5, 1.0, "bernoulli0.9", seed=B + N + D)
    got = run_layer(q, k, v, mask, bias, d_o, bias_type=bias_type)
    assert_parity(oracle_on_rounded(q, k, v, mask, bias, d_o), got, dbias_type=bias_type, tag=f"B={B} N={N} H={H} D={D}")


@pytest.mark.parametrize("resid", [True, False])
@pytest.mark.parametrize("D", [16, 64])
@pytest.mark.parametrize("head_major", [True, False])
def test_equals_two_phases(D, resid, head_major):
    """Against the prep kernel, which a backward in two phases runs: the same terms, bit for bit."""
    import _evoattn
    B, N, H = 3, 104, 4
    q, k, v, mask, bias, d_o = (t.cuda().to(torch.bfloat16) for t in evo_ref.make_inputs(B, 1, N, H, D, 0.5, 1.0, "bernoulli0.9", seed=D))
    st, dims = torch.cuda.current_stream().cuda_stream, _evoattn.EvoDims(B, 1, N, H, D)
    if head_major:                          # stored [B][S][H][N][D]
        q, k, v, d_o = (t.transpose(2, 3).contiguous().transpose(2, 3) for t in (q, k, v, d_o))
    strides = _evoattn.EvoStrides(*q.stride()[:4]) if head_major else None
    o, res, lse = torch.empty_like(q), torch.empty_like(q), torch.empty((B, 1, H, N), device="cuda")
    _evoattn.fwd_gated(dims, strides, q, k, v, bias, mask, None, o, None, res, lse, 0.0, st)
    ws = torch.empty(_evoattn.bwd_workspace_bytes(dims), dtype=torch.uint8, device="cuda")
    both = _evoattn.BWD_PHASE_DBIAS | _evoattn.BWD_PHASE_DQKV
    outs = []
    for phases in ((both,), (_evoattn.BWD_PHASE_DBIAS, _evoattn.BWD_PHASE_DQKV)):
        out = [torch.empty_like(q) for _ in range(3)] + [torch.empty((B, H, N, N), device="cuda")]
        for ph in phases:
            _evoattn.bwd_gated(dims, strides, q, k, v, bias, mask, None, o, res if resid else None, lse, d_o, *out[:3], None, out[3], ws, 0.0,
                               ph, 0, st)
        outs.append(out)
    _evoattn.device_status()
    for name, a, b in zip(("dq", "dk", "dv"), *outs):
        assert torch.equal(a, b), name
    # a quarter of the dBias kernel's exponentials at D <= 32 are polynomials, relative error 7.5e-5
    a, b = outs[0][3], outs[1][3]
    assert (a - b).abs().max() <= 1e-4 * b.abs().max()
