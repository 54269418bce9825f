"""Small problems, whose backward has kernels fewer (dBias added up and converted by the dQ/dK/dV kernel, one kernel for one S row of one tile), on other
layouts than contiguous ones and with infinities and NaN."""
import pytest
import torch

from oracle import evo_ref

pytestmark = pytest.mark.gpu
bf = torch.bfloat16
SHAPES = [(1, 8, 64, 2), (2, 3, 104, 3), (3, 1, 104, 2), (1, 1, 128, 4)]      # (B, S, N, H): one step a CTA


def _views(kind, ts):
    B, S, N, H, D = ts[0].shape
    if kind == "fused":
        return torch.stack(ts, 3).unbind(3)
    if kind == "fused by heads":
        return torch.cat(ts, 4).split(D, 4)
    return [t.transpose(1, 2).contiguous().transpose(1, 2) for t in ts]


@pytest.mark.parametrize("kind", ["fused", "fused by heads", "ending"])
@pytest.mark.parametrize("D", [16, 32, 64])
@pytest.mark.parametrize("B,S,N,H", SHAPES)
def test_views_equal_copies(B, S, N, H, D, kind):
    from tk_evo_attention_layer import TKEvoAttention
    q, k, v, mask, bias, d_o = (t.cuda().to(bf) for t in evo_ref.make_inputs(B, S, N, H, D, 0.5, 1.0, "bernoulli0.9", seed=N + D))
    mask, bias = mask.reshape(B, S, 1, 1, N), bias.reshape(B, 1, H, N, N)
    outs = []
    for ts in ((q, k, v), _views(kind, [q, k, v])):
        wrt = [t.detach().requires_grad_() for t in (*ts, bias)]
        o = TKEvoAttention.apply(*wrt[:3], mask, wrt[3])
        outs.append([o.detach(), *torch.autograd.grad(o, wrt, d_o)])
    for name, a, b in zip(("o", "dq", "dk", "dv", "dbias"), *outs):
        if name == "dbias" and S > 2:      # up to eight fp32 terms in any order, rounded to bf16 once
            assert (a.float() - b.float()).abs().max() <= 2.0 ** -8 * a.float().abs().max()
        else:
            assert torch.equal(a, b), name


@pytest.mark.parametrize("D", [16, 32, 64])
@pytest.mark.parametrize("B,S,N,H", SHAPES)
@pytest.mark.parametrize("what", ["row of -inf", "some -inf", "nan in q", "lowest mask"])
def test_ends_of_the_range_equal_two_phases(B, S, N, H, D, what):
    """Against the prep and dBias kernels, which a backward in two phases runs: the same results, NaN in the same places."""
    import _evoattn
    q, k, v, mask, bias, d_o = (t.cuda().to(bf) for t in evo_ref.make_inputs(B, S, N, H, D, 0.5, 1.0, "bernoulli0.9", seed=N + D))
    mask = mask.reshape(B, S, N).clone()
    if what == "row of -inf":
        mask[0, 0] = float("-inf")
    elif what == "some -inf":
        mask[:, :, 1::3] = float("-inf")
    elif what == "lowest mask":
        mask[:, :, 2::5] = torch.finfo(bf).min
    else:
        q[0, 0, 5, 0, 3] = float("nan")
    st, dims = torch.cuda.current_stream().cuda_stream, _evoattn.EvoDims(B, S, N, H, D)
    o, res, lse = torch.empty_like(q), torch.empty_like(q), torch.empty((B, S, H, N), device="cuda")
    _evoattn.fwd(dims, q, k, v, bias, mask, o, res, lse, 0.0, st)
    ws = torch.empty(_evoattn.bwd_workspace_bytes(dims), dtype=torch.uint8, device="cuda")
    both, outs = _evoattn.BWD_PHASE_DBIAS | _evoattn.BWD_PHASE_DQKV, []
    for phases in ((both,), (_evoattn.BWD_PHASE_DBIAS, _evoattn.BWD_PHASE_DQKV)):
        out = [torch.full_like(q, 7.0) for _ in range(3)] + [torch.full((B, H, N, N), 7.0, device="cuda")]
        for ph in phases:
            _evoattn.bwd_phased(dims, None, q, k, v, bias, mask, o, res, lse, d_o, *out, ws, 0.0, ph, 0, st)
        outs.append(out)
    _evoattn.device_status()
    for name, a, b in zip(("dq", "dk", "dv", "dbias"), *outs):
        if name == "dbias" and S == 1 and D <= 32 and what == "nan in q":
            continue        # (one S row's dBias has no polynomials, the dBias kernel's drop a NaN in their columns)
        assert torch.equal(a.isnan(), b.isnan()), name
        x, y = (t.nan_to_num(0.0, 0.0, 0.0) for t in (a, b))
        if name != "dbias":
            assert torch.equal(x, y), name
        else:               # one S row at D <= 32: polynomials on one side only (7.5e-5); else fp32 terms in any order
            assert (x - y).abs().max() <= (1e-4 if S == 1 and D <= 32 else 1e-5) * y.abs().max()
