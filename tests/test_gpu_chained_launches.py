"""Kernels of a step are programmatic launches: a wait of their own is what orders them behind the kernel ahead of them.

Calls are queued without a wait, each on what the one before wrote and with no other kernel in between, into buffers that hold NaN until
then; the other arm waits after every call and takes the backward in its two phases, whose kernels are launched in full order.  O, LSE, dK and dV are
bit-reproducible, and so is dQ of up to two kv tiles (two fp32 partial sums meet in either order); dBias of several slices of S is their fp32 sum
in any order, and one S row's comes from another kernel in a phased call (exp2 as a cubic, 7.5e-5): 1e-4 of the largest.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _given(B, S, N, H, D, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    q, k, v, d_o = (torch.randn((B, S, N, H, D), generator=gen, device="cuda").mul(0.5).bfloat16() for _ in range(4))
    bias = torch.randn((B, H, N, N), generator=gen, device="cuda").bfloat16()
    mask = torch.where(torch.rand((B, S, N), generator=gen, device="cuda") < 0.9, 0.0, -1e9).bfloat16()
    mask[..., 0] = 0
    return q, k, v, d_o, bias, mask


def _outputs(like, n):
    return [torch.full_like(like, float("nan")) for _ in range(n)]


@pytest.mark.parametrize("B,S,N,H,D", [
    (4, 1, 512, 16, 64),     # separate items
    (1, 8, 64, 2, 32),       # fewer blocks than SMs
    (1, 100, 264, 4, 32),    # rows that share bias tiles, several items a stream
    (1, 60, 200, 4, 128),
])
def test_forwards_without_a_wait(B, S, N, H, D):
    import _evoattn
    q, k, v, _, bias, mask = _given(B, S, N, H, D, 5)
    dims, st = _evoattn.EvoDims(B, S, N, H, D), torch.cuda.current_stream().cuda_stream

    def run(wait):
        outs = [(*_outputs(q, 2), torch.full((B, S, H, N), float("nan"), device="cuda")) for _ in range(12)]
        x = q
        torch.cuda.synchronize()
        for o, resid, lse in outs:
            _evoattn.fwd(dims, x, k, v, bias, mask, o, resid, lse, 0.0, st)
            if wait:
                torch.cuda.synchronize()
            x = o
        torch.cuda.synchronize()
        return outs

    for got, want in zip(run(False), run(True)):
        assert all(torch.isfinite(t).all() for t in want)
        assert all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("B,S,N,H,D", [
    (2, 1, 128, 4, 64),      # one S row: forward, prep, dQ/dK/dV
    (2, 8, 64, 2, 32),       # one tile: no finish kernel
    (1, 6, 200, 4, 32),      # segments: the finish kernel is ahead of the next forward
    (1, 40, 200, 4, 64),     # whole pairs and segments
    (1, 150, 136, 2, 16),
    (1, 5, 256, 2, 128),
])
def test_steps_without_a_wait(B, S, N, H, D):
    import _evoattn
    q0, k0, v, d_o, bias, mask = _given(B, S, N, H, D, 3)
    dims, st = _evoattn.EvoDims(B, S, N, H, D), torch.cuda.current_stream().cuda_stream
    ws = torch.empty(_evoattn.bwd_workspace_bytes(dims), dtype=torch.uint8, device="cuda")
    phases = (_evoattn.BWD_PHASE_DBIAS, _evoattn.BWD_PHASE_DQKV)

    def run(calls):
        outs = [_outputs(q0, 5) + [torch.full((B, S, H, N), float("nan"), device="cuda"), torch.full((B, H, N, N), float("nan"), device="cuda")]
                for _ in range(8)]
        ws.fill_(0x7f)
        q, k = q0, k0
        torch.cuda.synchronize()
        for o, resid, dq, dk, dv, lse, dbias in outs:
            _evoattn.fwd(dims, q, k, v, bias, mask, o, resid, lse, 0.0, st)
            for ph in calls:
                if len(calls) > 1:
                    torch.cuda.synchronize()
                _evoattn.bwd_phased(dims, None, q, k, v, bias, mask, o, resid, lse, d_o, dq, dk, dv, dbias, ws, 0.0, ph, 0, st)
            if len(calls) > 1:
                torch.cuda.synchronize()
            q, k = dq, dk                # written by the last kernels of the step
        torch.cuda.synchronize()
        _evoattn.device_status()
        return outs

    for got, want in zip(run((phases[0] | phases[1],)), run(phases)):
        assert all(torch.isfinite(t).all() for t in want)
        for name, a, b in zip(("o", "o_resid", "dq", "dk", "dv", "lse"), got, want):
            assert torch.equal(a, b), name
        assert (got[-1] - want[-1]).abs().max() <= 1e-4 * want[-1].abs().max()


# ... through the operator, on new inputs, behind the kernels that make them; the other arm waits between forward and backward.  dQ and dBias:
# fp32 sums in arbitrary order of up to three kv tiles' and all rows' parts, a few units of 2^-24 of sums of absolute values within 2^6 of the results,
# and one rounding to bf16 (2^-8) of dQ.
@pytest.mark.parametrize("S,N,H,D,bias_type", [
    (1, 128, 4, 64, torch.bfloat16),
    (8, 64, 2, 32, torch.bfloat16),      # all five kernels: dBias converted by the finish kernel
    (6, 200, 4, 32, torch.float32),      # an fp32 bias, whose cast comes ahead of the forward
    (40, 200, 4, 64, torch.float32),
    (5, 264, 2, 128, torch.bfloat16),
])
def test_operator_steps_without_a_wait(S, N, H, D, bias_type):
    from tk_evo_attention_layer import TKEvoAttention
    gen = torch.Generator(device="cuda").manual_seed(3)

    def inputs():
        q, k, v, d_o = (torch.randn((2, S, N, H, D), generator=gen, device="cuda").mul(0.5).bfloat16() for _ in range(4))
        bias = torch.randn((2, 1, H, N, N), generator=gen, device="cuda").to(bias_type)
        mask = torch.where(torch.rand((2, S, 1, 1, N), generator=gen, device="cuda") < 0.9, 0.0, -1e9).to(bias_type)
        mask[..., 0] = 0
        return [t.requires_grad_() for t in (q, k, v)], mask, bias.requires_grad_(), d_o

    def step(x, wait):
        (q, k, v), mask, bias, d_o = x
        o = TKEvoAttention.apply(q, k, v, mask, bias)
        if wait:
            torch.cuda.synchronize()
        g = torch.autograd.grad(o, [q, k, v, bias], d_o)
        if wait:
            torch.cuda.synchronize()
        return [t.detach().clone() for t in (o, *g)]

    queued = [(x, step(x, False)) for x in (inputs() for _ in range(12))]
    torch.cuda.synchronize()
    for x, got in queued:
        want = step(x, True)
        for name, a, b in zip(("o", "dq", "dk", "dv", "dbias"), got, want):
            if name in ("o", "dk", "dv"):
                assert torch.equal(a, b), name
            else:
                a, b = a.float(), b.float()
                step_of = 2.0 ** -8 if name == "dq" or bias_type == torch.bfloat16 else 2.0 ** -16
                assert (a - b).abs().max() <= step_of * b.abs().max(), name
                assert (a - b).norm() <= 2.0 ** -10 * b.norm(), name
