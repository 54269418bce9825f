"""Kernels of a step whose blocks may be placed before the kernel ahead of them has ended (programmatic launches).

Steps on new inputs are queued without a wait, each behind the torch kernels that write its inputs, and compared with the same steps
run one kernel's results at a time.  O, dK and dV are bit-reproducible; dQ and dBias are sums of fp32 partial sums in arbitrary order
of up to `rows` rows and two kv tiles: a few units of 2^-24 of sums of absolute values within 2^6 of the results, and one rounding to
bf16 (2^-8) of dQ.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,N,H,D,bias_type", [
    (1, 128, 4, 64, torch.bfloat16),     # one S row: forward, prep, dQ/dK/dV
    (8, 64, 2, 32, torch.bfloat16),      # all five kernels
    (6, 200, 4, 32, torch.float32),      # segments, and an fp32 bias, whose cast comes ahead of the forward
    (40, 200, 4, 64, torch.float32),     # whole pairs and segments
    (5, 264, 2, 128, torch.bfloat16),
])
def test_steps_without_a_wait(S, N, H, D, bias_type):
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
