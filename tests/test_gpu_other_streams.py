"""Kernels of another stream beside a step's: blocks of the step's next kernel must not queue for SMs ahead of them while the kernel before
still has most of its work to do.

A second stream of the same priority runs twelve elementwise kernels of 4 MB (some 3 us each, one SM's room short beside the step's kernels)
beside queued steps.  They get in where SMs become idle, between two kernels of a step: together they take 0.4 to 0.5 of a step's time.
With every kernel's successor queued from its start they took 1.25 to 2 times a step's.  The bound of one step lies between, a factor
of 1.25 and more from both."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,N,H,D", [(512, 384, 8, 32), (128, 1024, 4, 64), (64, 768, 4, 128)])
def test_another_streams_kernels_get_in(S, N, H, D):
    from tk_evo_attention_layer import TKEvoAttention

    def normal(*shape, std=1.0):
        return (torch.randn(shape, device="cuda") * std).bfloat16()

    q, k, v = (normal(1, S, N, H, D, std=0.5).requires_grad_() for _ in range(3))
    bias, mask, d_o = normal(1, 1, H, N, N).requires_grad_(), torch.zeros((1, S, 1, 1, N), device="cuda").bfloat16(), normal(1, S, N, H, D)
    src = torch.randn(1 << 20, device="cuda")
    dst = torch.empty_like(src)
    other = torch.cuda.Stream()

    def events(n):
        return [torch.cuda.Event(enable_timing=True) for _ in range(n)]

    def measure():
        steps, (e0, e1, f0, f1) = 6, events(4)
        torch.cuda.synchronize()
        torch.cuda._sleep(20_000_000)              # some 10 ms: all that follows is queued behind it
        e0.record()
        other.wait_event(e0)
        for _ in range(steps):
            torch.autograd.grad(TKEvoAttention.apply(q, k, v, mask, bias), [q, k, v, bias], d_o)
        e1.record()
        with torch.cuda.stream(other):
            f0.record()
            for _ in range(12):
                torch.mul(src, 1.5, out=dst)
            f1.record()
        torch.cuda.synchronize()
        return f0.elapsed_time(f1), e0.elapsed_time(e1) / steps

    measure()                                      # warm-up
    took = [measure() for _ in range(3)]
    foreign, step = (min(t[i] for t in took) for i in range(2))
    assert foreign < step, took
