"""How many kernels a forward and a backward launch, as the library counts them while profiling."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,S,N,H,D,bias_type,launches", [
    (1, 40, 256, 8, 32, torch.bfloat16, 5),      # forward, prep, dBias, dQ/dK/dV, conversion
    (1, 40, 256, 8, 128, torch.float32, 4),      # whole pairs, fp32 dBias: nothing to convert
    (1, 32, 64, 4, 32, torch.bfloat16, 3),       # dBias added up and converted by the dQ/dK/dV kernel
    (1, 30, 64, 8, 32, torch.bfloat16, 4),       # two steps a CTA: converted by a kernel of its own
    (1, 30, 64, 8, 32, torch.float32, 3),
    (2, 1, 128, 4, 64, torch.bfloat16, 2),       # one S row of one tile
    (2, 1, 200, 4, 64, torch.bfloat16, 4),       # two tiles: prep, dQ of two tiles converted
])
def test_launches_of_a_step(B, S, N, H, D, bias_type, launches):
    import _evoattn
    from tk_evo_attention_layer import TKEvoAttention
    gen = torch.Generator(device="cuda").manual_seed(1)
    q, k, v, d_o = (torch.randn((B, S, N, H, D), generator=gen, device="cuda").mul(0.5).bfloat16().requires_grad_() for _ in range(4))
    bias = torch.randn((B, 1, H, N, N), generator=gen, device="cuda").to(bias_type).requires_grad_()
    mask = torch.zeros((B, S, 1, 1, N), device="cuda")

    def step():
        torch.autograd.grad(TKEvoAttention.apply(q, k, v, mask, bias), [q, k, v, bias], d_o)

    _evoattn.profile_enable(True)
    for kernel in range(4):
        _evoattn.profile_read(kernel)
    try:
        step()
        step()
    finally:
        _evoattn.profile_enable(False)
    step()                                       # (not counted)
    main = sum(_evoattn.profile_read(kernel)[1] for kernel in range(3))
    assert _evoattn.profile_read(_evoattn.PROFILE_ALL) == (0.0, 2 * launches) and main <= 2 * launches
    assert _evoattn.profile_read(_evoattn.PROFILE_ALL) == (0.0, 0)
