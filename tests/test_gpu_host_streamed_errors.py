"""What the library refuses in a host-buffer call is an EvoAttnError with its code on both chunk loops, and the engine serves the next call."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _inputs(N, view, seed=1):
    B, S, H, D, bf = 1, 5, 2, 32, torch.bfloat16
    gen = torch.Generator().manual_seed(seed)
    q, k, v, d_o = (view(torch.randn((B, S, N, H, D), generator=gen).mul(0.5).to(bf)) for _ in range(4))
    out = {n: torch.zeros((B, S, N, H, D), dtype=bf) for n in ("o", "dq", "dk", "dv")}
    out["dbias"] = torch.zeros((B, 1, H, N, N))
    return (q, k, v, torch.zeros((B, S, 1, 1, N), dtype=bf), torch.randn((B, 1, H, N, N), generator=gen).to(bf), d_o), out


@pytest.mark.parametrize("view", [lambda t: t, lambda t: t.transpose(1, 2).contiguous().transpose(1, 2)], ids=["contiguous", "transposed"])
def test_code_of_a_refused_call(view):
    import _evoattn
    from tk_evo_attention_layer import HostStreamedEvoAttention
    eng = HostStreamedEvoAttention("cuda")
    args, out = _inputs(12, view)                       # not a multiple of 8
    with pytest.raises(_evoattn.EvoAttnError) as e:
        eng.run(*args, out)
    assert e.value.code == -1                           # EVO_ERR_BAD_DIMS
    torch.cuda.synchronize()
    args, out = _inputs(16, view)
    eng.run(*args, out)
    torch.cuda.synchronize()
    want = _inputs(16, view)[1]
    HostStreamedEvoAttention("cuda").run(*args, want)
    torch.cuda.synchronize()
    assert torch.equal(out["o"], want["o"]) and out["o"].abs().max() > 0
