"""EVO_BWD_BESIDE_COPIES: how the first kernel of a backward is launched, not what it computes; the host-buffer path asks for it on both of its
loops."""
import pytest
import torch

from oracle import evo_ref


@pytest.mark.gpu
@pytest.mark.parametrize("S,N,D", [(6, 136, 32), (9, 64, 64), (4, 128, 128)])
def test_same_results(S, N, D):
    import _evoattn
    B, H = 1, 2
    q, k, v, mask, bias, d_o = (t.cuda().to(torch.bfloat16) for t in evo_ref.make_inputs(B, S, N, H, D, 0.5, 1.0, "bernoulli0.9", seed=S))
    st, dims = torch.cuda.current_stream().cuda_stream, _evoattn.EvoDims(B, S, N, H, D)
    o, res, lse = torch.empty_like(q), torch.empty_like(q), torch.empty((B, S, H, N), device="cuda")
    _evoattn.fwd(dims, q, k, v, bias, mask, o, res, lse, 0.0, st)
    ws = torch.empty(_evoattn.bwd_workspace_bytes(dims), dtype=torch.uint8, device="cuda")
    both, outs = _evoattn.BWD_PHASE_DBIAS | _evoattn.BWD_PHASE_DQKV, []
    for phases in (both, both | _evoattn.BWD_BESIDE_COPIES):
        out = [torch.full_like(q, float("nan")) for _ in range(3)] + [torch.full((B, H, N, N), float("nan"), device="cuda")]
        _evoattn.bwd_phased(dims, None, q, k, v, bias, mask, o, res, lse, d_o, *out, ws, 0.0, phases, 0, st)
        outs.append(out)
    _evoattn.device_status()
    for name, a, b in zip(("dq", "dk", "dv", "dbias"), *outs):
        # at most two partial sums of dQ: in either order; dBias: up to nine rows' fp32 terms in any order
        assert torch.equal(a, b) if name != "dbias" else (a - b).abs().max() <= 1e-6 * a.abs().max(), name


def test_python_chunks_ask_for_it(monkeypatch):
    import contextlib
    import tk_evo_attention_layer as L

    class Stream:
        cuda_stream = 0

        def wait_event(self, e):
            pass

    class Event:
        def record(self, s):
            pass

    eng = object.__new__(L.HostStreamedEvoAttention)
    S, N, H, D, bf = 3, 16, 1, 32, torch.bfloat16
    eng.s_in = eng.s_cmp = eng.s_out = Stream()
    eng.bias, eng.dbias = torch.zeros((1, H, N, N), dtype=bf), torch.zeros((1, H, N, N))
    names = ("q", "k", "v", "do", "o", "ores", "dq", "dk", "dv")
    one = {n: torch.zeros((1, S, N, H, D), dtype=bf) for n in names}
    one.update(mask=torch.zeros((1, S, N), dtype=bf), lse=torch.zeros((1, S, H, N)), dbias=torch.zeros((1, H, N, N)), ws=torch.zeros(1),
               ev_in=Event(), ev_cmp=Event(), ev_out=Event())
    eng.sets = [one] * 3
    phases = []
    monkeypatch.setattr(torch.cuda, "stream", lambda s: contextlib.nullcontext())
    monkeypatch.setattr(L._evoattn, "fwd", lambda *a: None)
    monkeypatch.setattr(L._evoattn, "bwd", lambda *a: phases.append(3))
    monkeypatch.setattr(L._evoattn, "bwd_phased", lambda *a: phases.append(a[-3]))
    acts = [torch.zeros((1, S, N, H, D), dtype=bf) for _ in range(4)]
    eng._run_chunks([(0, 0, 2), (0, 2, 1)], *acts[:3], torch.zeros((1, S, N), dtype=bf), acts[3], {n: torch.zeros((1, S, N, H, D), dtype=bf) for n in ("o", "dq", "dk", "dv")})
    assert phases == [7, 7]
