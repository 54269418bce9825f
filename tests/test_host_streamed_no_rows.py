"""A host-buffer call without rows (a rank of a short batch): dBias is zero, and the all-reduce takes place, without which the other ranks
would wait.  Streams and buffers of the device are stood in for on the CPU; on a GPU the call is made as it is."""
import contextlib

import pytest
import torch

SHAPES = [(1, 0, 16, 2, 32), (0, 3, 16, 2, 32)]


def _inputs(B, S, N, H, D):
    bf = torch.bfloat16
    acts = [torch.zeros((B, S, N, H, D), dtype=bf) for _ in range(4)]
    out = {n: torch.zeros((B, S, N, H, D), dtype=bf) for n in ("o", "dq", "dk", "dv")}
    out["dbias"] = torch.full((B, 1, H, N, N), 7.0)
    return (*acts[:3], torch.zeros((B, S, 1, 1, N), dtype=bf), torch.zeros((B, 1, H, N, N), dtype=bf), acts[3], out)


@pytest.mark.parametrize("dims", SHAPES)
def test_reaches_the_all_reduce(monkeypatch, dims):
    import tk_evo_attention_layer as L

    class Stream:
        def wait_stream(self, other):
            pass

    class Engine(L.HostStreamedEvoAttention):
        def __init__(self):
            self.dev, self.chunk_rows, self.pg = torch.device("cpu"), 64, "a group"
            self.s_in, self.s_cmp, self.s_out = Stream(), Stream(), Stream()

        def _buffers(self, B, N, H, D, R):
            assert R >= 1
            self.bias, self.dbias = torch.zeros((B, H, N, N), dtype=torch.bfloat16), torch.full((B, H, N, N), 5.0)
            self.sets = []

    reduced = []
    monkeypatch.setattr(L, "_native", lambda: None)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda dev: Stream())
    monkeypatch.setattr(torch.cuda, "stream", lambda s: contextlib.nullcontext())
    monkeypatch.setattr(torch.distributed, "all_reduce", lambda t, group: reduced.append((t.shape, group)))
    *args, out = _inputs(*dims)
    Engine().run(*args, out)
    B, _, N, H, _ = dims
    assert reduced == [((B, H, N, N), "a group")]
    assert (out["dbias"] == 0).all()


@pytest.mark.gpu
@pytest.mark.parametrize("dims", SHAPES)
def test_on_the_device(dims):
    from tk_evo_attention_layer import HostStreamedEvoAttention
    *args, out = _inputs(*dims)
    HostStreamedEvoAttention("cuda").run(*args, out)
    torch.cuda.synchronize()
    assert (out["dbias"] == 0).all()
