"""Which chunk loop a host-buffer call takes: the native one copies bytes of plain contiguous tensors in host memory, the Python one serves the
rest.  Streams and buffers of the device are stood in for on the CPU; the last test asks the operator as it is."""
import contextlib
import sys
import types

import pytest
import torch

B, S, N, H, D = 1, 3, 16, 2, 32


class Stream:
    stream_id = device_index = device_type = 0

    def wait_stream(self, other):
        pass


def _call():
    bf = torch.bfloat16
    x = {n: torch.ones((B, S, N, H, D), dtype=bf) for n in ("q", "k", "v", "d_o")}
    x["mask"], x["bias"] = torch.zeros((B, S, 1, 1, N), dtype=bf), torch.zeros((B, 1, H, N, N), dtype=bf)
    out = {n: torch.zeros((B, S, N, H, D), dtype=bf) for n in ("o", "dq", "dk", "dv")}
    out["dbias"] = torch.zeros((B, 1, H, N, N))
    return x, out


def _loops(monkeypatch, x, out, module):
    """Names of the loops that a call takes with `module` loaded as _evo_torch."""
    import tk_evo_attention_layer as L
    taken = []

    class Engine(L.HostStreamedEvoAttention):
        def __init__(self):
            self.dev, self.chunk_rows, self.pg = torch.device("cpu"), 64, None
            self.s_in, self.s_cmp, self.s_out = Stream(), Stream(), Stream()

        def _buffers(self, B, N, H, D, R):
            self.bias, self.dbias = torch.zeros((B, H, N, N), dtype=torch.bfloat16), torch.zeros((B, H, N, N))
            self.sets = [{n: None for n in self.NAMES}] * 3

        def _run_chunks(self, *args):
            taken.append("python")

    if hasattr(module, "host_chunks"):
        module.host_chunks = lambda *args: taken.append("native") or (0, "")
    monkeypatch.setitem(sys.modules, "_evo_torch", module)
    monkeypatch.setattr(L, "_native", lambda: None)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda dev: Stream())
    monkeypatch.setattr(torch.cuda, "stream", lambda s: contextlib.nullcontext())
    Engine().run(x["q"], x["k"], x["v"], x["mask"], x["bias"], x["d_o"], out)
    return taken


@pytest.mark.parametrize("module,loop", [(types.SimpleNamespace(host_chunks=None), "native"), (types.SimpleNamespace(apply=None), "python"), (None, "python")],
                         ids=["built", "built from earlier sources", "not loaded"])
def test_module(monkeypatch, module, loop):
    assert _loops(monkeypatch, *_call(), module) == [loop]
