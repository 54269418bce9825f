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


def _subclass(t):
    class Tagged(torch.Tensor):
        pass
    return t.as_subclass(Tagged)


def _transposed(t):
    return t.transpose(1, 2).contiguous().transpose(1, 2)


@pytest.mark.parametrize("name", ["q", "d_o", "o", "dv"])
@pytest.mark.parametrize("form,loop", [
    (lambda t: t, "native"),
    (lambda t: torch.cat([t, t])[1:], "native"),                     # at an offset of its storage
    (lambda t: torch.nn.Parameter(t, requires_grad=False), "native"),
    (_transposed, "python"),
    (lambda t: torch._neg_view(t), "python"),                        # its bytes have the other sign
    (_subclass, "python"),
    (lambda t: torch._efficientzerotensor(t.shape, dtype=t.dtype), "python"),      # has no bytes
    (lambda t: t.to("meta"), "python"),
], ids=["plain", "offset", "parameter", "transposed", "negated", "subclass", "zero", "meta"])
def test_form(monkeypatch, name, form, loop):
    x, out = _call()
    where = x if name in x else out
    where[name] = form(where[name])
    assert _loops(monkeypatch, x, out, types.SimpleNamespace(host_chunks=None)) == [loop]


@pytest.mark.parametrize("form", [lambda t: t.requires_grad_(), lambda t: t.float(), lambda t: t[:, :, :, :1].expand(t.shape)],
                         ids=["carries gradients", "fp32", "expanded"])
def test_form_of_a_result(monkeypatch, form):
    x, out = _call()
    out["dq"] = form(out["dq"])
    assert _loops(monkeypatch, x, out, types.SimpleNamespace(host_chunks=None)) == ["python"]


@pytest.mark.gpu
def test_on_the_device(monkeypatch):
    """With the extension that was built: contiguous tensors take the native loop, transposed and negated ones the Python loop, and
    the results are the same."""
    from tk_evo_attention_layer import HostStreamedEvoAttention as Host
    taken = []
    run_chunks = Host._run_chunks
    monkeypatch.setattr(Host, "_run_chunks", lambda self, *args: taken.append("python") or run_chunks(self, *args))
    outs = []
    for form, loops in ((lambda t: t, []), (_transposed, ["python"]), (lambda t: torch._neg_view(-t), ["python"])):
        x, out = _call()
        gen = torch.Generator().manual_seed(1)
        for n in ("q", "k", "v", "d_o"):
            x[n] = form(torch.randn((B, S, N, H, D), generator=gen).to(torch.bfloat16))
        taken.clear()
        Host("cuda").run(x["q"], x["k"], x["v"], x["mask"], x["bias"], x["d_o"], out)
        torch.cuda.synchronize()
        assert taken == loops
        outs.append(out)
    for other in outs[1:]:
        for n in ("o", "dq", "dk", "dv", "dbias"):       # (one tile, one chunk of three rows: dBias three fp32 terms in any order)
            a, b = outs[0][n], other[n]
            assert torch.equal(a, b) if n != "dbias" else (a - b).abs().max() <= 1e-6 * a.abs().max(), n
