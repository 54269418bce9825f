"""What the operator shares with other torch operators besides its values: fresh inputs, autograd's edges, other modes."""
import pytest
import torch

pytestmark = pytest.mark.gpu

B, S, N, H, D = 1, 4, 64, 2, 32
# the second head dim is padded by the layer and takes the Python host path
HEAD_DIMS = (32, 24)


def _inputs(d=D, seed=3):
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda *s: torch.randn(s, generator=g, device="cuda").to(torch.bfloat16)
    return r(B, S, N, H, d), r(B, S, N, H, d), r(B, S, N, H, d), torch.zeros(B, S, 1, 1, N, device="cuda"), r(B, 1, H, N, N)


def _apply(*a):
    from tk_evo_attention_layer import TKEvoAttention
    return TKEvoAttention.apply(*a)


@pytest.mark.parametrize("d", HEAD_DIMS)
def test_fp32_bias_is_read_anew(d):
    """A pair bias of another type is cast on every call: after a write that bumps no version counter, in inference mode, on
    another stream than that of an earlier call, and in a CUDA graph."""
    q, k, v, m, b = _inputs(d)
    b2 = _inputs(d, seed=4)[4]
    want, want2 = _apply(q, k, v, m, b), _apply(q, k, v, m, b2)
    assert not torch.equal(want, want2)
    f = b.float()
    assert torch.equal(_apply(q, k, v, m, f), want)
    f.data.copy_(b2)
    assert torch.equal(_apply(q, k, v, m, f), want2)
    with torch.inference_mode():
        assert torch.equal(_apply(q, k, v, m, b.float()), want)
    # the copy of the first call is still in the making when the second stream reads the same tensor
    f.copy_(b)
    one, two = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(one):
        torch.cuda._sleep(20_000_000)
        o1 = _apply(q, k, v, m, f)
    with torch.cuda.stream(two):
        o2 = _apply(q, k, v, m, f)
    torch.cuda.synchronize()
    assert torch.equal(o1, want) and torch.equal(o2, want)
    # captured: a replay reads the bias that is there then, and an eager call after the capture does not read the graph's
    g = torch.cuda.CUDAGraph()
    with torch.no_grad(), torch.cuda.graph(g):
        o = _apply(q, k, v, m, f)
    assert torch.equal(_apply(q, k, v, m, f), want)
    f.copy_(b2)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(o, want2)
    del g


@pytest.mark.parametrize("d", HEAD_DIMS)
@pytest.mark.parametrize("which", range(5))
def test_one_input_requires_grad(d, which):
    """Any one input that requires a gradient puts the output on the graph, with an edge per argument in the arguments'
    order; the mask's gets nothing."""
    x = list(_inputs(d))
    x[which] = x[which].requires_grad_(True)
    o = _apply(*x)
    assert o.requires_grad
    edges = [f is not None for f, _ in o.grad_fn.next_functions]
    assert edges == [i == which for i in range(5)]
    o.float().sum().backward()
    assert (x[which].grad is None) == (which == 3)


def test_gate_edge():
    x = list(_inputs())
    gate = torch.randn_like(x[0]).requires_grad_(True)
    o = _apply(*x, None, gate)
    assert [f is not None for f, _ in o.grad_fn.next_functions] == [False] * 6 + [True]
    o.float().sum().backward()
    assert gate.grad.shape == gate.shape


@pytest.mark.parametrize("d", HEAD_DIMS)
@pytest.mark.parametrize("which", range(5))
def test_forward_mode_is_refused(d, which):
    """There is no forward-mode derivative: a tangent is an error, not dropped."""
    import torch.autograd.forward_ad as fwad
    x = list(_inputs(d))
    with fwad.dual_level():
        x[which] = fwad.make_dual(x[which], torch.ones_like(x[which]))
        with pytest.raises(NotImplementedError):
            _apply(*x)


@pytest.mark.filterwarnings("ignore")
@pytest.mark.parametrize("d", HEAD_DIMS)
def test_jit_trace_records_the_operator(d):
    """A traced function computes on its own inputs, gradients included, not on those it was traced with."""
    q, k, v, m, b = _inputs(d)
    f = lambda *x: _apply(*x) * 1.0
    q1, q2 = q.clone().requires_grad_(True), (2 * q).requires_grad_(True)
    traced = torch.jit.trace(f, (q1, k, v, m, b), check_trace=False)
    o, want = traced(q2, k, v, m, b), f(q2, k, v, m, b)
    assert torch.equal(o, want)
    d_o = torch.randn_like(o)
    assert torch.equal(torch.autograd.grad(o, q2, d_o)[0], torch.autograd.grad(want, q2, d_o)[0])


@pytest.mark.parametrize("d", HEAD_DIMS)
def test_function_transforms_are_refused(d):
    """vmap and grad of torch.func are errors, whether or not they are over one of the operator's inputs."""
    q, k, v, m, b = _inputs(d)
    two = torch.stack([q, q])
    for call in (lambda: torch.func.vmap(lambda x: _apply(x, k, v, m, b))(two),
                 lambda: torch.func.vmap(lambda x: _apply(q, k, v, m, b) + x)(two),
                 lambda: torch.func.grad(lambda x: _apply(x, k, v, m, b).float().sum())(q),
                 lambda: torch.func.grad(lambda x: (_apply(q, k, v, m, b) * x).float().sum())(q)):
        with pytest.raises(RuntimeError, match="setup_context"):
            call()


def _off_by_one(t):
    """The same values two (or four) bytes off the alignment."""
    room = torch.empty(t.numel() + 1, dtype=t.dtype, device="cuda")
    return room[1:].view(t.shape).copy_(t)


@pytest.mark.parametrize("route", ["native", "python"])
@pytest.mark.parametrize("view", ["plain", "ending", "fused"])
@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("back", [lambda t: t.cuda(), _off_by_one])
def test_saved_tensor_hooks(route, view, gated, back):
    """Saved tensors that come back from a hook contiguous where they were views, or misaligned, give the same gradients."""
    from tk_evo_attention_layer import TKEvoAttention
    q, k, v, m, b = _inputs()
    if view == "fused":
        q, k, v = torch.stack([q, k, v], 3).unbind(3)
    elif view == "ending":
        q, k, v = (t.transpose(1, 2).contiguous().transpose(1, 2) for t in (q, k, v))
    x = [t.detach().requires_grad_(True) for t in (q, k, v, b)]
    gate = (q * 2).detach().requires_grad_(True) if gated else None
    d_o = torch.randn(q.shape, generator=torch.Generator(device="cuda").manual_seed(9), device="cuda").to(torch.bfloat16)
    call = TKEvoAttention.apply if route == "native" else super(TKEvoAttention, TKEvoAttention).apply

    def grads():
        o = call(x[0], x[1], x[2], m, x[3], None, gate) if gated else call(x[0], x[1], x[2], m, x[3])
        return o, torch.autograd.grad(o, x + ([gate] if gated else []), d_o)

    o, want = grads()
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t.cpu().contiguous(), back):
        o2, got = grads()
    assert torch.equal(o, o2)
    for i, (a, c) in enumerate(zip(want, got)):
        if i == 3:      # sums over slices of S meet in any order
            assert (a.float() - c.float()).abs().max() <= 2.0 ** -7 * a.float().abs().max()
        else:
            assert torch.equal(a, c), i


def test_saved_tensor_of_another_size_is_an_error():
    q, k, v, m, b = _inputs()
    q.requires_grad_(True)
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, lambda t: t[..., :8] if t.dim() == 5 else t):
        o = _apply(q, k, v, m, b)
    with pytest.raises(RuntimeError, match="another"):
        o.sum().backward()


def test_without_the_native_host_path(monkeypatch):
    import sys
    import tk_evo_attention_layer as L
    x = _inputs()
    want = _apply(*x)
    monkeypatch.setattr(L, "_native_apply", None)
    monkeypatch.setitem(sys.modules, "_evo_torch", None)
    with pytest.warns(RuntimeWarning, match="build.py"):
        assert torch.equal(_apply(*x), want)
