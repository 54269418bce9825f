"""Logits at the ends of their range: rows, or leading tiles of rows, masked by large finite terms, by the type's lowest
value and by -inf; NaN and +inf in one place.  What is expected is the softmax in 64 bits on the rounded inputs."""
import pytest
import torch

from oracle import evo_ref
from _util import bf16_round

pytestmark = pytest.mark.gpu

# head dims of the three forward kernels; one tile, a ragged second one, three
SHAPES = [(N, D) for D in (16, 32, 64, 96, 128) for N in (64, 136, 264)]
B, S, H = 1, 4, 3


def _inputs(N, D):
    q, k, v, _, bias, _ = evo_ref.make_inputs(B, S, N, H, D, 1.0, 1.0, "valid", seed=N + D)
    return bf16_round(q, k, v, torch.zeros(B, S, 1, 1, N), bias)


def _out(q, k, v, mask, bias):
    from tk_evo_attention_layer import TKEvoAttention
    import _evoattn
    c = lambda t: t.cuda().to(torch.bfloat16)
    o = TKEvoAttention.apply(c(q), c(k), c(v), c(mask), c(bias)).float().cpu()
    _evoattn.device_status()
    return o


def _ref(q, k, v, mask, bias):
    # sums in fp32, where a term of -1e30 absorbs the logit it is added to, then 64 bits
    return evo_ref.evo_attention_ref(q, k, v, mask, bias).double()


def _close(o, ref):
    # a bf16 output with bf16 P against values of order one: two bf16 steps of the largest
    assert torch.isfinite(o).all()
    assert (o.double() - ref).abs().max() <= 2.0 ** -7 * max(1.0, ref.abs().max().item())


@pytest.mark.parametrize("N,D", SHAPES)
@pytest.mark.parametrize("low", [-1e10, -1e30, -1e36])
def test_masked_by_large_terms(N, D, low):
    """Every residue of a row masked: the mean of V; the first tile masked: the softmax over the rest.  Through the mask and
    through the pair bias."""
    q, k, v, mask, bias = _inputs(N, D)
    low = torch.tensor(low).to(torch.bfloat16).float().item()
    m = mask.clone()
    m[:, 0] = low                           # row 0: nothing left
    m[:, 1, ..., :min(N - 8, 128)] = low    # row 1: the first tile (or all but eight residues) masked
    o = _out(q, k, v, m, bias)
    _close(o, _ref(q, k, v, m, bias))
    b = bias.clone()
    b[..., 3, :] = low                      # query 3: nothing left
    b[..., 5, :min(N - 8, 128)] = low
    o = _out(q, k, v, mask, b)
    _close(o, _ref(q, k, v, mask, b))


@pytest.mark.parametrize("N,D", SHAPES)
@pytest.mark.parametrize("low", [-1e38, -2e38, torch.finfo(torch.bfloat16).min])
def test_masked_by_lowest(N, D, low):
    """The padding of a ragged tile ranks below every finite mask: a row masked as far as bf16 goes is the mean of its N values."""
    q, k, v, mask, bias = _inputs(N, D)
    m = mask.clone()
    m[:, 0] = torch.tensor(low).to(torch.bfloat16).float()
    o = _out(q, k, v, m, torch.zeros_like(bias))
    _close(o[:, 0], v[:, 0].double().mean(1, keepdim=True).expand(B, N, H, D))
    _close(o[:, 1:], _ref(q, k, v, mask, torch.zeros_like(bias))[:, 1:])


@pytest.mark.parametrize("N,D", SHAPES)
def test_masked_by_infinity(N, D):
    """-inf in the mask or the pair bias: excluded; a row or query with nothing else has no softmax and is NaN, no other is."""
    q, k, v, mask, bias = _inputs(N, D)
    ninf = float("-inf")
    m = mask.clone()
    m[:, 0] = ninf
    m[:, 1, ..., :min(N - 8, 128)] = ninf
    b = bias.clone()
    b[..., 3, :] = ninf
    b[..., 5, :min(N - 8, 128)] = ninf
    ref = _ref(q, k, v, m, b)
    gone = ref.isnan()
    assert gone[:, 0].all() and gone[:, :, 3].all() and not gone[:, 1:, 5].any()
    o = _out(q, k, v, m, b)
    assert torch.equal(o.isnan(), gone)
    _close(o[~gone], ref[~gone])


@pytest.mark.parametrize("N,D", SHAPES)
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_nan_and_inf_show(N, D, bad):
    """One NaN or +inf in the pair bias (any column residue mod 8, as pairs of columns take different routes through the exponential),
    in the mask or in K makes NaN of the queries that see it, and of no other."""
    q, k, v, mask, bias = _inputs(N, D)
    b = bias.clone()
    for c in range(8):
        b[:, :, :, 2 * c, N - 8 + c] = bad      # query 2 c, in the last tile
        b[:, :, :, 2 * c + 17, c] = bad         # ... in the first
    o = _out(q, k, v, mask, b)
    hit = sorted([2 * c for c in range(8)] + [2 * c + 17 for c in range(8)])
    assert o[:, :, hit].isnan().all()
    rest = [i for i in range(N) if i not in hit]
    _close(o[:, :, rest], _ref(q, k, v, mask, bias)[:, :, rest])
    for c in (0, 6):
        m = mask.clone()
        m[:, 2, ..., N - 8 + c] = bad
        o = _out(q, k, v, m, bias)
        assert o[:, 2].isnan().all() and torch.isfinite(o[:, :2]).all() and torch.isfinite(o[:, 3:]).all()
    k2 = k.clone()
    k2[:, 1, 7, 1, 3] = float("nan")
    o = _out(q, k2, v, mask, bias)
    assert o[:, 1, :, 1].isnan().all() and torch.isfinite(o[:, 0]).all() and torch.isfinite(o[:, 1, :, 0]).all()
