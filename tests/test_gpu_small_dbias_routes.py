"""dBias of small problems, whichever kernel forms it: a backward in one call may add it up in the dQ/dK/dV kernel, a backward in two phases takes
the dBias kernel."""
import pytest
import torch

from oracle import evo_ref

pytestmark = pytest.mark.gpu


def _one_call_and_phases(B, S, N, H, D, calls=1):
    """dBias, fp32, of `calls` backwards in one call and of one in two phases, on the same inputs."""
    import _evoattn
    q, k, v, mask, bias, d_o = (t.cuda().to(torch.bfloat16) for t in evo_ref.make_inputs(B, S, N, H, D, 0.5, 1.0, "bernoulli0.9", seed=N + S))
    st, dims = torch.cuda.current_stream().cuda_stream, _evoattn.EvoDims(B, S, N, H, D)
    o, res, lse = torch.empty_like(q), torch.empty_like(q), torch.empty((B, S, H, N), device="cuda")
    _evoattn.fwd(dims, q, k, v, bias, mask, o, res, lse, 0.0, st)
    ws = torch.empty(_evoattn.bwd_workspace_bytes(dims), dtype=torch.uint8, device="cuda")
    both = _evoattn.BWD_PHASE_DBIAS | _evoattn.BWD_PHASE_DQKV
    outs = []
    for phases in [(both,)] * calls + [(_evoattn.BWD_PHASE_DBIAS, _evoattn.BWD_PHASE_DQKV)]:
        dbias, grads = torch.full((B, H, N, N), float("nan"), device="cuda"), [torch.empty_like(q) for _ in range(3)]
        for ph in phases:
            _evoattn.bwd_phased(dims, None, q, k, v, bias, mask, o, res, lse, d_o, *grads, dbias, ws, 0.0, ph, 0, st)
        outs.append(dbias)
    _evoattn.device_status()
    return outs


@pytest.mark.parametrize("D", [16, 32, 64])
@pytest.mark.parametrize("B,S,N,H", [(1, 32, 64, 4), (1, 3, 128, 8), (2, 17, 40, 2), (4, 8, 128, 4), (1, 16, 256, 8), (1, 9, 200, 4), (1, 32, 128, 16), (1, 3, 256, 4), (1, 8, 392, 2), (1, 128, 128, 4)])
def test_one_call_equals_two_phases(B, S, N, H, D):
    """The same exponentials on both routes (at D <= 32 polynomials in the same columns, 7.5e-5 from the others): what is left are products
    and sums of up to 128 fp32 terms rounded in another order, below 128 * 2^-23 of the sum of their absolute values; at
    1e-5 of the largest entry with terms that hardly cancel in it."""
    one, two = _one_call_and_phases(B, S, N, H, D)
    assert (one - two).abs().max() <= 1e-5 * two.abs().max()


@pytest.mark.parametrize("D", [32, 64])
@pytest.mark.parametrize("B,S,N,H", [
    (8, 4, 128, 16),        # 128 tiles of dBias: a slice for each; four steps
    (8, 8, 128, 8),
    (1, 4, 512, 8),         # ... by segments at D = 64
    (1, 3, 768, 4),
    (2, 2, 136, 3),         # two slices: two terms onto zero, in either order
    (4, 3, 128, 16),
])
def test_few_slices_repeat(B, S, N, H, D):
    """Where the dBias kernel has a dBias tile's sum in one slice of S, or in two, dBias is the same bit for bit in every call,
    and in two phases."""
    *calls, phased = _one_call_and_phases(B, S, N, H, D, calls=4)
    for x in calls:
        assert torch.equal(x, phased)


@pytest.mark.parametrize("B,S,N,H,D,added", [
    (1, 32, 64, 4, 32, True), (1, 32, 64, 4, 64, True), (1, 3, 128, 8, 16, True),
    (1, 33, 64, 4, 32, False), (1, 33, 64, 4, 64, False), (1, 512, 40, 1, 64, False),       # rows that meet in a sum
    (1, 128, 128, 8, 64, True), (1, 100, 128, 2, 32, True), (1, 129, 128, 4, 64, False), (1, 64, 120, 2, 64, False),      # ... of whole tiles
    (1, 32, 128, 16, 32, True), (1, 30, 128, 20, 32, False),                                # four steps a CTA, five
    (1, 32, 128, 32, 64, True), (1, 32, 128, 33, 64, False),                                # seven, eight
    (1, 4, 512, 8, 64, False), (2, 2, 136, 3, 64, False),                                   # one slice, two
    (1, 9, 200, 4, 32, True), (1, 9, 200, 4, 64, True), (1, 8, 392, 2, 16, True), (1, 4, 640, 1, 32, False),      # by segments
    (1, 4, 128, 4, 128, False),
])
def test_which_kernel_forms_dbias(B, S, N, H, D, added):
    import _evoattn
    _evoattn.profile_enable(True)
    for k in range(3):
        _evoattn.profile_read(k)
    try:
        _one_call_and_phases(B, S, N, H, D)
    finally:
        _evoattn.profile_enable(False)
    launches = [_evoattn.profile_read(k)[1] for k in range(3)]
    assert launches == [1, 2, 1 if added else 2]              # (the phased call has one of its own)
