"""Programmatic launches in the orders of kernels that small problems leave out or bring in: the steps of test_gpu_chained_launches.py at shapes
on either side of the rules that choose the kernels."""
import pytest
import torch

import test_gpu_chained_launches as chained

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,N,H,D,bias_type", [          # (two batches)
    (40, 128, 8, 32, torch.bfloat16),      # all five kernels: dBias of several slices, converted by the finish kernel
    (40, 200, 4, 64, torch.bfloat16),
    (16, 128, 6, 32, torch.bfloat16),      # two steps a CTA: dBias added up by the dQ/dK/dV kernel, converted by the finish kernel
    (16, 128, 6, 64, torch.bfloat16),
    (8, 64, 2, 64, torch.bfloat16),        # one step: converted by the dQ/dK/dV kernel
    (1, 200, 4, 64, torch.bfloat16),       # one S row with its prep kernel: two tiles,
    (1, 128, 80, 32, torch.bfloat16),      # ... more pairs than SMs
    (1, 128, 80, 64, torch.float32),
])
def test_operator_steps_without_a_wait(S, N, H, D, bias_type):
    chained.test_operator_steps_without_a_wait(S, N, H, D, bias_type)


@pytest.mark.parametrize("B,S,N,H,D", [
    (2, 1, 200, 4, 64),      # forward, prep, dQ/dK/dV
    (2, 1, 128, 80, 32),
    (2, 16, 128, 6, 64),     # forward, prep, dQ/dK/dV with dBias
    (2, 40, 128, 8, 32),     # ... with the dBias kernel
])
def test_steps_without_a_wait(B, S, N, H, D):
    chained.test_steps_without_a_wait(B, S, N, H, D)
