"""Decode steps of latent attention whose sums come in many parts, most of them empty or all of them filled."""
import pytest
import torch

from tests import test_gpu_latent_steps as steps

pytestmark = pytest.mark.gpu


# (heads, dim, rot, vdim, rank, window), tokens; f32 caches and ranks beyond 512 go through one part a split
@pytest.mark.parametrize("shape,T", [((4, 64, 16, 40, 128, 5000), 40), ((4, 64, 16, 40, 128, 3000), 700), ((2, 40, 8, 24, 1000, 2100), 300), ((20, 24, 8, 33, 520, 700), 650)])
@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
def test_steps(gpu_ctx, shape, T, dt):
    steps.test_steps_behind_a_prompt(gpu_ctx, shape, T, dt)
