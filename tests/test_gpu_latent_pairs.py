"""Portions of prompts on the latent attention's tensor-core kernel: two rows an MMA (at most 8 heads), tiles copied ahead,
against the plain softmax."""
import pytest

import test_gpu_rigotar as rigotar

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rank, heads", [(256, 8), (256, 7), (192, 1), (512, 8), (64, 8), (256, 9), (256, 16)])
def test_portions_of_several_requests(rank, heads):
    rigotar.test_latent_attention_portions_of_several_requests(rank, heads)
