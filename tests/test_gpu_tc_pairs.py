"""The pair of K = 16 steps and its commit, as the Aggregator's kernel issues it, against a host product.

Operands are whole numbers of at most 3, so every sum is exact in fp32.
"""
import numpy as np
import pytest
import torch

from hashpoint import native
from test_gpu_tc_forms import PLAIN, SW64, SW128, image, window_start

pytestmark = pytest.mark.gpu


def _images(a_form, a_k, b_form, b_k, seed):
    native.build_testing()
    L = native.testing_lib()
    rng = np.random.default_rng(seed)
    A, B = rng.integers(-3, 4, (128, a_k)).astype(np.float32), rng.integers(-3, 4, (256, b_k)).astype(np.float32)
    img = [torch.from_numpy(image(m, f, L.hp_tc_check_image_bytes(i))).cuda() for i, (m, f) in enumerate(((A, a_form), (B, b_form)))]
    return L, A, B, img


@pytest.mark.parametrize("accumulate", [0, 1])
@pytest.mark.parametrize("a_form,a_k,a_k0,b_form,b_k,b_k0", [
    (SW128, 320, 0, SW64, 32, 0), (SW128, 320, 32, SW64, 32, 0), (SW128, 320, 224, SW64, 32, 0), (SW64, 32, 0, SW64, 32, 0),
    (SW128, 320, 64, SW128, 64, 32)])
def test_pair_of_steps(a_form, a_k, a_k0, b_form, b_k, b_k0, accumulate):
    L, A, B, (a, b) = _images(a_form, a_k, b_form, b_k, a_k0 + accumulate)
    d = torch.empty(128, 256, dtype=torch.float32, device="cuda")
    rc = L.hp_tc_check_mma2(a.data_ptr(), b.data_ptr(), a_form, window_start(a_form, a_k0, 128), b_form,
                            window_start(b_form, b_k0, 256), accumulate, d.data_ptr(),
                            torch.cuda.current_stream().cuda_stream)
    native.check(rc, "hp_tc_check_mma2", L)
    want = A[:, a_k0:a_k0 + 32] @ B[:, b_k0:b_k0 + 32].T
    if accumulate:
        want = want + A[:, a_k0:a_k0 + 16] @ B[:, b_k0:b_k0 + 16].T
    assert np.array_equal(d.cpu().numpy(), want)


def test_pair_refuses_windows_beyond_a_row():
    L, _, _, (a, b) = _images(SW128, 64, SW64, 32, 0)
    d = torch.empty(128, 256, dtype=torch.float32, device="cuda")
    for a_form, a_off, b_form, b_off in ((SW128, 96, SW64, 0), (SW128, 0, SW64, 32), (PLAIN, 0, SW64, 0)):
        assert L.hp_tc_check_mma2(a.data_ptr(), b.data_ptr(), a_form, a_off, b_form, b_off, 0, d.data_ptr(), None) != 0
