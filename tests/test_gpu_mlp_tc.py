"""The tensor-core network's forms give the same bits: grey albedo (three tiles
in flight on an SM) and coloured (two, the tail once per channel), whatever
tile and round a feature set falls into, rows on and off 16-byte boundaries."""
import numpy as np
import pytest

from tests.test_gpu_mlp_fp32 import sets

pytestmark = pytest.mark.gpu


def run(feat, gamma, sr, precision, shift=0):
    import torch

    import mrpnn_b200 as M
    M.init()
    buf = torch.empty(feat.size + shift, device="cuda")
    t = buf[shift:].view(feat.shape[0], 576)
    t.copy_(torch.from_numpy(feat))
    g = torch.from_numpy(gamma).cuda()
    torch.cuda.synchronize()
    return M.predict_features(t, g, 0.857, sr, precision).cpu().numpy()


@pytest.mark.parametrize("precision", [1, 2])   # BF16, FP8
@pytest.mark.parametrize("n", [1, 127, 128, 129, 700, 148 * 3 * 128 + 129])
def test_forms_agree(n, precision):
    feat, gamma = sets(n)
    grey = run(feat, gamma, (0.99,) * 3, precision)
    assert np.isfinite(grey).all()
    np.testing.assert_array_equal(grey[:, 0], grey[:, 2])
    np.testing.assert_array_equal(run(feat, gamma, (0.99,) * 3, precision, shift=1), grey)
    a = run(feat, gamma, (0.99, 0.99, 0.93), precision)
    b = run(feat, gamma, (0.93, 0.97, 0.99), precision, shift=3)
    np.testing.assert_array_equal(a[:, :2], grey[:, :2])
    np.testing.assert_array_equal(b[:, 2], grey[:, 2])
    np.testing.assert_array_equal(a[:, 2], b[:, 0])
    k = n // 2
    np.testing.assert_array_equal(run(feat[k:], gamma[k:], (0.99,) * 3, precision), grey[k:])


@pytest.mark.parametrize("precision", [1, 2])   # BF16, FP8
def test_split_tiles_agree(precision):
    """Calls of no more tiles than SMs give a row three threads: the same bits
    as the same sets among more tiles."""
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    feat, gamma = sets(sms * 128 + 1)
    grey = run(feat, gamma, (0.97,) * 3, precision)
    for k in (1, 31, 128, 129, 300, sms * 128):
        np.testing.assert_array_equal(run(feat[:k], gamma[:k], (0.97,) * 3, precision), grey[:k])
    np.testing.assert_array_equal(run(feat[-77:], gamma[-77:], (0.97,) * 3, precision, shift=1), grey[-77:])
