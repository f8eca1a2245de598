"""The FP32 network at the edges of its tiles (32 and 64 pixels), of the rule
that picks one (128 pixels per SM), for every pattern of equal and different
albedo channels, and for feature rows that do not start on 16 bytes."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def sets(n, seed=11):
    rng = np.random.default_rng(seed)
    feat = np.concatenate([np.log1p(np.clip(rng.uniform(-0.2, 1.0, (n, 192)), 0, None)), rng.uniform(0, 1, (n, 192)),
                           np.log1p(2 * rng.uniform(0, 1, (n, 192)) ** 8)], axis=1).astype(np.float32)
    return feat, rng.uniform(0, np.pi, n).astype(np.float32)


def run(feat, gamma, sr, shift=0):
    import torch

    import mrpnn_b200 as M
    M.init()
    buf = torch.empty(feat.size + shift, device="cuda")
    t = buf[shift:].view(feat.shape[0], 576)
    t.copy_(torch.from_numpy(feat))
    g = torch.from_numpy(gamma).cuda()
    torch.cuda.synchronize()
    return M.predict_features(t, g, 0.857, sr).cpu().numpy()


# the network's contract against the oracle
RTOL, ATOL = 1e-4, 1e-6


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 64, 65, 127, 129, 300])
@pytest.mark.parametrize("sr", [(0.99, 0.99, 0.99), (0.99, 0.97, 0.93), (0.99, 0.99, 0.93), (0.99, 0.93, 0.99),
                                (0.93, 0.99, 0.99)])
def test_small(n, sr):
    feat, gamma = sets(n)
    np.testing.assert_allclose(run(feat, gamma, sr), O.mlp_f32(feat, gamma, 0.857, np.array(sr, np.float32)), rtol=RTOL,
                               atol=ATOL)


@pytest.mark.parametrize("sr", [(0.99, 0.99, 0.99), (0.99, 0.97, 0.93)])
def test_tiling_does_not_show(sr):
    """An output is its own sum whatever tile its pixel lies in: a large batch
    (64-pixel tiles) and its pieces (32-pixel tiles), rows on and off 16 bytes,
    give the same bits."""
    import torch
    n = 128 * torch.cuda.get_device_properties(0).multi_processor_count + 37
    feat, gamma = sets(n)
    whole = run(feat, gamma, sr)
    np.testing.assert_array_equal(run(feat, gamma, sr, shift=1), whole)
    for a, b in [(0, 1), (5, 70), (n - 37, n), (1000, 1999)]:
        np.testing.assert_array_equal(run(feat[a:b], gamma[a:b], sr), whole[a:b])
        np.testing.assert_array_equal(run(feat[a:b], gamma[a:b], sr, shift=3), whole[a:b])
    pick = np.linspace(0, n - 1, 200).astype(int)
    np.testing.assert_allclose(whole[pick], O.mlp_f32(feat[pick], gamma[pick], 0.857, np.array(sr, np.float32)),
                               rtol=RTOL, atol=ATOL)
