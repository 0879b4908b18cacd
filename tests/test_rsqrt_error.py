"""The FP64 reciprocal root of the pair terms over (0, h^2], against a root in extended or quadruple precision: within the
1 ulp that CUDA documents for rsqrt(double), and closer in the mean than a rounded root and a rounded division."""
import numpy as np
import pytest


@pytest.mark.gpu
def test_rsqrt_against_a_longer_root():
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(5)
    h2 = float(np.float32(0.0457)) ** 2
    x = np.concatenate([h2 * rng.random(100_000), h2 * np.exp(-60 * rng.random(100_000))])
    got = torch.rsqrt(torch.from_numpy(x).cuda()).cpu().numpy()
    two = 1.0 / np.sqrt(x)
    ref = np.longdouble(1) / np.sqrt(x.astype(np.longdouble))
    ulp = np.spacing(ref.astype(np.float64)).astype(np.longdouble)
    err, err2 = ((abs(v.astype(np.longdouble) - ref) / ulp).astype(np.float64) for v in (got, two))
    assert err.max() <= 1.0
    assert np.sqrt(np.mean(err ** 2)) < np.sqrt(np.mean(err2 ** 2))
