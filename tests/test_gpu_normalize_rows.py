"""normalize per contiguous row (both statistics computed): row lengths at the edges of the halving tree's dealing
to lanes and of the one-pass kernel's range, against the oracle as in the general normalize test."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from gpu_util import dev, host  # noqa: E402
from rpp_b200 import audio  # noqa: E402
from rpp_b200.types import generic_desc  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cols", [1, 2, 31, 32, 33, 64, 65, 129, 511, 513, 544, 1025, 1601, 2049, 4096, 4097])
def test_rows_equal_oracle(gpu, oracle, cols):
    r = np.random.default_rng(cols)
    n, R = 5, 19
    src = (r.standard_normal((n, R, cols)) * 3 + 1).astype(np.float32)
    src[1, 2] = 0.5                                  # no variance
    roi = np.zeros((n, 4), np.uint32)
    roi[:, 2] = r.integers(1, R + 1, n)
    roi[:, 3] = r.integers((cols + 1) // 2, cols + 1, n)
    roi[0, 2:] = (R, cols)
    roi[4, 2] = 0                                    # no rows: zeros only
    size = int(roi[:, 2].max())
    mean, std = np.full(n * size, 3.0, np.float32), np.full(n * size, 4.0, np.float32)
    m_ref, s_ref = mean.copy(), std.copy()
    exp = np.full((n, R, cols), 7.0, np.float32)
    oracle.normalize_2d(src, exp, 2, m_ref, s_ref, 3, 1.5, 0.25, roi.ravel())
    d = generic_desc((n, R, cols))
    out = torch.full((n, R, cols), 7.0, device="cuda")
    m, s = dev(mean), dev(std)
    assert audio.normalize(dev(src), d, out, d, 2, m, s, 3, 1.5, 0.25, roi.ravel(), gpu) == 0
    np.testing.assert_allclose(host(out), exp, rtol=1e-5, atol=1e-5)
    np.testing.assert_array_equal(host(m), m_ref)
    np.testing.assert_allclose(host(s), s_ref, rtol=1e-6, atol=0)
    if cols <= 1025:                                 # in place
        a = dev(src)
        assert audio.normalize(a, d, a, d, 2, dev(mean), dev(std), 3, 1.5, 0.25, roi.ravel(), gpu) == 0
        np.testing.assert_array_equal(host(a), host(out))


def test_rows_past_the_destination_have_statistics(gpu, oracle):
    """A destination of fewer rows than the roi: its rows normalized, every roi row's statistics written."""
    r = np.random.default_rng(3)
    n, R, kept, cols = 3, 11, 7, 130
    src = (r.standard_normal((n, R, cols)) * 3 + 1).astype(np.float32)
    roi = np.zeros((n, 4), np.uint32)
    roi[:, 2], roi[:, 3] = R, cols
    m_ref, s_ref = np.zeros(n * R, np.float32), np.zeros(n * R, np.float32)
    exp = np.zeros((n, R, cols), np.float32)
    oracle.normalize_2d(src, exp, 2, m_ref, s_ref, 3, 1.0, 0.0, roi.ravel())
    out = torch.full((n, kept, cols), 7.0, device="cuda")
    m, s = torch.full((n * R,), 5.0, device="cuda"), torch.full((n * R,), 5.0, device="cuda")
    assert audio.normalize(dev(src), generic_desc((n, R, cols)), out, generic_desc((n, kept, cols)), 2, m, s, 3, 1.0,
                           0.0, roi.ravel(), gpu) == 0
    np.testing.assert_array_equal(host(m), m_ref)
    np.testing.assert_allclose(host(s), s_ref, rtol=1e-6, atol=0)
    np.testing.assert_allclose(host(out), exp[:, :kept], rtol=1e-5, atol=1e-5)
