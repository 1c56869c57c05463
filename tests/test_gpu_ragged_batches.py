"""The work list of uneven batches at batch sizes around a warp, a block and several clips per thread: pre-emphasis of
whole numbers by one half is exact in float32, so every sample is checked for equality."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from gpu_util import dev, host  # noqa: E402
from rpp_b200 import audio  # noqa: E402
from rpp_b200.types import RpptAudioBorderType, audio_desc  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("clips", [1, 31, 32, 33, 65, 511, 512, 1023, 1024, 1025, 2049, 5000])
def test_work_list(gpu, clips):
    r = np.random.default_rng(clips)
    lens = r.integers(0, 9000 if clips < 1000 else 3000, clips).astype(np.int32)
    lens[r.integers(0, clips, clips // 5)] = 0
    lens[-1] = 17   # the last clip's chunk is the list's last unit
    L = int(lens.max())
    x = r.integers(-1000, 1000, (clips, L)).astype(np.float32)
    want = x.copy()
    want[:, 1:] -= 0.5 * x[:, :-1]
    out = torch.full((clips, L), -12345.0, device="cuda")
    coeff = torch.full((clips,), 0.5, device="cuda")
    d = audio_desc(clips, L)
    assert audio.pre_emphasis_filter(dev(x), d, out, d, dev(lens), coeff, RpptAudioBorderType.ZERO, gpu) == 0
    want[np.arange(L) >= np.maximum(lens, 1)[:, None]] = -12345.0   # an empty clip's first sample is written, as in the reference
    assert np.array_equal(host(out), want)
