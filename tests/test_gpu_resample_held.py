"""resample with 16-lobe windows: the kernel that holds a block's weights across the blocks that share them.  Bit
for bit the oracle's samples at the edges of its rule: rates with short, long and no phase period, ratios whose
span does and does not fit, clips that end around a block or an item, odd row widths, down-mixed channels."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from gpu_util import canvas, dev, host  # noqa: E402
from rpp_b200 import audio  # noqa: E402
from rpp_b200.types import audio_desc  # noqa: E402
from rpp_b200.windows import kaiser_sinc  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("channels", [1, 2, 3])
@pytest.mark.parametrize("rates", [(48000, 16000), (44100, 16000), (22050, 16000), (32000, 16000), (8000, 16000),
                                   (16000, 22050), (16000, 48000), (96000, 16000), (44100.5, 16000), (61440, 16000)])
def test_held_weights_equal_oracle(gpu, oracle, rates, channels):
    r = np.random.default_rng(int(rates[0]) + channels)
    ratio = rates[0] / rates[1]
    outs = [1, 255, 256, 257, 1279, 1281, 5 * 256 * 3 + 7, 30000]
    lens = np.array([max(1, int(o * ratio)) for o in outs], np.int32)
    n, L = len(lens), int(lens.max()) + 1   # rows of odd and even width over the rates
    x = r.normal(0, 0.3, (n, L * channels)).astype(np.float32)
    lut, scale, center, lobes = kaiser_sinc(16)
    ir, orr = np.full(n, rates[0], np.float32), np.full(n, rates[1], np.float32)
    width = int(np.ceil(L / ratio)) + 9
    ones = np.stack([lens, np.ones(n, np.int32)], 1).astype(np.int32)
    dims = np.stack([lens, np.full(n, channels, np.int32)], 1).astype(np.int32)
    mono = x
    if channels > 1:
        mono = np.zeros((n, L), np.float32)
        oracle.down_mixing(x, mono, dims.ravel(), False)
    ref = np.full((n, width), -12345.0, np.float32)
    oracle.resample(mono, ref, ir, orr, ones.ravel(), lut, scale, center, lobes)
    lut_d, xd, sd = dev(lut), dev(x), audio_desc(n, L, channels=channels, num_dims=3 if channels > 1 else 2)

    def call(w):
        out = canvas((n, w))
        if channels > 1:
            assert audio.downmix_resample(xd, sd, out, audio_desc(n, w), dev(ir), dev(orr), dev(dims), False, lut_d,
                                          scale, center, lobes, gpu) == 0
        else:
            win = audio.resampling_window(lut_d, scale, center, lobes)
            assert audio.resample(xd, sd, out, audio_desc(n, w), dev(ir), dev(orr), dev(dims), win, gpu) == 0
        return host(out)

    np.testing.assert_array_equal(call(width), ref)
    np.testing.assert_array_equal(call(1000), ref[:, :1000])   # rows too narrow for the longer clips
