"""The spectrogram of 128 and 512 points: clips that end around a frame tile, steps and row widths that are odd,
batches whose clips are shorter than a CTA's run of tiles, both layouts; within 1e-5 of each frame's largest bin of
the FP64 oracle, nothing written outside the frames."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from gpu_util import SPEC_FRAME_REL, canvas, dev, frame_rel_err, host  # noqa: E402
from rpp_b200 import audio  # noqa: E402
from rpp_b200.types import RpptLayout, audio_desc, spectra_desc  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nft", [True, False])
@pytest.mark.parametrize("nfft,window,hop,center,power,clips", [
    (512, 400, 160, True, 2, 40), (512, 400, 161, True, 2, 12), (512, 511, 97, True, 1, 12), (512, 512, 512, False, 2, 12),
    (512, 64, 1, True, 2, 6), (128, 128, 32, True, 2, 12), (128, 99, 50, False, 1, 12), (512, 400, 160, True, 2, 700)])
def test_tiles(gpu, oracle, nfft, window, hop, center, power, clips, nft):
    r = np.random.default_rng(nfft + hop + clips)
    tile = 32 if nfft == 128 else 16
    frames = np.array([1, 2, tile - 1, tile, tile + 1, 2 * tile, 2 * tile + 1, 5 * tile + 3] * clips)[:clips]
    lens = np.maximum(1, (frames - 1) * hop + r.integers(0, hop, clips) + (0 if center else window)).astype(np.int32)
    if clips > 8:
        lens[8:11] = (0, 1, window - 1)
    L = int(lens.max()) + 3
    x = r.normal(0, 0.3, (clips, L)).astype(np.float32)
    ref = oracle.spectrogram_f64(x, lens, center, True, None, nfft, power, window, hop, nft)
    bins, F = nfft // 2 + 1, [max(0, oracle.num_windows(int(l), window, hop, center)) for l in lens]
    out = canvas(ref.shape)
    d = spectra_desc(clips, *ref.shape[1:], RpptLayout.NFT if nft else RpptLayout.NTF)
    assert audio.spectrogram(dev(x), audio_desc(clips, L), out, d, dev(lens), center, True, None, nfft, power, window, hop,
                             gpu) == 0
    got = host(out)
    for b in range(clips):
        g, e = (got[b], ref[b]) if nft else (got[b].T, ref[b].T)
        assert g.shape[0] == bins
        assert (g[:, F[b]:] == -12345.0).all()
        assert frame_rel_err(g[:, :F[b]], e[:, :F[b]]) <= SPEC_FRAME_REL
