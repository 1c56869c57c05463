"""non_silent_region_detection decides from energy intervals and replays a reset block's float chain only where
they do not settle an end, and every block where intervals do not help: inputs at the edges of that rule, whole numbers
equal to the oracle's, and the replay of every block spread over the GPU."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from gpu_util import dev, host  # noqa: E402
from rpp_b200 import audio  # noqa: E402
from rpp_b200.types import audio_desc  # noqa: E402

pytestmark = pytest.mark.gpu


def clips(seed):
    """One clip per situation, of 3 samples to 41000, zero-padded into one batch."""
    r = np.random.default_rng(seed)
    noise = lambda n, a=0.3: r.normal(0, a, n).astype(np.float32)  # noqa: E731
    quiet_end = noise(30000)
    quiet_end[21000:] = 0.0                                  # the running sum decays to rounding residue
    quiet_begin = noise(30000)
    quiet_begin[:9000] = 0.0                                 # a whole silent reset block of 8192
    island = np.zeros(41000, np.float32)
    island[20000:20100] = noise(100)
    floor = noise(40000, 1e-3)                               # a floor 60 dB below the loud part, give or take
    floor[15000:25000] = noise(10000, 1.0)
    fade = (noise(40000) * np.exp(-np.arange(40000) / 2500.0)).astype(np.float32)
    gaps = noise(33000)
    for s in range(0, 33000, 6000):
        gaps[s:s + 3500] = 0.0
    flat = np.full(20000, 0.1, np.float32)                   # every full window ties with the maximum
    spike = np.zeros(10000, np.float32)
    spike[[0, 9999]] = 0.5, 0.7
    big = noise(9000)
    big[4000] = np.inf
    return [quiet_end, quiet_begin, island, floor, fade, gaps, flat, spike, big, noise(12000, 1e-21),
            np.zeros(5000, np.float32), noise(3), noise(63), noise(64), noise(65), noise(8192), noise(8193),
            noise(2048, 1e-6), np.zeros(0, np.float32), np.concatenate([noise(8192, 1e-4), noise(8192, 1.0), noise(9000, 1e-4)])]


@pytest.mark.parametrize("pad", [0, 3])
@pytest.mark.parametrize("reset,window,ref,cut", [
    (8192, 2048, 0.0, -60.0), (8192, 2048, 0.0, 0.0), (8192, 2048, 0.0, -0.05), (8192, 2048, 0.0, -120.0),
    (4096, 256, 0.0, -40.0), (4096, 255, 0.0, -40.0), (1000, 333, 0.0, -59.9), (64, 512, 0.0, -30.0),
    (63, 512, 0.0, -30.0), (-1, 2048, 0.0, -60.0), (100, 4096, 0.0, -80.0), (8192, 65536, 0.0, -20.0),
    (8192, 2048, 0.09, 0.0), (8192, 2048, 0.01, 0.0), (8192, 2048, -1.0, -20.0), (8192, 2048, 1e-30, -30.0)])
def test_region_equals_oracle(gpu, oracle, reset, window, ref, cut, pad):
    c = clips(5)
    lens = np.array([len(v) for v in c], np.int32)
    x = np.zeros((len(c), int(lens.max()) + pad), np.float32)   # pad 3: rows that are not 16-byte aligned
    for i, v in enumerate(c):
        x[i, :len(v)] = v
    with np.errstate(over="ignore", invalid="ignore"):
        b_ref, l_ref = oracle.nsr(x, lens, cut, window, ref, reset)
    begin = torch.full((len(lens),), -7, dtype=torch.int32, device="cuda")
    length = torch.full((len(lens),), -7, dtype=torch.int32, device="cuda")
    assert audio.non_silent_region_detection(dev(x), audio_desc(len(lens), x.shape[1]), dev(lens), begin, length, cut,
                                             window, ref, reset, gpu) == 0
    np.testing.assert_array_equal(host(begin), b_ref)
    np.testing.assert_array_equal(host(length), l_ref)


def detect(gpu, x, lens, window, reset, cut=-60.0, ref=0.0):
    """(begin, length) on the host, and a repeatable call."""
    begin = torch.full((len(lens),), -7, dtype=torch.int32, device="cuda")
    length = torch.full((len(lens),), -7, dtype=torch.int32, device="cuda")
    xd, ld, sd = dev(x), dev(lens), audio_desc(len(lens), x.shape[1])

    def call():
        assert audio.non_silent_region_detection(xd, sd, ld, begin, length, cut, window, ref, reset, gpu) == 0
    call()
    return host(begin), host(length), call


# 262144 samples: the prefix energies that a CTA holds in shared memory; 524288: the runs whose maxima it keeps
@pytest.mark.parametrize("reset,window,cut", [(8192, 2048, -60.0), (8192, 2048, 0.0), (8192, 2048, -0.02),
                                              (8192, 200, -60.0), (-1, 2048, -60.0), (50000, 2048, -60.0)])
def test_long_clips_equal_oracle(gpu, oracle, reset, window, cut):
    r = np.random.default_rng(11)
    lens = np.array([262143, 262144, 262145, 600000, 600001, 300], np.int32)
    x = np.zeros((len(lens), 600001), np.float32)
    for i, n in enumerate(lens):
        x[i, n // 9:n - n // 7] = r.normal(0, 0.1, n - n // 7 - n // 9)   # silence at both ends
    x[3, 540000:543000] *= 3.0                                           # the maximum past the kept runs
    x[4, 1000:] = 0.1 * np.sin(np.arange(599001) * 0.05)                 # a steady level: every block may hold it
    b_ref, l_ref = oracle.nsr(x, lens, cut, window, 0.0, reset)
    begin, length, _ = detect(gpu, x, lens, window, reset, cut)
    np.testing.assert_array_equal(begin, b_ref)
    np.testing.assert_array_equal(length, l_ref)


@pytest.mark.parametrize("reset,window,ref", [(8192, 100, 0.0), (8192, 3, 0.05), (32, 500, 0.0), (1, 2, 0.0)])
def test_many_clips_with_every_block_replayed(gpu, oracle, reset, window, ref):
    """More clips, and more blocks in a clip, than a CTA replays side by side; a clip with a NaN."""
    r = np.random.default_rng(12)
    n = 700
    lens = r.integers(1, 9000 if reset == 1 else 40000, n).astype(np.int32)
    x = np.zeros((n, int(lens.max())), np.float32)
    for i, k in enumerate(lens):
        x[i, k // 8:k - k // 6] = r.normal(0, 0.2, k - k // 6 - k // 8)
    x[6, lens[6] // 2] = np.nan
    with np.errstate(invalid="ignore"):
        b_ref, l_ref = oracle.nsr(x, lens, -60.0, window, ref, reset)
    begin, length, _ = detect(gpu, x, lens, window, reset, -60.0, ref)
    np.testing.assert_array_equal(begin, b_ref)
    np.testing.assert_array_equal(length, l_ref)


@pytest.mark.parametrize("scale", [1.0, 1e-18])   # 1e-18: intervals do not hold, every block is replayed
@pytest.mark.parametrize("cut", [-60.0, -0.01, 0.0])
@pytest.mark.parametrize("blocks", [7, 8])
def test_few_blocks(gpu, oracle, blocks, cut, scale):
    """As many reset blocks as the CTA of a clip replays itself, and one more."""
    r = np.random.default_rng(16)
    n, reset, window = 40, 700, 300
    width = blocks * reset
    lens = r.integers(width - 2 * reset, width + 1, n).astype(np.int32)
    lens[:2] = width, width - reset
    x = np.zeros((n, width), np.float32)
    for i, k in enumerate(lens):
        v = r.normal(0, 0.2, k) if i % 3 else 0.2 * np.sin(np.arange(k) * 0.03)
        v[k - 90 * (i % 5):] = 0.0
        x[i, :k] = v * scale
    b_ref, l_ref = oracle.nsr(x, lens, cut, window, 0.0, reset)
    begin, length, _ = detect(gpu, x, lens, window, reset, cut)
    np.testing.assert_array_equal(begin, b_ref)
    np.testing.assert_array_equal(length, l_ref)


@pytest.mark.parametrize("reset,window,top", [(8192, 2048, 9000), (8192, 512, 1500), (512, 300, 3000),
                                               (-1, 2048, 9000), (8192, 100, 2000), (30, 40, 900), (8192, 9000, 3000)])
@pytest.mark.parametrize("n", [1023, 1024, 1500])
def test_many_short_clips(gpu, oracle, n, reset, window, top):
    """Either side of the number of clips from which short ones have their moving mean squares stored."""
    r = np.random.default_rng(14)
    lens = r.integers(0, top + 1, n).astype(np.int32)
    x = np.zeros((n, top + 3), np.float32)
    for i, k in enumerate(lens):
        x[i, k // 8:k - k // 3] = r.normal(0, 0.2, k - k // 3 - k // 8)
    k = int(np.argmax(lens))
    x[k, lens[k] // 2] = np.nan
    x[k - 1, :] = np.where(np.arange(top + 3) == lens[k - 1] // 2, np.inf, x[k - 1])
    with np.errstate(invalid="ignore"):
        b_ref, l_ref = oracle.nsr(x, lens, -60.0, window, 0.0, reset)
    begin, length, _ = detect(gpu, x, lens, window, reset)
    np.testing.assert_array_equal(begin, b_ref)
    np.testing.assert_array_equal(length, l_ref)


def best_time(call):
    times = []
    for _ in range(7):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        call()
        b.record()
        b.synchronize()
        times.append(a.elapsed_time(b))
    return min(times)


def test_many_short_clips_are_spread_over_the_gpu(gpu):
    """16 times as many clips that end in silence, each replayed by a CTA of its own, take 10 times as long."""
    r = np.random.default_rng(15)
    lens = r.integers(2000, 4001, 8192).astype(np.int32)
    x = r.normal(0, 0.1, (8192, 4000)).astype(np.float32)
    x[np.arange(4000)[None] > lens[:, None] * 0.65] = 0.0
    few, many = detect(gpu, x[:512], lens[:512], 512, 8192)[2], detect(gpu, x, lens, 512, 8192)[2]
    assert best_time(many) < 5 * best_time(few)


def test_replay_of_every_block_is_spread_over_the_gpu(gpu):
    """A long clip with a window just below the intervals' range: its 586 blocks replayed one after the other, a few
    at a time, take some hundred times the call with a window just inside."""
    x = np.random.default_rng(13).normal(0, 0.1, (1, 4800000)).astype(np.float32)
    lens = np.array([4800000], np.int32)

    def best(window):
        return best_time(detect(gpu, x, lens, window, 8192)[2])

    assert best(255) < 8 * best(256)
