"""Timing cases of the batched audio front end: the calls its users make, through rpp_b200.audio.

Each case is a batch of ragged clips and one call, or one short sequence of calls, on it.  Clip
lengths come from the case alone (uniform over [lo, hi] samples, seeded by "lengths"); samples come
from the caller's seed, with the signal model of rpp_b200.synth: three tones, Gaussian noise of
sigma 0.1 and, per clip, up to three silent spans.  Rows are `hi` samples wide, so an odd `hi` gives
rows that are not 16-byte aligned.  `exact` restates each path in 64 bits with torch.
"""
import math

import numpy as np
import torch

from rpp_b200 import audio, lib
from rpp_b200.types import RpptDataType, RpptLayout, audio_desc, frontend_params, generic_desc, spectra_desc
from rpp_b200.windows import kaiser_sinc

COEFF = 0.97
CUTOFF_DB, MULTIPLIER = -80.0, 10.0
LOBES = 16
RATES = (16000, 22050, 44100, 48000)
# transform length, window, step, mel filters, sample rate: the speech front end with its two filter
# counts, and windows of the whole transform at a quarter step
SHAPES = ((512, 400, 160, 128, 16000), (512, 400, 160, 80, 16000), (512, 512, 128, 128, 16000),
          (1024, 1024, 256, 128, 16000), (1024, 1024, 256, 80, 22050), (2048, 2048, 512, 128, 44100),
          (256, 256, 64, 40, 16000))


def _stft_case(kind, clips, lo, hi, shape=SHAPES[0], lengths=1, border=0, power=2, **more):
    nfft, window, step, mel, rate = shape
    return dict(kind=kind, clips=clips, lo=lo, hi=hi, lengths=lengths, nfft=nfft, window=window, step=step, mel=mel,
                rate=rate, border=border, power=power, **more)


def listed():
    return [
        # one utterance of a second, as an interactive recognizer sends it: launch latency
        _stft_case("frontend", 1, 16000, 16000) | {"name": "frontend_1"},
        # a small uneven batch with odd row widths and 80 filters, as a serving step or a validation batch has
        _stft_case("frontend", 37, 4801, 77777, SHAPES[1], 2) | {"name": "frontend_37_odd"},
        # the training batch of the benchmark: 256 clips of 1 to 16 s
        _stft_case("frontend", 256, 16000, 256000) | {"name": "frontend_256"},
        # fixed 10 s clips with the longer transform of the precision study
        _stft_case("frontend", 128, 160000, 160000, SHAPES[3]) | {"name": "frontend_1024_128"},
        # the drop-in path: the four separate calls on the training batch, every tensor kept
        _stft_case("chain", 256, 16000, 256000) | {"name": "chain_256"},
        # the spectrogram alone on 8 short clips: a small drop-in call
        _stft_case("spectrogram", 8, 16000, 60000, ntf=False) | {"name": "spectrogram_8"},
        # trimming: the non-silent region of every clip of the training batch
        dict(kind="silence", clips=256, lo=16000, hi=256000, lengths=1, name="silence_256"),
        # loading decoded WAV data: 16-bit PCM to float, the non-silent region, the trimmed clip
        dict(kind="ingest", clips=64, lo=16000, hi=256000, lengths=3, name="ingest_64"),
        # stereo clips of mixed rates to 16 kHz mono, then the front end with 80 filters
        dict(kind="multirate", clips=512, seconds=4.0, channels=2, lengths=4, name="multirate_512"),
        # mono clips to 16 kHz through the plain resampling call
        dict(kind="resample", clips=64, seconds=6.0, channels=1, lengths=5, name="resample_64"),
        # per-filter normalization over time of the training batch's decibels
        dict(kind="normalize", clips=256, lo=101, hi=1601, lengths=6, mel=128, name="normalize_256"),
        # the front end on the training batch in pinned host memory, result in host memory
        _stft_case("host", 256, 16000, 256000) | {"name": "host_256"},
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(("frontend", "frontend", "frontend", "chain", "spectrogram", "silence", "ingest", "multirate",
                       "resample", "normalize", "host"))
    lengths = rng.randrange(1000, 1000000)
    if kind in ("multirate", "resample"):
        return dict(kind=kind, clips=_log(rng, 1, 400 if kind == "multirate" else 200),
                    seconds=round(rng.uniform(1.0, 4.0), 3), channels=2 if kind == "multirate" else 1, lengths=lengths)
    if kind == "normalize":
        hi = _log(rng, 30, 1601)
        return dict(kind=kind, clips=_log(rng, 1, 256), lo=max(1, hi // rng.choice((1, 2, 10))), hi=hi,
                    lengths=lengths, mel=rng.choice((40, 80, 128)))
    hi = _log(rng, 8000, 256000)
    lo = max(1, hi // rng.choice((1, 2, 4, 16)))
    if kind in ("silence", "ingest"):
        return dict(kind=kind, clips=_log(rng, 1, 256 if kind == "silence" else 128), lo=lo, hi=hi, lengths=lengths)
    more = {"ntf": rng.random() < 0.5} if kind == "spectrogram" else {}
    return _stft_case(kind, _log(rng, 1, 160 if kind == "host" else 110), lo, hi, rng.choice(SHAPES), lengths,
                      rng.randrange(3), rng.choice((2, 2, 2, 1)), **more)


# ---------------------------------------------------------------- inputs

def _clips(case):
    """Per-clip input lengths, input rates and the row width in samples."""
    rng = np.random.Generator(np.random.PCG64(case["lengths"]))
    n = case["clips"]
    if "seconds" in case:
        dur = np.clip(rng.lognormal(math.log(case["seconds"]), 0.25, n), 0.5, 30.0)
        rates = rng.choice(np.array(RATES, np.float32), n)
        lens = np.maximum(1, (dur * rates).astype(np.int64)).astype(np.int32)
        return lens, rates, int(lens.max())
    lens = rng.integers(case["lo"], case["hi"] + 1, n).astype(np.int32)
    return lens, np.full(n, case.get("rate", 16000), np.float32), case["hi"]


def _resampled(lens, rates, out_rate=16000):
    """Output lengths in the float arithmetic that defines them."""
    r = np.float32(out_rate)
    return np.array([int(l) if q == r else int(np.ceil(np.float32(np.float32(l) * r) / q)) for l, q in zip(lens, rates)],
                    np.int32)


def _frames(case, lens):
    return (np.asarray(lens) // case["step"] + 1).astype(np.int32)


def _signal(lens, rates, width, channels, seed, gaps=True):
    """[n][width * channels] float32 on the GPU, zero past each clip's end."""
    dev = torch.device("cuda")
    g = torch.Generator(device=dev)
    g.manual_seed(int(seed))
    n = len(lens)
    x = torch.zeros((n, width, channels), device=dev)
    lens_d = torch.from_numpy(lens).to(dev)[:, None]
    rates_d = torch.from_numpy(rates).to(dev)[:, None]
    for c0 in range(0, n, 64):
        s = slice(c0, min(n, c0 + 64))
        k = s.stop - s.start
        at = torch.arange(width, device=dev)[None, :]
        t = at / rates_d[s]
        tones = torch.zeros((k, width), device=dev)
        for _ in range(3):
            f, a, p = (torch.rand((k, 1), device=dev, generator=g) for _ in range(3))
            tones += (0.05 + 0.45 * a) * torch.sin(2 * math.pi * ((100.0 + 5900.0 * f) * t + p))
        live = at < lens_d[s]
        if gaps:
            for i in range(3):
                start, length, has = (torch.rand((k, 1), device=dev, generator=g) for _ in range(3))
                first = start * lens_d[s]
                live = live & ~((has < 0.5) & (at >= first) & (at < first + (0.1 + 0.9 * length) * rates_d[s]))
        for c in range(channels):
            noise = torch.randn((k, width), device=dev, generator=g) * 0.1
            x[s, :, c] = torch.where(live, tones + noise, 0.0)
    return x.view(n, width * channels)


def _pairs(a, b):
    return torch.from_numpy(np.stack([np.broadcast_to(a, np.shape(b) or np.shape(a)),
                                      np.broadcast_to(b, np.shape(a) or np.shape(b))], 1).astype(np.int32)).cuda()


def _params(case):
    return frontend_params(nfft=case["nfft"], window_length=case["window"], window_step=case["step"],
                           num_filter=case["mel"], sample_rate=case["rate"], max_freq=case["rate"] / 2,
                           cut_off_db=CUTOFF_DB, multiplier=MULTIPLIER, border=case["border"], power=case["power"])


MULTIRATE = dict(nfft=512, window=400, step=160, mel=80, rate=16000, border=0, power=2)


def _input(case, seed):
    lens, rates, width = _clips(case)
    if case["kind"] == "ingest":
        x = _signal(lens, rates, width, 1, seed)
        return lens, rates, width, (x * 16384).round().clamp(-32768, 32767).to(torch.int16)
    if case["kind"] == "normalize":
        g = torch.Generator(device="cuda")
        g.manual_seed(int(seed))
        x = (torch.randn((len(lens), case["mel"], width), device="cuda", generator=g) * 15 - 40).clamp(-80, 0)
        return lens, rates, width, x
    return lens, rates, width, _signal(lens, rates, width, case.get("channels", 1), seed,
                                       gaps=case["kind"] not in ("multirate", "resample"))


def prepare(case, seed):
    kind = case["kind"]
    lens, rates, width, x = _input(case, seed)
    n = len(lens)
    s = dict(kind=kind, case=case, x=x, h=lib.Handle(n, torch.cuda.current_stream().cuda_stream),
             lens=torch.from_numpy(lens).cuda(), sd=audio_desc(n, width),
             coeff=torch.full((n,), COEFF, device="cuda"))
    if kind in ("frontend", "chain", "spectrogram", "host"):
        frames = _frames(case, lens)
        mf, bins = int(frames.max()), case["nfft"] // 2 + 1
        s.update(md=spectra_desc(n, case["mel"], mf), params=_params(case))
        if kind == "spectrogram":
            s["layout"] = RpptLayout.NTF if case["ntf"] else RpptLayout.NFT
            shape = (mf, bins) if case["ntf"] else (bins, mf)
            s.update(spec=torch.zeros((n,) + shape, device="cuda"), spd=spectra_desc(n, *shape, s["layout"]))
        elif kind == "host":
            s.update(x=x.cpu().pin_memory(), db=torch.zeros((n, case["mel"], mf)).pin_memory(),
                     lens=torch.from_numpy(lens).pin_memory(), coeff=torch.full((n,), COEFF).pin_memory())
        else:
            s["db"] = torch.zeros((n, case["mel"], mf), device="cuda")
        if kind == "chain":
            s.update(pre=torch.zeros_like(x), spec=torch.zeros((n, bins, mf), device="cuda"),
                     mel=torch.zeros((n, case["mel"], mf), device="cuda"), spd=spectra_desc(n, bins, mf),
                     dims=_pairs(bins, frames), patches=_pairs(frames, case["mel"]))
    if kind in ("silence", "ingest"):
        s.update(begin=torch.zeros(n, dtype=torch.int32, device="cuda"),
                 length=torch.zeros(n, dtype=torch.int32, device="cuda"))
    if kind == "ingest":
        pcm = audio_desc(n, width)
        pcm.dataType = RpptDataType.I16
        s.update(pcm=pcm, wave=torch.zeros((n, width), device="cuda"), cut=torch.zeros((n, width), device="cuda"),
                 gd=generic_desc((n, width)), fill=torch.zeros(1, device="cuda"), roi=_pairs(0, lens))
    if kind in ("multirate", "resample"):
        out = _resampled(lens, rates)
        lut, scale, center, lobes = kaiser_sinc(LOBES)
        ow = int(out.max())
        s.update(sd=audio_desc(n, width, channels=case["channels"], num_dims=3), od=audio_desc(n, ow),
                 mono=torch.zeros((n, ow), device="cuda"), dims=_pairs(lens, case["channels"]),
                 rates=torch.from_numpy(rates).cuda(), out_rates=torch.full((n,), 16000.0, device="cuda"),
                 lut=torch.from_numpy(lut).cuda(), table=(scale, center, lobes), lens=torch.from_numpy(out).cuda())
        if kind == "resample":
            s["win"] = audio.resampling_window(s["lut"], scale, center, lobes)
        else:
            mf = int(_frames(MULTIRATE, out).max())
            s.update(db=torch.zeros((n, MULTIRATE["mel"], mf), device="cuda"),
                     md=spectra_desc(n, MULTIRATE["mel"], mf), params=_params(MULTIRATE))
    if kind == "normalize":
        m = case["mel"]
        roi = np.stack([np.zeros(n), np.zeros(n), np.full(n, m), lens], 1).astype(np.int32)
        s.update(gd=generic_desc((n, m, width)), roi=torch.from_numpy(roi), y=torch.zeros_like(x),
                 mean=torch.zeros(n * m, device="cuda"), inv=torch.zeros(n * m, device="cuda"))
    return s


# ---------------------------------------------------------------- the calls

def _ok(status):
    if status != 0:
        raise RuntimeError(f"status {status}: {lib.last_error()}")


def run(s):
    kind, h, c = s["kind"], s["h"], s["case"]
    if kind == "frontend":
        _ok(audio.frontend(s["x"], s["sd"], s["db"], s["md"], s["lens"], s["coeff"], s["params"], h))
        return s["db"]
    if kind == "host":
        _ok(audio.frontend_host(s["x"], s["sd"], s["db"], s["md"], s["lens"], s["coeff"], s["params"], 0, h))
        return s["db"]
    if kind == "spectrogram":
        _ok(audio.spectrogram(s["x"], s["sd"], s["spec"], s["spd"], s["lens"], True, True, None, c["nfft"], c["power"],
                              c["window"], c["step"], h))
        return s["spec"]
    if kind == "chain":
        _ok(audio.pre_emphasis_filter(s["x"], s["sd"], s["pre"], s["sd"], s["lens"], s["coeff"], c["border"], h))
        _ok(audio.spectrogram(s["pre"], s["sd"], s["spec"], s["spd"], s["lens"], True, True, None, c["nfft"],
                              c["power"], c["window"], c["step"], h))
        _ok(audio.mel_filter_bank(s["spec"], s["spd"], s["mel"], s["md"], s["dims"], c["rate"] / 2, 0.0, 0, c["mel"],
                                  c["rate"], True, h))
        _ok(audio.to_decibels(s["mel"], s["md"], s["db"], s["md"], s["patches"], CUTOFF_DB, MULTIPLIER, 0.0, h))
        return {"pre": s["pre"], "spec": s["spec"], "mel": s["mel"], "db": s["db"]}
    if kind == "silence":
        _ok(audio.non_silent_region_detection(s["x"], s["sd"], s["lens"], s["begin"], s["length"], -60.0, 2048, 0.0,
                                              8192, h))
        return {"begin": s["begin"], "length": s["length"]}
    if kind == "ingest":
        _ok(audio.pcm16_to_f32(s["x"], s["pcm"], s["wave"], s["sd"], s["lens"], h))
        _ok(audio.non_silent_region_detection(s["wave"], s["sd"], s["lens"], s["begin"], s["length"], -60.0, 2048, 0.0,
                                              8192, h))
        _ok(audio.slice(s["wave"], s["gd"], s["cut"], s["gd"], s["begin"], s["length"], s["fill"], True, s["roi"], h))
        return {"wave": s["wave"], "begin": s["begin"], "length": s["length"], "cut": s["cut"]}
    if kind == "resample":
        _ok(audio.resample(s["x"], s["sd"], s["mono"], s["od"], s["rates"], s["out_rates"], s["dims"], s["win"], h))
        return s["mono"]
    if kind == "multirate":
        scale, center, lobes = s["table"]
        _ok(audio.downmix_resample(s["x"], s["sd"], s["mono"], s["od"], s["rates"], s["out_rates"], s["dims"], False,
                                   s["lut"], scale, center, lobes, h))
        _ok(audio.frontend(s["mono"], s["od"], s["db"], s["md"], s["lens"], s["coeff"], s["params"], h))
        return {"mono": s["mono"], "db": s["db"]}
    _ok(audio.normalize(s["x"], s["gd"], s["y"], s["gd"], 2, s["mean"], s["inv"], 3, 1.0, 0.0, s["roi"], h))
    return {"y": s["y"], "mean": s["mean"], "inv": s["inv"]}


# ---------------------------------------------------------------- what a pass cannot do without

def work(case):
    kind = case["kind"]
    lens, rates, _ = _clips(case)
    L = float(lens.astype(np.int64).sum())
    if kind in ("multirate", "resample"):
        out = _resampled(lens, rates).astype(np.int64)
        total, frames = float(out.sum()), float(_frames(MULTIRATE, out).sum())
        w = {"bytes": 4 * case["channels"] * L + 4 * total,
             "flops": 4.0 * LOBES * float(out[rates != 16000].sum()) + 2 * (case["channels"] - 1) * L}
        if kind == "multirate":
            w["bytes"] += 4 * MULTIRATE["mel"] * frames
            w["flops"] += 2 * total + frames * (2.5 * 512 * 9 + 512 + 4 * 257)
        return w
    if kind == "silence":
        return {"bytes": 4 * L, "flops": 3 * L}
    if kind == "ingest":
        return {"bytes": 2 * L + 4 * L + 4 * L, "flops": 4 * L}
    if kind == "normalize":
        return {"bytes": 8 * L * case["mel"], "flops": 6 * L * case["mel"]}
    F = float(_frames(case, lens).astype(np.int64).sum())
    nfft, mel = case["nfft"], case["mel"]
    bins = nfft // 2 + 1
    fft = 2.5 * nfft * math.log2(nfft) + case["window"] + 3 * bins
    if kind == "spectrogram":
        return {"bytes": 4 * L + 4 * bins * F, "flops": F * fft}
    flops = 2 * L + F * (fft + 4 * bins + 2 * mel)
    if kind == "chain":
        return {"bytes": 8 * L + 4 * F * (bins + 2 * mel), "flops": flops}
    return {"bytes": 4 * L + 4 * F * mel, "flops": flops}


# ---------------------------------------------------------------- the same in 64 bits

def _mel_matrix(mel, nfft, rate):
    fsp, log_hz, step_log = 200.0 / 3, 1000.0, math.log(6.4) / 27
    to_mel = lambda hz: hz / fsp if hz < log_hz else log_hz / fsp + math.log(hz / log_hz) / step_log  # noqa: E731
    to_hz = lambda m: m * fsp if m < log_hz / fsp else log_hz * math.exp(step_log * (m - log_hz / fsp))  # noqa: E731
    top = to_mel(rate / 2)
    edge = [to_hz(top * i / (mel + 1)) for i in range(mel + 2)]
    w = np.zeros((mel, nfft // 2 + 1))
    i = 0
    for k in range(nfft // 2):   # the bin at half the rate belongs to no filter
        f = k * rate / nfft
        while i <= mel and f >= edge[i + 1]:
            i += 1
        down = (edge[i + 1] - f) / (edge[i + 1] - edge[i])
        if i < mel:
            w[i, k] = (1 - down) * 2 / (edge[i + 2] - edge[i])
        if i > 0:
            w[i - 1, k] = down * 2 / (edge[i + 1] - edge[i - 1])
    return torch.from_numpy(w).cuda()


def _emphasize(x, border):
    first = {0: x.new_zeros(()), 1: x[0], 2: x[min(1, len(x) - 1)]}[border]
    return x - float(np.float32(COEFF)) * torch.cat([first.view(1), x[:-1]])


def _power(x, c, frames):
    W, nfft, L = c["window"], c["nfft"], len(x)
    at = torch.arange(frames, device="cuda")[:, None] * c["step"] - W // 2 + torch.arange(W, device="cuda")
    if L < 2:
        at = torch.zeros_like(at)
    else:
        at = at % (2 * (L - 1))
        at = torch.where(at < L, at, 2 * (L - 1) - at)
    t = torch.arange(W, device="cuda", dtype=torch.float64)
    z = torch.fft.rfft(x[at] * (0.5 * (1 - torch.cos(2 * math.pi * (t + 0.5) / W))), nfft)
    return (z.abs() if c["power"] == 1 else z.real ** 2 + z.imag ** 2).T


def _decibels(m):
    top = m.max()
    return MULTIPLIER * torch.log10((m / top if top != 0 else m).clamp(min=10.0 ** (CUTOFF_DB / MULTIPLIER)))


def _interpolate(x, ratio, count):
    """`count` samples of x at multiples of `ratio`, by the windowed-sinc table."""
    lut, scale, center, lobes = kaiser_sinc(LOBES)
    lut = torch.from_numpy(lut).cuda().double()
    pos = torch.arange(count, device="cuda", dtype=torch.float64) * ratio
    y = torch.zeros(count, device="cuda", dtype=torch.float64)
    for k in range(-lobes, lobes):
        l = torch.ceil(pos).long() + k
        p = (l - pos) * scale + center
        i = p.floor().clamp(0, len(lut) - 2).long()
        w = lut[i] + (p - i) * (lut[i + 1] - lut[i])
        y += torch.where((l >= 0) & (l < len(x)), x[l.clamp(0, len(x) - 1)] * w, 0.0)
    return y


def exact(case, seed):
    kind = case["kind"]
    if kind == "silence":
        return None   # whole numbers
    lens, rates, width, x = _input(case, seed)
    n = len(lens)
    zeros = lambda *shape: torch.zeros(shape, device="cuda", dtype=torch.float64)  # noqa: E731
    if kind == "ingest":
        wave = x.double() / 32768
        return {"wave": wave, "begin": None, "length": None, "cut": None}
    if kind == "normalize":
        y, mean, inv = zeros(*x.shape), zeros(n, case["mel"]), zeros(n, case["mel"])
        for b in range(n):
            v = x[b, :, :lens[b]].double()
            mean[b] = v.mean(1)
            var = (v - mean[b][:, None]).square().mean(1)
            inv[b] = torch.where(var > 0, var.rsqrt(), 0.0)
            y[b, :, :lens[b]] = (v - mean[b][:, None]) * inv[b][:, None]
        return {"y": y, "mean": mean.view(-1), "inv": inv.view(-1)}
    if kind in ("multirate", "resample"):
        out = _resampled(lens, rates)
        c, mono = MULTIRATE, zeros(n, int(out.max()))
        for b in range(n):
            v = x[b].view(-1, case["channels"])[:lens[b]].double().mean(1)
            mono[b, :out[b]] = v if rates[b] == 16000 else _interpolate(v, float(rates[b]) / 16000, int(out[b]))
        if kind == "resample":
            return mono
        signal, lens = mono, out
    else:
        c, signal = case, x
    frames = _frames(c, lens)
    mf, bins = int(frames.max()), c["nfft"] // 2 + 1
    weights = _mel_matrix(c["mel"], c["nfft"], c["rate"])
    chain = kind == "chain"
    pre = zeros(n, width) if chain else None
    spec = zeros(n, bins, mf) if kind in ("chain", "spectrogram") else None
    mel = zeros(n, c["mel"], mf) if chain else None
    db = zeros(n, c["mel"], mf)
    for b in range(n):
        v = signal[b, :lens[b]].double()
        if kind != "spectrogram":
            v = _emphasize(v, c["border"])
        p = _power(v, c, int(frames[b]))
        if spec is not None:
            spec[b, :, :frames[b]] = p
        if kind == "spectrogram":
            continue
        m = weights @ p
        db[b, :, :frames[b]] = _decibels(m)
        if chain:
            pre[b, :lens[b]], mel[b, :, :frames[b]] = v, m
    if kind == "spectrogram":
        return spec.transpose(1, 2).contiguous() if case["ntf"] else spec
    if chain:
        return {"pre": pre, "spec": spec, "mel": mel, "db": db}
    if kind == "multirate":
        return {"mono": mono, "db": db}
    return db.cpu() if kind == "host" else db
