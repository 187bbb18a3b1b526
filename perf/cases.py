"""The work that users have this library do, as measured cases.

A case is one call, or one round of calls, through the public C entry points
(``akvisqol_b200.native.lib``; ``native.Server`` for the request server), on
synthetic audio or speech of the shapes that ``bench.py``, the tests and the
request mix use. ``prepare`` holds what a program has before the call: the
signals (host arrays, or device tensors where the program keeps its audio
there), the pointer tables of the C call, the long-lived context, and, for
prepared references, their handle. ``run`` makes the call and copies the
results out. ``exact`` restates the whole model in 64-bit torch and numpy.

Results come back as the C struct's doubles; those of the ``fast`` form, whose
scores carry single precision, are kept as float32, as a program that stores
them would.
"""

import ctypes
import functools
import math
import os

import numpy as np
import torch

from akvisqol_b200 import native

RADIUS = 60
TIMES = ("ref_start", "ref_end", "deg_start", "deg_end")
PATCH_ROW = np.dtype([("similarity", "f8")] + [(t, "f8") for t in TIMES] + [("pointers", "u8", 3)])
FEATURES = ("fvnsim", "fvnsim10", "fstdnsim", "fvdegenergy")


# ---- the cases ------------------------------------------------------------
# what: "pair" (visqol_measure), "batch" (visqol_measure_batch), "device"
# (visqol_b200_measure_batch, signals in HBM), "prepared" (one reference
# prepared, many degraded signals in HBM), "grad"
# (visqol_b200_measure_batch_grad), "server" (requests to a warm server).
# A batch's lengths are log-uniform in [min_s, max_s] (equal where both agree).

def _case(name, what, mode, rate, form, pairs, min_s, max_s, pcm=True, pinned=False):
    return {"name": name, "what": what, "mode": mode, "rate": rate, "form": form, "pairs": pairs,
            "min_s": min_s, "max_s": max_s, "pcm": pcm, "pinned": pinned}


def listed():
    return [
        # the smallest call: one short utterance, default precision, host arrays
        _case("speech_pair", "pair", "speech", 16000, "exact", 1, 2.491, 2.491, pcm=False),
        # one clip from a script or a notebook: 10 s of decoded 16-bit audio, default precision
        _case("audio_pair", "pair", "audio", 48000, "exact", 1, 10.0, 10.0),
        # one clip that is on the GPU already (a codec's training loop checking a sample), low latency
        _case("audio_pair_device_fast", "device", "audio", 48000, "fast", 1, 6.37, 6.37, pcm=False),
        # a whole minute (the longest item of the request mix), float samples
        _case("audio_minute", "pair", "audio", 48000, "exact", 1, 60.0, 60.0, pcm=False),
        # a listening-test set of utterances, default precision, host arrays
        _case("speech_batch", "batch", "speech", 16000, "exact", 48, 2.0, 15.0, pcm=False),
        # utterances synthesised on the GPU, scored there
        _case("speech_batch_device", "device", "speech", 16000, "balanced", 64, 2.0, 15.0, pcm=False),
        # the benchmark's batch: 10 s clips in HBM, fast form
        _case("audio_batch_device_fast", "device", "audio", 48000, "fast", 64, 10.0, 10.0),
        # uneven clips in HBM, f64 with FMA
        _case("audio_uneven_device", "device", "audio", 48000, "balanced", 40, 3.0, 30.0, pcm=False),
        # a conformance set: 10 s clips in page-locked host memory, default precision
        _case("audio_batch", "batch", "audio", 48000, "exact", 32, 10.0, 10.0, pinned=True),
        # a codec sweep: one CD-rate reference, many encodes of it
        _case("codec_sweep", "prepared", "audio", 44100, "balanced", 24, 7.9, 7.9),
        # one step of perceptual fine-tuning: scores and gradients
        _case("gradients", "grad", "audio", 48000, "exact", 2, 2.2, 3.1, pcm=False),
        # a serving burst: audio and speech requests into a warm server
        _case("server_burst", "server", "mixed", 48000, "fast", 40, 2.0, 20.0),
    ]


def draw(rng):
    """One more case of the same ranges."""
    def log_uniform(a, b):
        return math.exp(rng.uniform(math.log(a), math.log(b)))

    what = rng.choice(["pair", "pair", "batch", "device", "device", "prepared", "grad", "server"])
    mode = "mixed" if what == "server" else rng.choice(["audio", "audio", "speech"])
    rate = 16000 if mode == "speech" else rng.choice([48000, 48000, 44100])
    form = rng.choice(["exact", "exact", "balanced", "fast"])
    pairs, top = 1, 60.0 if mode == "audio" else 20.0
    if what in ("batch", "device", "prepared"):
        pairs, top = int(round(log_uniform(1 if what == "device" else 2, 48))), 20.0
    elif what == "grad":
        pairs, top = rng.choice([1, 2]), 4.0
    elif what == "server":
        pairs, top, form = int(round(log_uniform(4, 40))), 20.0, rng.choice(["fast", "balanced"])
    a, b = sorted(round(log_uniform(2.0, top), 4) for _ in range(2))
    if pairs == 1 or what == "prepared":
        a = b
    case = _case("", what, mode, rate, form, pairs, a, b, pcm=rng.random() < 0.5,
                 pinned=what == "batch" and rng.random() < 0.3)
    del case["name"]
    return case


# ---- inputs ---------------------------------------------------------------

def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _pcm16(x):
    return torch.clamp(torch.round(x * 32768.0), -32768, 32767) / 32768.0


def _rand(g, n):
    return torch.rand(n, generator=g, device=g.device, dtype=torch.float64)


def _audio(g, n, rate):
    """Music-like: pink noise at -20 dBFS and six tones under a slow envelope."""
    dev = g.device
    spec = torch.fft.rfft(torch.randn(n, generator=g, device=dev, dtype=torch.float64))
    f = torch.arange(spec.numel(), device=dev, dtype=torch.float64).clamp(min=1.0)
    spec = spec / f.sqrt()
    spec[0] = 0.0
    x = torch.fft.irfft(spec, n)
    x = 0.1 * x / x.square().mean().sqrt()
    t = torch.arange(n, device=dev, dtype=torch.float64) / rate
    freqs = 100.0 * 120.0 ** _rand(g, 6)
    phase = 2.0 * math.pi * _rand(g, 6)
    tones = (0.08 * torch.sin(2.0 * math.pi * freqs[:, None] * t + phase[:, None])).sum(0)
    return x + (0.5 - 0.5 * torch.cos(8.0 * math.pi * t)) * tones


def _speech(g, n, rate):
    """Speech-like: harmonics of a drifting pitch under moving formants, in
    voiced runs with silences between them."""
    dev = g.device
    t = torch.arange(n, device=dev, dtype=torch.float64) / rate
    r = _rand(g, 4).tolist()
    drift = 2.0 * math.pi * (0.1 + 0.3 * r[0])
    pitch = 160.0 + 60.0 * torch.sin(drift * t + 6.28 * r[1])
    phase = 2.0 * math.pi * (160.0 * t + 60.0 / drift * (math.cos(6.28 * r[1]) - torch.cos(drift * t + 6.28 * r[1])))
    x = torch.zeros_like(t)
    for h in range(1, 28):
        f = h * pitch
        amp = 0.02 + sum(a / (1.0 + ((f - c * (1.0 + 0.3 * torch.sin(2.0 * math.pi * m * t + 6.28 * r[2]))) / w) ** 2)
                         for a, c, w, m in ((1.0, 500.0, 90.0, 1.7), (0.5, 1500.0, 140.0, 2.3), (0.3, 2800.0, 200.0, 1.1)))
        x += torch.where(f < 0.45 * rate, amp / h ** 0.5 * torch.sin(h * phase), torch.zeros_like(t))
    mask = torch.zeros_like(t)
    runs, pos, k = _rand(g, 256).tolist(), int((0.05 + 0.25 * r[3]) * rate), 0
    while pos < n:
        run = int((0.3 + 0.9 * runs[k % 256]) * rate)
        mask[pos:pos + run] = 1.0
        pos, k = pos + run + int((0.1 + 0.4 * runs[(k + 1) % 256]) * rate), k + 2
    x = x * mask
    return 0.3 * x / x.abs().max().clamp(min=1e-9)


def _degrade_audio(g, ref, rate, cutoff, snr_db, delay, slip):
    """Low-pass, noise, a delay in front, and for some clips a few samples
    more half way through; 16-bit, as a decoder writes it."""
    n = ref.numel()
    f = torch.fft.rfftfreq(n, 1.0 / rate, device=ref.device, dtype=torch.float64)
    y = torch.fft.irfft(torch.fft.rfft(ref) / torch.sqrt(1.0 + (f / cutoff) ** 8), n)
    noise = torch.randn(n, generator=g, device=ref.device, dtype=torch.float64)
    y = y + noise * y.square().mean().sqrt() * 10.0 ** (-snr_db / 20.0)
    zeros = functools.partial(torch.zeros, device=ref.device, dtype=torch.float64)
    return _pcm16(torch.cat([zeros(delay), y[:n // 2], zeros(slip), y[n // 2:]]))


def _degrade_speech(g, ref, rate, delay):
    """8-bit mu-law round trip, a delay, and 3% of 20 ms frames lost."""
    c = torch.sign(ref) * torch.log1p(255.0 * ref.abs()) / math.log1p(255.0)
    q = torch.round((c + 1.0) * 127.5) / 127.5 - 1.0
    y = torch.sign(q) * (256.0 ** q.abs() - 1.0) / 255.0
    frame = rate // 50
    lost = _rand(g, y.numel() // frame + 1) < 0.03
    y = y * (~lost).repeat_interleave(frame)[:y.numel()].to(y.dtype)
    return torch.cat([torch.zeros(delay, device=y.device, dtype=y.dtype), y])


def _shapes(case):
    """Per pair (mode, rate, reference samples, delay in seconds, slip): a
    batch's lengths are its own, whatever signals fill them."""
    u = np.random.RandomState(1000 + case["pairs"])
    lo, hi = case["min_s"], case["max_s"]
    for _ in range(case["pairs"]):
        seconds = lo if lo == hi else math.exp(u.uniform(math.log(lo), math.log(hi)))
        mode, rate = case["mode"], case["rate"]
        if mode == "mixed":  # the request mix: 70% audio, 30% speech
            mode, rate = ("audio", rate) if u.rand() < 0.7 else ("speech", 16000)
        yield mode, rate, int(round(seconds * rate)), u.uniform(0, 0.2), u.rand()


def _slots(case):
    """Rows kept for each pair's patches: the VAD and the alignment leave at most this many."""
    rows = []
    for mode, rate, n, _, _ in _shapes(case):
        window, hop = _geometry(rate)
        rows.append((1 + (n - window) // hop) // (30 if mode == "audio" else 20) + 1)
    return rows


def _signals(case, seed):
    """Per pair (mode, rate, ref, deg); a pure function of the case and the seed."""
    dev = _device()
    g = torch.Generator(device=dev)
    g.manual_seed((int(seed) * 1000003 + 17) % (1 << 62))
    u = np.random.RandomState(int(seed) % (1 << 31))
    pairs, ref = [], None
    for mode, rate, n, delay, slip in _shapes(case):
        cutoff, snr = u.uniform(4000, 16000), u.uniform(10, 40)
        if ref is None or case["what"] != "prepared":
            ref = _audio(g, n, rate) if mode == "audio" else _speech(g, n, rate)
            ref = _pcm16(ref) if case["pcm"] else ref
        if mode == "audio":
            deg = _degrade_audio(g, ref, rate, min(cutoff, 0.45 * rate), snr, int(delay * rate),
                                 int(3 + 20 * slip) if slip < 0.3 else 0)
        else:
            deg = _degrade_speech(g, ref, rate, int(0.1 * delay * rate))
        pairs.append((mode, rate, ref, deg))
    return pairs


# ---- the calls ------------------------------------------------------------

_MODES = {"audio": native.MODE_AUDIO, "speech": native.MODE_SPEECH}


def _check(code):
    if code != native.OK:
        raise native.error_for(code)


@functools.lru_cache(maxsize=None)
def _context(mode, form):
    """The program's long-lived context for this mode and form."""
    options = native.make_options(precision=form, mode=_MODES[mode], search_window_radius=RADIUS,
                                  use_lattice_model=False)
    handle = ctypes.c_void_p()
    _check(native.lib.visqol_create(ctypes.byref(options), ctypes.byref(handle)))
    return handle


@functools.lru_cache(maxsize=None)
def _server(form):
    return native.Server(precision=form)


class _PreparedRef:
    def __init__(self, context, ptrs, lens, rate):
        self.handle = ctypes.c_void_p()
        _check(native.lib.visqol_b200_prepare(context, 1, ptrs, lens, rate, native.DEVICE_INPUTS,
                                               ctypes.byref(self.handle)))

    def __del__(self):
        native.lib.visqol_b200_prepared_free(self.handle)


def prepare(case, seed):
    pairs = _signals(case, seed)
    what, n = case["what"], len(pairs)
    on_device = what in ("device", "prepared", "server")

    def hold(x):
        if on_device:
            return x.contiguous()
        x = x.cpu()
        return x.pin_memory().numpy() if case["pinned"] else x.numpy().copy()

    refs, degs = [hold(p[2]) for p in pairs], [hold(p[3]) for p in pairs]
    address = (lambda x: x.data_ptr()) if on_device else (lambda x: x.ctypes.data)
    state = {"what": what, "n": n, "refs": refs, "degs": degs, "rate": pairs[0][1],
             "first": np.concatenate([[0], np.cumsum(_slots(case))]), "nb": 32 if case["mode"] == "audio" else 21,
             "real": np.float32 if case["form"] == "fast" else np.float64,
             "modes": [p[0] for p in pairs], "rates": [p[1] for p in pairs]}
    table = lambda xs: (ctypes.c_void_p * len(xs))(*[address(x) for x in xs])  # noqa: E731
    lengths = lambda xs: (ctypes.c_size_t * len(xs))(*[len(x) for x in xs])  # noqa: E731
    state["r"], state["rl"], state["d"], state["dl"] = table(refs), lengths(refs), table(degs), lengths(degs)
    if on_device:
        torch.cuda.synchronize()
    if what == "server":
        state["server"] = _server(case["form"])
        return state
    state["context"] = _context(case["mode"], case["form"])
    state["out"] = (ctypes.POINTER(native.Result) * n)()
    state["status"] = (ctypes.c_int32 * n)()
    if what == "prepared":
        state["prepared"] = _PreparedRef(state["context"], state["r"], state["rl"], state["rate"])
        state["index"] = (ctypes.c_size_t * n)()
    if what == "grad":
        state["grads"] = [np.zeros(len(d)) for d in degs]
        state["g"] = (ctypes.c_void_p * n)(*[a.ctypes.data for a in state["grads"]])
    return state


def _collect(results, state):
    """The results' values as arrays, patches in their pairs' rows (zeros
    behind the last); the results are freed."""
    nb, real, first, read = state["nb"], state["real"], state["first"], ctypes.string_at
    scores, features = [], []
    patches = np.zeros(first[-1], PATCH_ROW)
    for i, p in enumerate(results):
        r = p.contents
        scores += (r.moslqo, r.vnsim, r.alignment_lag_s)
        features.append(b"".join(read(getattr(r, f), 8 * nb) for f in FEATURES))
        rows = np.frombuffer(read(r.patch_sims, PATCH_ROW.itemsize * r.num_patches), PATCH_ROW)
        patches[first[i]:first[i] + rows.size] = rows
        native.lib.visqol_result_free(p)
    scores = np.array(scores).reshape(-1, 3)
    features = np.frombuffer(b"".join(features)).reshape(-1, 4, nb)
    out = {"moslqo": scores[:, 0].astype(real), "vnsim": scores[:, 1].astype(real), "lag_s": scores[:, 2],
           "similarity": patches["similarity"].astype(real)}
    for k, f in enumerate(FEATURES):
        out[f] = features[:, k].astype(real)
    for t in TIMES:
        out[t] = patches[t].copy()
    return out


def run(state):
    lib, what, n = native.lib, state["what"], state["n"]
    if what == "server":
        return _serve(state)
    c, out, status = state["context"], state["out"], state["status"]
    r, rl, d, dl, rate = state["r"], state["rl"], state["d"], state["dl"], state["rate"]
    if what == "pair":
        D = ctypes.POINTER(ctypes.c_double)
        rc = lib.visqol_measure(c, ctypes.cast(r[0], D), rl[0], ctypes.cast(d[0], D), dl[0], rate, out)
    elif what == "batch":
        rc = lib.visqol_measure_batch(c, n, r, rl, d, dl, rate, 0, out, status)
    elif what == "device":
        rc = lib.visqol_b200_measure_batch(c, n, r, rl, d, dl, rate, native.DEVICE_INPUTS, out, status, None)
    elif what == "prepared":
        rc = lib.visqol_b200_measure_prepared(c, state["prepared"].handle, n, state["index"], d, dl,
                                              native.DEVICE_INPUTS, out, status)
    else:
        rc = lib.visqol_b200_measure_batch_grad(c, n, r, rl, d, dl, rate, 0, out, status, state["g"])
    _check(rc)
    got = _collect(out, state)
    if what == "grad":
        got["grad"] = np.concatenate(state["grads"])
    return got


def _serve(state):
    server, real = state["server"], state["real"]
    order = {}
    for i in range(state["n"]):
        ticket = server.submit(_MODES[state["modes"][i]], state["r"][i], state["d"][i], state["rates"][i],
                               device_inputs=True, ref_len=state["rl"][i], deg_len=state["dl"][i])
        order[ticket] = i
    got = [None] * state["n"]
    while order:
        ticket, code, result = server.next()
        _check(code)
        got[order.pop(ticket)] = result
    out = {"moslqo": np.array([g["moslqo"] for g in got], real), "vnsim": np.array([g["vnsim"] for g in got], real),
           "lag_s": np.array([g["alignment_lag_s"] for g in got])}
    for f in FEATURES:
        out[f] = np.concatenate([g[f] for g in got]).astype(real)
    rows = {k: np.zeros(state["first"][-1]) for k in ("similarity",) + TIMES}
    for i, g in enumerate(got):
        for k, p in enumerate(g["patch_sims"], state["first"][i]):
            rows["similarity"][k] = p["similarity"]
            for t in TIMES:
                rows[t][k] = p[t.replace("_", "_patch_") + "_time"]
    out.update(rows, similarity=rows["similarity"].astype(real))
    return out


def work(case):
    """The definition's arithmetic on the signals: the envelope correlation
    (two complex transforms), four biquads, window and square per gammatone
    sample (31 operations) for both signals, 33 per NSIM cell. Signals read
    once, results written. A gradient: the filter forward, its recomputation
    and its transpose for the degraded signal."""
    total_b = total_f = 0.0
    refs = 1 if case["what"] == "prepared" else case["pairs"]
    seconds = case["min_s"] if case["min_s"] == case["max_s"] else \
        (case["max_s"] - case["min_s"]) / math.log(case["max_s"] / case["min_s"])
    parts = [(case["mode"], case["rate"], case["pairs"])]
    if case["mode"] == "mixed":
        parts = [("audio", case["rate"], 0.7 * case["pairs"]), ("speech", 16000, 0.3 * case["pairs"])]
    for mode, rate, pairs in parts:
        nb, patch = (32, 30) if mode == "audio" else (21, 20)
        n = seconds * rate
        window, hop = round(rate * 0.08), int(round(rate * 0.08) * 0.25)
        frames = max(1.0, (n - window) / hop)
        patches = max(1.0, frames / patch - 0.5)
        fft = 2.0 ** math.ceil(math.log2(2 * n))
        filtered = 1.0 if case["what"] == "prepared" else 2.0
        total_f += pairs * (filtered * 31.0 * window * nb * frames + 10.0 * fft * math.log2(fft) +
                            33.0 * patches * frames * nb * patch)
        total_b += 8.0 * n * (pairs + min(refs, pairs)) + pairs * 8.0 * (4 * nb + 8 * patches)
        if case["what"] == "grad":
            total_f += pairs * 3 * 31.0 * window * nb * frames
            total_b += pairs * 8.0 * n
    return {"bytes": total_b, "flops": total_f}


# ---- the model in 64 bits -------------------------------------------------
# The same measurement restated on torch and numpy doubles: envelope lag,
# level match, gammatone spectrograms, NSIM table, patch alignment, per-patch
# realignment, pooling and the MOS mapping.

def _geometry(rate):
    window = int(math.floor(rate * 0.08 + 0.5))
    return window, int(window * 0.25)


@functools.lru_cache(maxsize=None)
def _filterbank(nb, rate):
    """Per band {n0..n3 first-tap ratios, gain, d1, d2} of the gammatone as four biquads."""
    high = min(8000.0, rate / 2.0) if nb == 21 else rate / 2.0
    q, bw, T = 9.26449, 24.7, 1.0 / rate
    e = (-math.log(high + q * bw) + math.log(50.0 + q * bw)) / nb
    cf = (-q * bw + np.exp(np.arange(1, nb + 1) * e) * (high + q * bw))[::-1].copy()
    B = 1.019 * 2 * np.pi * (cf / q + bw)
    w = 2 * np.pi * cf * T
    roots = np.array([math.sqrt(3 + 2 ** 1.5), -math.sqrt(3 + 2 ** 1.5), math.sqrt(3 - 2 ** 1.5),
                      -math.sqrt(3 - 2 ** 1.5)])
    taps = [-T * np.exp(-B * T) * (np.cos(w) + s * np.sin(w)) for s in roots]
    z = np.exp(2j * w)
    num = 1.0
    for s in (-roots[2], roots[2], -roots[0], roots[0]):
        num = num * (-2 * z * T + 2 * np.exp(-B * T + 1j * w) * T * (np.cos(w) + s * np.sin(w)))
    den = (-2 / np.exp(2 * B * T) - 2 * z + 2 * (1 + z) / np.exp(B * T)) ** 4
    gain = np.abs(num / den)
    return cf, taps, T, gain, -2 * np.cos(w) * np.exp(-B * T), np.exp(-2 * B * T)


def _rms(frames, nb, rate):
    """Gammatone RMS [nb, F] of windowed frames [W, F], sample by sample."""
    _, taps, T, gain, d1, d2 = _filterbank(nb, rate)
    dev = frames.device
    col = lambda v: torch.as_tensor(np.broadcast_to(v, (nb,)).copy(), device=dev)[:, None]  # noqa: E731
    first, rest = [col(T / gain)] + [col(T)] * 3, [col(taps[0] / gain)] + [col(t) for t in taps[1:]]
    nd1, nd2 = col(-d1), col(-d2)
    shape = (nb, frames.shape[1])
    c0 = [torch.zeros(shape, device=dev, dtype=torch.float64) for _ in range(4)]
    c1 = [torch.zeros(shape, device=dev, dtype=torch.float64) for _ in range(4)]
    total = torch.zeros(shape, device=dev, dtype=torch.float64)
    for i in range(frames.shape[0]):
        x = frames[i][None, :]
        for k in range(4):
            y = torch.addcmul(c0[k], first[k], x)
            c0[k] = torch.addcmul(torch.addcmul(c1[k], rest[k], x), nd1, y)
            c1[k] = nd2 * y
            x = y
        total.addcmul_(x, x)
    return torch.sqrt(total / frames.shape[0])


def _spectrograms(signals, nb, rate):
    """One spectrogram [nb, nf] per signal, all filtered together."""
    window, hop = _geometry(rate)
    hann = torch.as_tensor(0.5 - 0.5 * np.cos(2 * np.pi * np.arange(window) / (window - 1.0)), device=signals[0].device)
    cut = [s.unfold(0, window, hop) if s.numel() >= window else s.new_zeros((0, window)) for s in signals]
    frames = (torch.cat(cut) * hann).T.contiguous()
    rms = torch.cat([_rms(f, nb, rate) for f in frames.split(1 << 16, 1)], 1)
    return [r.contiguous() for r in rms.split([c.shape[0] for c in cut], 1)]


def _envelope(x):
    n = x.numel()
    pow2 = 32
    while pow2 < n:
        pow2 *= 2
    mean = x.mean()
    sign = 1.0 - 2.0 * (torch.arange(n, device=x.device) % 2)
    centred = x - mean
    return (2.0 * (centred - sign * (sign * centred).sum() / pow2) - 1e-6).abs() + mean


def _best_lag(a, b):
    """The lag whose envelope correlation is largest in magnitude."""
    a, b = _envelope(a), _envelope(b)
    most = max(a.numel(), b.numel())
    n = 1
    while n < 2 * most - 1:
        n *= 2
    corr = torch.fft.irfft(torch.fft.rfft(a, n) * torch.fft.rfft(b, n).conj(), n)
    at = torch.cat([corr[n - (most - 1):], corr[:most]]) if most > 1 else corr[:1]
    return int(at.abs().argmax()) - (most - 1)


def _decibels(ref, deg):
    to = lambda v: (10.0 * torch.log10(torch.where(v == 0, torch.full_like(v, 2.0 ** -52), v.abs()))).clamp(min=-45.0)  # noqa: E731
    r, d = to(ref), to(deg)
    m = min(r.shape[1], d.shape[1])
    floor = torch.maximum(r[:, :m].amax(0), d[:, :m].amax(0)) - 45.0
    r[:, :m] = torch.maximum(r[:, :m], floor)
    d[:, :m] = torch.maximum(d[:, :m], floor)
    lowest = torch.minimum(r.min(), d.min())
    return r - lowest, d - lowest


def _smooth(x):
    """3x3 Gaussian window over the last two axes, edges replicated."""
    x = torch.cat([x[..., :1, :], x, x[..., -1:, :]], -2)
    x = torch.cat([x[..., :1], x, x[..., -1:]], -1)
    corner, edge, centre = 0.0113033910173052, 0.0838251475442633, 0.619485845753726
    rows = lambda a, b: a * (x[..., :-2] + x[..., 2:]) + b * x[..., 1:-1]  # noqa: E731
    outer, inner = rows(corner, edge), rows(edge, centre)
    return outer[..., :-2, :] + inner[..., 1:-1, :] + outer[..., 2:, :]


def _cells(r, d):
    """NSIM of every cell of patches r against d (broadcast over leading axes)."""
    mr, md = _smooth(r), _smooth(d)
    vr, vd, cov = _smooth(r * r) - mr * mr, _smooth(d * d) - md * md, _smooth(r * d) - mr * md
    c1, c3 = 0.01 ** 2, 0.03 ** 2 / 2.0
    prod = vr * vd
    den = torch.where(prod < 0, torch.full_like(prod, c3), prod.clamp(min=0).sqrt() + c3)
    return (2.0 * mr * md + c1) / (mr * mr + md * md + c1) * ((cov + c3) / den)


def _band_stats(r, d):
    cells = _cells(r, d)
    sd = cells.std(1) if r.shape[1] > 1 else torch.zeros_like(cells[:, 0])
    means = cells.mean(1)
    return [v.cpu().numpy() for v in (means, sd, d.mean(1))] + [float(means.mean())]


def _patch_starts(mode, ref, nf, patch, window):
    first = patch // 2
    if mode == "audio":
        return list(range(first - 1, max(nf - patch, first + 1) - 1, patch))
    hop, first = int(window * 0.25), first - 1
    patches = (nf - first) // patch
    chunks = patches * patch
    x = ref.cpu().numpy()
    x = np.concatenate([x / x.max(), np.zeros(first + chunks * hop)])[first:first + chunks * hop].reshape(chunks, hop)
    s = np.trunc(np.clip(x * 32768.0, -32768.0, 32767.0))
    loud = np.sqrt((s * s).mean(1)) >= 5000.0
    active = np.ones(max(chunks, 2), bool)
    active[2:chunks] = loud[2:chunks] | loud[1:chunks - 1] | loud[:chunks - 2]
    return [first + p * patch for p in range(patches) if active[p * patch:(p + 1) * patch].any()]


def _align_patches(sims, lo, hi):
    """Dynamic programming over the similarity table: offset and validity per patch."""
    count, cols = sims.shape
    score, back = np.zeros((count, cols)), np.zeros((count, cols), np.int64)
    score[0, lo[0]:hi[0] + 1] = sims[0, lo[0]:hi[0] + 1]
    back[0, lo[0]:hi[0] + 1] = -1
    for p in range(1, count):
        prev, a, b = score[p - 1], lo[p], hi[p]
        seen = prev[lo[p - 1]:b]
        run = np.maximum.accumulate(seen)
        at = np.maximum.accumulate(np.where(seen == run, np.arange(seen.size), 0)) + lo[p - 1]
        run, at = np.concatenate([[-np.inf], run]), np.concatenate([[-1], at])
        s = np.arange(a, b + 1)
        moved, stay = sims[p, a:b + 1] + run[s - lo[p - 1]], prev[a:b + 1]
        keep = stay > moved
        score[p, a:b + 1] = np.where(keep, stay, moved)
        back[p, a:b + 1] = np.where(keep, s, at[s - lo[p - 1]])
    offset, valid = np.full(count, -1), np.ones(count, bool)
    cur = lo[-1] + int(np.argmax(score[-1, lo[-1]:hi[-1] + 1]))
    for p in range(count - 1, -1, -1):
        offset[p], nxt = cur, back[p, cur]
        valid[p] = nxt != cur
        if nxt < 0:
            break
        cur = nxt
    return offset, valid


def _slice(x, t0, t1, rate):
    """Samples between two times, zeros in front for what lies outside."""
    n = x.numel()
    first, last = max(0, int(t0 * rate)), min(n - 1, int(t1 * rate))
    pad = (int(t1 * rate - n) if t1 * rate > n else 0) + (int(-t0 * rate) if t0 < 0 else 0)
    body = x[first:last] if last > first else x[:0]
    return torch.cat([x.new_zeros(pad), body])


def _window_of(x, start, length):
    """length samples from start on, zeros outside."""
    pre = min(max(0, -start), length)
    body = x[max(0, start):max(0, start + length)]
    return torch.cat([x.new_zeros(pre), body, x.new_zeros(length - pre - body.numel())])


@functools.lru_cache(maxsize=None)
def _svr():
    gamma = rho = None
    coef, vectors = [], []
    path = os.path.join(os.path.dirname(native.__file__), "model", "libsvm_nu_svr_model.txt")
    with open(path) as f:
        for line in f:
            w = line.split()
            if len(w) == 2 and w[0] == "gamma":
                gamma = float(w[1])
            elif len(w) == 2 and w[0] == "rho":
                rho = float(w[1])
            elif w and ":" in line:
                coef.append(float(w[0]))
                v = np.zeros(32)
                for item in w[1:]:
                    k, x = item.split(":")
                    v[int(k) - 1] = float(x)
                vectors.append(v)
    return gamma, rho, np.array(coef), np.array(vectors)


def _model(pairs, mode, rate):
    """Results of (ref, deg) pairs, each a dict of values, in 64 bits."""
    nb, patch = (32, 30) if mode == "audio" else (21, 20)
    window, hop = _geometry(rate)
    step = hop / float(rate)
    aligned, lag_s = [], []
    for ref, deg in pairs:
        lag = _best_lag(ref, deg)
        lag = 0 if abs(lag) > ref.numel() // 2 else lag
        al = deg[min(-lag, deg.numel()):] if lag < 0 else torch.cat([deg.new_zeros(lag), deg])
        level = lambda x: 20.0 * math.log10(math.sqrt(float(x.square().sum()) / x.numel()) / 0.00002)  # noqa: E731
        aligned.append(al * 10.0 ** ((level(ref) - level(al)) / 20.0))
        lag_s.append(lag / float(rate))
    specs = _spectrograms([r for r, _ in pairs] + aligned, nb, rate)
    found, todo = [], []
    for i, (ref, _) in enumerate(pairs):
        r, d = _decibels(specs[i], specs[len(pairs) + i])
        nfr, nfd = r.shape[1], d.shape[1]
        starts = _patch_starts(mode, ref, nfr, patch, window)
        while starts and starts[-1] >= patch // 2 and starts[-1] - patch // 2 > nfd:
            starts.pop()
        lo = [max(0, s - RADIUS * patch) for s in starts]
        hi = [max(a, min(s + RADIUS * patch, nfd - 1)) for a, s in zip(lo, starts)]
        wide = torch.cat([d, d.new_zeros((nb, patch))], 1).unfold(1, patch, 1).permute(1, 0, 2)  # [offset, nb, patch]
        sims = np.zeros((len(starts), nfd))
        for p, s in enumerate(starts):
            for a in range(lo[p], hi[p] + 1, 4096):
                b = min(a + 4096, hi[p] + 1)
                sims[p, a:b] = _cells(r[:, s:s + patch], wide[a:b]).mean((1, 2)).cpu().numpy()
        offset, valid = _align_patches(sims, lo, hi)
        matches = []
        for p, s in enumerate(starts):
            m = {"means": np.zeros(nb), "sd": np.zeros(nb), "energy": np.zeros(nb), "similarity": 0.0,
                 "times": [0.0, 0.0, 0.0, 0.0]}
            if offset[p] >= 0:
                m["means"], m["sd"], m["energy"], m["similarity"] = _band_stats(r[:, s:s + patch], wide[offset[p]])
                m["times"][:2] = [s * step, s * step + step * patch]
                if valid[p]:
                    m["times"][2:] = [offset[p] * step, offset[p] * step + step * patch]
                    t = m["times"]
                    a, b = _slice(ref, t[0], t[1], rate), _slice(aligned[i], t[2], t[3], rate)
                    if a.numel() >= window and b.numel() >= window:
                        todo.append((m, a, b))
                else:
                    m["means"], m["similarity"] = np.zeros(nb), 0.0
            matches.append(m)
        found.append(matches)
    # realignment: the slices' own lag, trimmed to the same length and compared again
    trimmed = []
    for m, a, b in todo:
        lag = _best_lag(a, b)
        lag = 0 if abs(lag) > a.numel() // 2 else lag
        length, head = a.numel(), 0
        blen = b.numel() - min(-lag, b.numel()) if lag < 0 else b.numel() + lag
        if a.numel() > blen:
            length = blen
        elif a.numel() < blen and lag > 0:
            head = int(lag / float(rate) * rate)
            length = a.numel() - head
        if length >= window:
            trimmed.append((m, _window_of(a, head, length), _window_of(b, head - lag, length), lag / float(rate), length))
    specs = _spectrograms([t[1] for t in trimmed] + [t[2] for t in trimmed], nb, rate) if trimmed else []
    for k, (m, _, _, shift, length) in enumerate(trimmed):
        stats = _band_stats(*_decibels(specs[k], specs[len(trimmed) + k]))
        if stats[3] >= m["similarity"]:
            m["means"], m["sd"], m["energy"], m["similarity"] = stats
            t = m["times"]
            if shift > 0:
                t[0] += shift
            else:
                t[2] -= shift
            t[1], t[3] = t[0] + length / float(rate), t[2] + length / float(rate)
    return [_pool(matches, lag_s[i], mode, nb, step) for i, matches in enumerate(found)]


def _pool(matches, lag, mode, nb, step):
    means = np.array([m["means"] for m in matches])
    sd = np.array([m["sd"] for m in matches])
    fvnsim, n = means.mean(0), len(matches)
    low = np.sort(means, 0)[:max(1, int(n * 0.10))].mean(0)
    frames = np.array([math.ceil((m["times"][1] - m["times"][0]) / step) for m in matches], float)[:, None]
    var = (((frames - 1) * sd ** 2 + frames * means ** 2).sum(0) - fvnsim ** 2 * frames.sum()) / (frames.sum() - 1)
    if mode == "audio":
        gamma, rho, coef, vectors = _svr()
        mos = float(coef @ np.exp(-gamma * ((vectors - fvnsim) ** 2).sum(1)) - rho)
    else:
        mos = (-262.847869 + math.exp(0.0154302525 * (float(fvnsim.mean()) + 361.063949))) * float(np.float32(1.245063))
    mos = 1.0 if fvnsim.mean() < 0.15 else min(max(mos, 1.0), 5.0)
    return {"moslqo": mos, "vnsim": float(fvnsim.mean()), "lag_s": lag, "fvnsim": fvnsim, "fvnsim10": low,
            "fstdnsim": np.sqrt(np.maximum(var, 0.0)), "fvdegenergy": np.mean([m["energy"] for m in matches], 0),
            "similarity": [m["similarity"] for m in matches], "times": [m["times"] for m in matches]}


def exact(case, seed):
    """What run returns, in 64 bits (a gradient has no value here)."""
    pairs = _signals(case, seed)
    got = [None] * len(pairs)
    for mode, rate in sorted({p[:2] for p in pairs}):
        at = [i for i, p in enumerate(pairs) if p[:2] == (mode, rate)]
        for i, r in zip(at, _model([pairs[i][2:] for i in at], mode, rate)):
            got[i] = r
    mixed = case["what"] == "server"
    out = {k: np.array([g[k] for g in got]) for k in ("moslqo", "vnsim", "lag_s")}
    for f in FEATURES:
        out[f] = np.concatenate([g[f] for g in got]) if mixed else np.stack([g[f] for g in got])
    first = np.concatenate([[0], np.cumsum(_slots(case))])
    out.update({k: np.zeros(first[-1]) for k in ("similarity",) + TIMES})
    for i, g in enumerate(got):
        rows = slice(first[i], first[i] + len(g["times"]))
        out["similarity"][rows] = g["similarity"]
        for k, t in enumerate(TIMES):
            out[t][rows] = [times[k] for times in g["times"]]
    if case["what"] == "grad":
        out["grad"] = None
    return out
