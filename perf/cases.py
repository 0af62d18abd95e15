"""What this library's users have it do, as cases that can be timed and checked.

A case is a dict of plain values.  `prepare` makes what a program holds before
the call (blocks of IQ in device memory, an admitted runner, a detector),
`run` is one pass through the public entry points (the `gpudemod` package, or
the C ABI that it binds, as a cgo program calls it), `work` what the pass
cannot do without and `exact` the same outputs in 64 bits.

The kinds of work, one for each part of the library that a program binds:

  runner    the batched / serving runner: one IQ block through every channel
  extract   StreamingExtractGPU: a host block and its extraction jobs
  launcher  the drop-in streaming polyphase launcher, one signal
  slots     the legacy slot chain: shift, FIR and decimation per job and stream
  pilot     long-window stereo pilot decision for a batch of stations
  rds       RDS symbol and group decoding for a batch of stations
  welch     the surveillance spectrum
  event     a recorded event turned into audio in one call

Streams are periodic over their blocks (every tone on the period's frequency
grid), so a runner that is fed them again and again sees one unbroken signal.
"""
from __future__ import annotations

import ctypes as C
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "argus-sdr_b200"))

import gpudemod as G  # noqa: E402
from gpudemod import synth  # noqa: E402
from gpudemod._lib import ChannelResult, lib  # noqa: E402

TWO_PI = 2.0 * math.pi
DEV = "cuda"
WARM_BLOCKS = 4  # blocks that a prepared runner has had: pilot loops in lock, stereo on
PERIOD = {"fm": 4, "narrow": 4, "serving": 8, "headroom": 4}  # blocks of a stream
MODE = {"WFM": G.MODE_WFM_STEREO, "NFM": G.MODE_NFM, "AM": G.MODE_AM, "USB": G.MODE_USB, "LSB": G.MODE_LSB,
        "CW": G.MODE_CW}
# WFM .30 / NFM .30 / AM .20 / SSB .15 / CW .05: the requests of the serving stream
SERVING_MIX = (("WFM", 0.30), ("NFM", 0.30), ("AM", 0.20), ("USB", 0.08), ("LSB", 0.07), ("CW", 0.05))
NARROW_MIX = (("NFM", 40 / 120), ("AM", 30 / 120), ("USB", 15 / 120), ("LSB", 15 / 120), ("CW", 20 / 120))
HEADROOM_MIX = (("WFM", 0.30), ("NFM", 0.233), ("AM", 0.175), ("USB", 0.088), ("LSB", 0.087), ("CW", 0.117))


# --------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------

def listed():
    return [
        # One broadcast station at a small receiver's rate in odd blocks, IQ
        # emitted beside its audio: the smallest serving call, bound by latency
        # and launches.
        {"name": "one_wfm", "kind": "runner", "mix": "fm", "fs": 2_400_000, "block": 61_439, "channels": 1,
         "taps": 128, "decim": 8, "pcm": 0, "emit_iq": 1, "pop": 1},
        # The FM broadcast band: 40 stereo stations with RDS from one 10 MS/s
        # block, 48 kHz audio (float, so that rounding is seen as it is).
        {"name": "fm_band", "kind": "runner", "mix": "fm", "fs": 10_000_000, "block": 1 << 20, "channels": 40,
         "taps": 256, "decim": 32, "pcm": 2, "emit_iq": 0, "pop": 2},
        # 120 narrow channels of five modes, uneven taps and decimations, their
        # audio as the 48 kHz s16le stream that goes to listeners.
        {"name": "mixed_120", "kind": "runner", "mix": "narrow", "fs": 10_000_000, "block": 1 << 20, "channels": 120,
         "taps": 0, "decim": 0, "pcm": 1, "emit_iq": 0, "pop": 3},
        # The serving stream at its cap: 512 requests of all modes at random
        # frequencies, on stations and on noise, one 26 ms block.
        {"name": "serving_512", "kind": "runner", "mix": "serving", "fs": 10_000_000, "block": 262_144,
         "channels": 512, "taps": 0, "decim": 0, "pcm": 2, "emit_iq": 0, "pop": 4},
        # Headroom: 2048 channels of 64..1024 taps and decimations 16..2400 at
        # 61.44 MS/s, outputs left on the device for the consumers there.
        {"name": "headroom_2048", "kind": "runner", "mix": "headroom", "fs": 61_440_000, "block": 960_000,
         "channels": 2048, "taps": 0, "decim": 0, "pcm": 0, "emit_iq": 0, "pop": 6},
        # The detector's extraction jobs of one 50 ms frame of a live capture:
        # two broadcast signals at 512 kS/s and six narrow ones.
        {"name": "extract_8", "kind": "extract", "fs": 4_096_000, "n": 204_803, "jobs": 8, "taps": 101},
        # One signal through the drop-in streaming launcher of the cgo path.
        {"name": "launcher_one", "kind": "launcher", "fs": 4_096_000, "n": 204_800, "taps": 257, "decim": 20},
        # The RDS extraction of the live FM band: four stations, each its own
        # stream of shift, 101-tap FIR and decimation to 256 kS/s.
        {"name": "slots_4", "kind": "slots", "fs": 4_096_000, "n": 409_600, "jobs": 4, "taps": 101, "decim": 16},
        # Stereo pilot decisions for the 40 stations of the band, once a cadence.
        {"name": "pilot_40", "kind": "pilot", "stations": 40, "fs": 312_500, "n": 163_840},
        # RDS decoding of four seconds of the same stations.
        {"name": "rds_40", "kind": "rds", "stations": 40, "fs": 19_531, "n": 78_125},
        # The surveillance spectrum of a frame: Welch over 16 half-overlapping
        # windows of 4096.
        {"name": "welch_16", "kind": "welch", "fft": 4096, "segs": 16},
        # A recorded two-second event of a broadcast station, host IQ in, 48 kHz
        # stereo out.
        {"name": "event_wfm", "kind": "event", "mode": "BATCH", "fs": 2_400_000, "n": 4_800_000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    """One more case of the listed ones' ranges."""
    kind = rng.choice(["fm", "fm", "narrow", "narrow", "serving", "serving", "headroom", "extract", "launcher",
                       "slots", "pilot", "rds", "welch", "event"])
    pop = rng.randrange(1 << 20)
    if kind == "fm":
        small = rng.random() < 0.3
        fs = 2_400_000 if small else 10_000_000
        return {"kind": "runner", "mix": "fm", "fs": fs, "block": _log(rng, 50_000, 1 << 20) | rng.randrange(2),
                "channels": rng.randrange(1, 5) if small else _log(rng, 2, 45), "taps": rng.randrange(96, 321),
                "decim": 8 if small else rng.choice([32, 32, 40]), "pcm": rng.choice([0, 2, 2]),
                "emit_iq": rng.randrange(2), "pop": pop}
    if kind in ("narrow", "serving"):
        return {"kind": "runner", "mix": kind, "fs": 10_000_000, "block": _log(rng, 60_000, 1 << 20) | rng.randrange(2),
                "channels": _log(rng, 5, 240 if kind == "narrow" else 512), "taps": 0, "decim": 0,
                "pcm": 1 if kind == "narrow" else 2, "emit_iq": 0, "pop": pop}
    if kind == "headroom":
        return {"kind": "runner", "mix": "headroom", "fs": 61_440_000, "block": rng.choice([480_000, 960_000]),
                "channels": _log(rng, 100, 1500), "taps": 0, "decim": 0, "pcm": 0, "emit_iq": 0, "pop": pop}
    if kind == "extract":
        return {"kind": "extract", "fs": 4_096_000, "n": _log(rng, 20_000, 800_000) | 1, "jobs": rng.randrange(1, 25),
                "taps": rng.choice([101, rng.randrange(64, 400)])}
    if kind == "launcher":
        return {"kind": "launcher", "fs": 4_096_000, "n": _log(rng, 10_000, 262_144), "taps": rng.randrange(65, 513),
                "decim": rng.choice([4, 8, 16, 20, 32, 64, 80])}
    if kind == "slots":
        return {"kind": "slots", "fs": 4_096_000, "n": _log(rng, 40_000, 1_000_000) | 1, "jobs": rng.randrange(1, 9),
                "taps": 101, "decim": rng.choice([8, 16, 20, 32])}
    if kind == "pilot":
        return {"kind": "pilot", "stations": _log(rng, 1, 60), "fs": rng.choice([256_000, 312_500, 320_000, 512_000]),
                "n": _log(rng, 20_000, 400_000)}
    if kind == "rds":
        return {"kind": "rds", "stations": _log(rng, 1, 60), "fs": rng.choice([19_200, 19_531, 20_000]),
                "n": _log(rng, 4_000, 120_000)}
    if kind == "welch":
        return {"kind": "welch", "fft": rng.choice([1024, 2048, 4096, 8192]), "segs": rng.randrange(1, 49)}
    return {"kind": "event", "mode": rng.choice(["BATCH", "BATCH", "NFM", "AM", "USB", "WFM_STEREO"]),
            "fs": rng.choice([2_400_000, 2_048_000]), "n": _log(rng, 200_000, 4_800_000)}


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------

def _rng(*key):
    return np.random.default_rng([int(k) for k in key])


def _running_sum(v):
    """cumsum in a fixed order of additions: rows of 4096, then the rows."""
    n = v.numel()
    rows = torch.cat([v, v.new_zeros(-n % 4096)]).view(-1, 4096).cumsum(1)
    ends = rows[:, -1].expand(2, -1).contiguous().cumsum(1)[0]
    rows[1:] += ends[:-1, None]
    return rows.view(-1)[:n]


def _fm(rng, n, fs, deviation, mpx):
    """exp(j of the integral of the modulation), closing on itself after n."""
    total = _running_sum(mpx)
    total -= (total[-1] / n) * torch.arange(1, n + 1, dtype=torch.float64, device=DEV)
    return torch.exp(1j * (total * (TWO_PI * deviation / fs) + rng.uniform(0, TWO_PI)))


def _station(rng, kind, n, fs):
    """Baseband of one station over a period of n samples (complex128, level 1)."""
    t = torch.arange(n, dtype=torch.float64, device=DEV) / fs
    grid = fs / n

    def tone(f, a):
        return a * torch.sin((TWO_PI * max(1, round(f / grid)) * grid) * t + rng.uniform(0, TWO_PI))

    if kind == "WFM":
        left = sum(tone(f, 0.2 / (1 + f / 1500.0) ** 2) for f in rng.uniform(100.0, 15000.0, 3))
        right = sum(tone(f, 0.2 / (1 + f / 1500.0) ** 2) for f in rng.uniform(100.0, 15000.0, 3))
        w = TWO_PI * max(1, round(19_000.0 / grid)) * grid
        pilot = w * t
        bits = max(2, round(1187.5 * n / fs))
        sym = torch.as_tensor(2.0 * rng.integers(0, 2, bits + 1) - 1.0, device=DEV)
        sym[bits] = sym[0]
        pos = t * (bits * fs / n)
        k = torch.clamp(pos.long(), 0, bits - 1)
        c = 0.5 * (1 + torch.cos(math.pi * (pos - k)))
        rds = sym[k] * c + sym[k + 1] * (1 - c)
        mpx = 0.5 * (left + right) + 0.5 * (left - right) * torch.sin(2 * pilot) + 0.1 * torch.sin(pilot) \
            + 0.05 * rds * torch.cos(3 * pilot + rng.uniform(0, TWO_PI))
        return _fm(rng, n, fs, 75_000.0, mpx)
    freqs, amps = rng.uniform(300.0, 2700.0, 3), rng.uniform(0.3, 1.0, 3)
    amps = amps / amps.sum()
    if kind == "NFM":
        return _fm(rng, n, fs, 2500.0, sum(tone(f, a) for f, a in zip(freqs, amps)))
    if kind == "AM":
        return (1.0 + 0.6 * sum(tone(f, a) for f, a in zip(freqs, amps))).to(torch.complex128)
    if kind in ("USB", "LSB"):
        s = 1.0 if kind == "USB" else -1.0
        return sum(a * torch.exp(1j * ((s * TWO_PI * max(1, round(f / grid)) * grid) * t + rng.uniform(0, TWO_PI)))
                   for f, a in zip(freqs, amps))
    keys = torch.as_tensor(rng.integers(0, 2, max(2, round(20.0 * n / fs))).astype(np.float64), device=DEV)
    return keys[torch.clamp((t * (len(keys) * fs / n)).long(), 0, len(keys) - 1)].to(torch.complex128)


def _stream(seed, fs, n, stations, noise):
    """Sum of stations [(kind, offset Hz, level)] and noise over a period of n
    samples: complex64 on the device."""
    rng = _rng(seed, 11)
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    x = torch.view_as_complex(torch.randn(n, 2, generator=g, device=DEV, dtype=torch.float64)) * (noise / math.sqrt(2))
    i = torch.arange(n, dtype=torch.float64, device=DEV)
    for kind, off, level in stations:
        k = round(off * n / fs)
        ph = torch.remainder(i * k, n) * (TWO_PI / n)
        x += level * _station(rng, kind, n, fs) * torch.exp(1j * ph)
    return x.to(torch.complex64)


def _population(case):
    """The channels of a runner case, equal ones one after another: dicts with
    kind, T, D and bandwidth (and where they may sit, from the seed)."""
    mix, n, rng = case["mix"], case["channels"], _rng(case["pop"], 7)
    if mix == "fm":
        return [{"kind": "WFM", "T": case["taps"], "D": case["decim"], "bw": 250_000.0} for _ in range(n)]
    table = {"narrow": NARROW_MIX, "serving": SERVING_MIX, "headroom": HEADROOM_MIX}[mix]
    chans = []
    for kind, share in table:
        rate, taps, bw = synth.MODE_TABLE[kind]
        # the shares rounded up, cut to the count below: small populations keep every mode
        for _ in range(math.ceil(share * n)):
            D = case["fs"] // rate if mix != "headroom" else 192
            if mix == "headroom":
                taps = int(rng.integers(64, 1025))
                if kind != "WFM":
                    divs = [d for d in range(16, 2401) if case["block"] % d == 0 and case["fs"] % d == 0]
                    u = rng.uniform(math.log(16), math.log(2400))
                    D = min(divs, key=lambda d: abs(math.log(d) - u))
            chans.append({"kind": kind, "T": taps, "D": D, "bw": bw})
    while len(chans) > n:
        chans.pop(int(rng.integers(len(chans))))
    order = [k for k, _ in table]
    return sorted(chans, key=lambda c: (order.index(c["kind"]), c["T"], c["D"]))


def _scene(case, seed):
    """(stream of PERIOD blocks, channels with their offsets)."""
    fs, mix = case["fs"], case["mix"]
    chans, rng = _population(case), _rng(seed, 3)
    n = PERIOD[mix] * case["block"]
    if mix == "fm":
        step = 200_000.0
        slots = int(0.9 * fs / step)
        at = np.sort(rng.choice(slots, size=len(chans), replace=False)) - (slots - 1) / 2
        for c, a in zip(chans, at):
            c["off"] = float(a) * step
        stations = [("WFM", c["off"], math.sqrt(10 ** (rng.uniform(10.0, 40.0) / 10)) * 0.01) for c in chans]
        return _stream(seed, fs, n, stations, 0.01 * math.sqrt(fs / 200_000.0)), chans
    if mix == "narrow":
        grid = np.arange(-0.49 * fs, 0.49 * fs, 25_000.0)
        for c, off in zip(chans, rng.choice(grid, size=len(chans), replace=False)):
            c["off"] = float(off)
        stations = [(c["kind"], c["off"], math.sqrt(10 ** (rng.uniform(5.0, 35.0) / 10)) * 0.01
                     * math.sqrt(c["bw"] / 12_500.0)) for c in chans]
        return _stream(seed, fs, n, stations, 0.01 * math.sqrt(fs / 12_500.0)), chans
    # serving, headroom: stations over the band, requests on them and on noise
    wfm = rng.choice(np.arange(-0.47 * fs, 0.47 * fs, 400_000.0), size=12, replace=False)
    narrow = [(k, float(f)) for k, f in zip(["NFM"] * 16 + ["AM"] * 12 + ["USB"] * 6 + ["LSB"] * 6 + ["CW"] * 8,
                                            rng.choice(np.arange(-0.49 * fs, 0.49 * fs, 25_000.0), 48, False))]
    stations = [("WFM", float(f), math.sqrt(10 ** (rng.uniform(5.0, 35.0) / 10)) * 0.01) for f in wfm]
    stations += [(k, f, math.sqrt(10 ** (rng.uniform(5.0, 35.0) / 10)) * 0.01
                  * math.sqrt(synth.MODE_TABLE[k][2] / 12_500.0)) for k, f in narrow]
    for c in chans:
        on = [f for k, f, _ in stations if k == c["kind"]]
        near = on and rng.random() < (0.8 if c["kind"] == "WFM" and mix == "headroom" else 0.5)
        c["off"] = float(on[int(rng.integers(len(on)))] if near else rng.uniform(-0.48 * fs, 0.48 * fs))
    return _stream(seed, fs, n, stations, 0.01 * math.sqrt(fs / 200_000.0)), chans


def _baseband(seed, stations, n, fs):
    """FM multiplex basebands of `stations` stations (complex64 rows, noisy)."""
    rows = []
    for s in range(stations):
        rng = _rng(seed, 5, s)
        rows.append(_stream(seed * 131 + s, fs, n, [("WFM", 0.0, 1.0)], 10 ** (-rng.uniform(5.0, 35.0) / 20)))
    return rows


def _rds_baseband(seed, stations, n, fs):
    """57 kHz RDS basebands: BPSK groups with PI, PS and RT, noisy, with a
    carrier phase, as the runner's RDS output carries them."""
    rows = []
    t = np.arange(n) / fs
    for s in range(stations):
        rng = _rng(seed, 9, s)
        pi, ps, rt = synth.random_station_text(rng)
        sym = synth.rds_symbols(synth.rds_bits(synth.rds_groups(pi, ps, rt), int(n * 1187.5 / fs) + 8))
        pos = t * 1187.5 + rng.uniform(0, 1)
        k = pos.astype(np.int64)
        c = 0.5 * (1 + np.cos(math.pi * (pos - k)))
        z = (sym[k] * c + sym[k + 1] * (1 - c)) * np.exp(1j * rng.uniform(0, TWO_PI))
        z = 0.05 * (z + 10 ** (-rng.uniform(8.0, 30.0) / 20) * (rng.standard_normal(n) + 1j * rng.standard_normal(n)))
        rows.append(torch.from_numpy(z.astype(np.complex64)).to(DEV))
    return rows


# --------------------------------------------------------------------------
# the runner
# --------------------------------------------------------------------------

class _Classes:
    """Reads one block's payload out of the runner.  Channels of one class
    were admitted one after another, so their payload lies at equal distances
    in the block's output arena: the first and the last of a class give a view
    over all of them, without a copy."""

    def __init__(self, runner, chans, slots):
        self.runner, self.r = runner, runner._r
        self.runs = []  # (kind, slots of the class in order)
        for c, s in zip(chans, slots):
            key = (c["kind"], c["T"], c["D"])
            if not self.runs or self.runs[-1][0] != key:
                self.runs.append((key, []))
            self.runs[-1][1].append(s)
        self.a, self.b = ChannelResult(), ChannelResult()

    def read(self, slot, into):
        if lib.gpud_runner_result(self.r, slot, C.byref(into)) != 0:
            raise RuntimeError("no result")

    def view(self, first, last, count, n, dtype):
        at = C.cast(first, C.c_void_p).value
        if not at or n <= 0:
            return np.zeros((count, 0), dtype)
        pitch = (C.cast(last, C.c_void_p).value - at) // (count - 1) if count > 1 else n * np.dtype(dtype).itemsize
        arena = (C.c_char * (pitch * (count - 1) + n * np.dtype(dtype).itemsize)).from_address(at)
        arena.owner = self.runner  # the view keeps the runner and so its arena
        return np.ndarray((count, n), dtype, np.frombuffer(arena, np.uint8), 0, (pitch, np.dtype(dtype).itemsize))

    def all(self, case):
        out = {}
        for i, ((kind, _, _), slots) in enumerate(self.runs):
            a, b, m = self.a, self.b, len(slots)
            self.read(slots[0], a)
            self.read(slots[-1], b)
            got = {}
            if case["pcm"] == 1:
                got["pcm"] = self.view(a.pcm, b.pcm, m, a.n_pcm, np.int16)
            elif case["pcm"] == 2:
                got["pcm"] = self.view(a.pcm_f32, b.pcm_f32, m, a.n_pcm, np.float32)
            else:
                got["audio"] = self.view(a.audio, b.audio, m, a.n_audio, np.float32)
            if kind == "WFM":
                got["rds"] = self.view(a.rds, b.rds, m, a.n_rds, np.complex64)
            if case["emit_iq"]:
                got["iq"] = self.view(a.iq, b.iq, m, a.n_iq, np.complex64)
            out["%d_%s" % (i, kind)] = got
        return out


class _OnDevice:
    """Payload left on the device: every channel's samples gathered out of the
    arena by kind.  The block length is a multiple of every decimation, so the
    arena's layout is the same in every block and is read once."""

    class _Raw:
        def __init__(self, at, n, typestr):
            self.__cuda_array_interface__ = {"data": (at, False), "shape": (n,), "typestr": typestr, "version": 3}

    def __init__(self, runner, chans, slots):
        self.r, self.slots, self.res = runner._r, slots, ChannelResult()
        self.index, self.views = {}, {}
        spans = {"audio": {}, "rds": {}}
        for c, s in zip(chans, slots):
            lib.gpud_runner_result(self.r, s, C.byref(self.res))
            for what, p, n in (("audio", self.res.audio, self.res.n_audio), ("rds", self.res.rds, self.res.n_rds)):
                if n > 0:
                    spans[what].setdefault(c["kind"], []).append((C.cast(p, C.c_void_p).value, n))
        lib.gpud_runner_result(self.r, slots[0], C.byref(self.res))
        for what, size in (("audio", 4), ("rds", 8)):
            base = C.cast(getattr(self.res, what), C.c_void_p).value
            if any(at < base for v in spans[what].values() for at, _ in v):
                raise RuntimeError("the first channel does not lead the arena")
            for kind, v in spans[what].items():
                self.index[what, kind] = torch.from_numpy(np.concatenate(
                    [np.arange(n) + (at - base) // size for at, n in v])).to(DEV)
            self.views[what] = {}
        self.length = {w: max([int(i.max()) + 1 for (q, _), i in self.index.items() if q == w] or [0])
                       for w in ("audio", "rds")}

    def all(self, case):
        lib.gpud_runner_result(self.r, self.slots[0], C.byref(self.res))
        out = {}
        for what, typestr in (("audio", "<f4"), ("rds", "<c8")):
            if not self.length[what]:
                continue
            at = C.cast(getattr(self.res, what), C.c_void_p).value
            if at not in self.views[what]:
                self.views[what][at] = torch.as_tensor(self._Raw(at, self.length[what], typestr), device=DEV)
            for (w, kind), index in self.index.items():
                if w == what:
                    out[kind + "_" + what] = self.views[what][at][index]
        return out


def _flags(case, kind):
    f = G.CH_RDS if kind == "WFM" else 0
    f |= G.CH_EMIT_IQ if case["emit_iq"] else 0
    return f | (0, G.CH_AUDIO48K, G.CH_AUDIO48K | G.CH_PCM_F32)[case["pcm"]]


def _prepare_runner(case, seed):
    x, chans = _scene(case, seed)
    blocks = list(x.view(PERIOD[case["mix"]], case["block"]))
    runner = G.ChannelRunner(case["fs"], case["block"], max_channels=len(chans), max_taps=1024)
    slots = [runner.admit(i + 1, c["off"], c["bw"], case["fs"] // c["D"], c["T"], MODE[c["kind"]],
                          _flags(case, c["kind"])) for i, c in enumerate(chans)]
    on_device = case["mix"] == "headroom"
    runner.set_host_outputs(not on_device)
    torch.cuda.synchronize()
    for b in range(WARM_BLOCKS):
        runner.process_block(blocks[b % len(blocks)])
    reader = (_OnDevice if on_device else _Classes)(runner, chans, slots)
    return {"kind": "runner", "case": case, "runner": runner, "blocks": blocks, "at": WARM_BLOCKS % len(blocks),
            "reader": reader, "wait": torch.cuda.current_stream() if on_device else None}


def _run_runner(s):
    if s["wait"] is not None:
        s["wait"].synchronize()  # the consumer of the last block's payload has read it
    s["runner"].process_block(s["blocks"][s["at"]])
    s["at"] = (s["at"] + 1) % len(s["blocks"])
    return s["reader"].all(s["case"])


# --------------------------------------------------------------------------
# prepare and run
# --------------------------------------------------------------------------

def _jobs(case, rng):
    """Extraction jobs of a frame: every fourth a broadcast signal at 512 kS/s,
    the others at the exact rate nearest 200 kS/s."""
    fs, jobs = case["fs"], []
    for i in range(case["jobs"]):
        wide = i % 4 == 0
        rate = 512_000 if wide else 204_800
        off, bw = float(rng.uniform(-0.4 * fs, 0.4 * fs)), 250_000.0 if wide else float(rng.uniform(20_000, 60_000))
        jobs.append(G.StreamingExtractJob(i + 1, off, bw, rate, case["taps"],
                                          G.StreamingConfigHash(i + 1, off, bw, rate, case["taps"], fs)))
    return jobs


def _live(case, seed, n):
    """n samples of a live capture: a few stations and noise."""
    rng = _rng(seed, 21)
    fs = case["fs"]
    stations = [("WFM", float(f), 0.3) for f in rng.uniform(-0.4 * fs, 0.4 * fs, 3)]
    stations += [(k, float(f), 0.1) for k, f in zip(("NFM", "AM"), rng.uniform(-0.45 * fs, 0.45 * fs, 2))]
    return _stream(seed, fs, n, stations, 0.05)


def _factor(rate, target):
    """Decimation nearest to a target rate, halves upwards."""
    return max(1, int(rate / target + 0.5))


def _launcher_setup(case, seed):
    rng = _rng(seed, 23)
    off = float(rng.uniform(-0.4, 0.4)) * case["fs"]
    h = _taps32(200_000.0, case["fs"], case["taps"])
    return off, h, _live(case, seed, case["n"])


def _slot_setup(case, seed):
    rng = _rng(seed, 25)
    offs = [float(o) for o in rng.uniform(-0.4, 0.4, case["jobs"]) * case["fs"]]
    starts = [float(p) for p in rng.uniform(-3.0, 3.0, case["jobs"])]
    return offs, starts, _taps32(200_000.0, case["fs"], case["taps"]), _live(case, seed, case["n"])


def _event_setup(case, seed):
    rng = _rng(seed, 27)
    off = float(rng.uniform(-0.3, 0.3)) * case["fs"]
    kind = case["mode"] if case["mode"] in ("NFM", "AM", "USB") else "WFM"
    x = _stream(seed, case["fs"], case["n"], [(kind, off, 1.0)], 0.2)
    return off, {"WFM": 180_000.0, "NFM": 12_500.0, "AM": 10_000.0, "USB": 3_000.0}[kind], x


def prepare(case, seed):
    kind, seed = case["kind"], int(seed)
    if kind == "runner":
        return _prepare_runner(case, seed)
    if kind == "extract":
        iq = _live(case, seed, case["n"]).cpu().numpy()
        return {"kind": kind, "runner": G.NewBatchRunner(case["n"], case["fs"]), "iq": iq,
                "jobs": _jobs(case, _rng(seed, 22))}
    if kind == "launcher":
        off, h, x = _launcher_setup(case, seed)
        T, D = case["taps"], case["decim"]
        poly = G.BuildPolyphaseTapsPhaseMajor(h, D)
        buf = {k: torch.zeros(m, dtype=torch.complex64, device=DEV) for k, m in
               (("sh", case["n"]), ("hist", T - 1), ("scr", T - 1), ("out", case["n"] // D + 2))}
        return {"kind": kind, "x": x, "poly": torch.from_numpy(poly).to(DEV), "case": case, "buf": buf,
                "hl": C.c_int(0), "pc": C.c_int(0), "ph": C.c_double(0.0), "n_out": C.c_int(0),
                "inc": -TWO_PI * off / case["fs"]}
    if kind == "slots":
        offs, starts, h, x = _slot_setup(case, seed)
        n, slots = case["n"], []
        for off, start in zip(offs, starts):
            st = C.c_void_p()
            if lib.gpud_stream_create(C.byref(st)) != 0:
                raise RuntimeError("stream")
            slots.append({"stream": st, "inc": -TWO_PI * off / case["fs"], "start": start,
                          "taps": torch.from_numpy(h).to(DEV),
                          **{k: torch.empty(m, dtype=torch.complex64, device=DEV) for k, m in
                             (("sh", n), ("flt", n), ("dec", n // case["decim"]))}})
        return {"kind": kind, "x": x, "case": case, "slots": slots}
    if kind == "pilot":
        n = min(case["n"], case["fs"])
        return {"kind": kind, "iq": _baseband(seed, case["stations"], n, case["fs"]),
                "rates": [case["fs"]] * case["stations"],
                "det": G.StereoPilotDetector(case["stations"], case["fs"])}
    if kind == "rds":
        iq = _rds_baseband(seed, case["stations"], case["n"], case["fs"])
        return {"kind": kind, "jobs": [(x, case["fs"], i) for i, x in enumerate(iq)],
                "dec": G.RDSDecoder(case["stations"], case["n"])}
    if kind == "welch":
        n = case["fft"] + (case["segs"] - 1) * (case["fft"] // 2)
        return {"kind": kind, "iq": _live({"fs": 4_096_000}, seed, n), "case": case,
                "sp": G.Spectrum(case["fft"], case["segs"])}
    off, bw, x = _event_setup(case, seed)
    return {"kind": "event", "case": case, "off": off, "bw": bw, "iq": x.cpu().numpy()}


def run(s):
    kind = s["kind"]
    if kind == "runner":
        return _run_runner(s)
    if kind == "extract":
        return [r.IQ for r in s["runner"].StreamingExtractGPU(s["iq"], s["jobs"])]
    if kind == "launcher":
        c, b = s["case"], s["buf"]
        rc = lib.gpud_launch_streaming_polyphase_stateful_cuda(
            s["x"].data_ptr(), c["n"], b["sh"].data_ptr(), s["poly"].data_ptr(), s["poly"].numel(), c["decim"],
            c["taps"], b["hist"].data_ptr(), b["scr"].data_ptr(), c["taps"] - 1, C.byref(s["hl"]), C.byref(s["pc"]),
            C.byref(s["ph"]), s["inc"], b["out"].data_ptr(), b["out"].numel(), C.byref(s["n_out"]))
        if rc != 0:
            raise RuntimeError("launcher: %d" % rc)
        return b["out"][:s["n_out"].value], b["hist"][:s["hl"].value], s["ph"].value, s["pc"].value
    if kind == "slots":
        c, x, n = s["case"], s["x"].data_ptr(), s["case"]["n"]
        for q in s["slots"]:
            sh, flt, dec = q["sh"].data_ptr(), q["flt"].data_ptr(), q["dec"].data_ptr()
            rc = lib.gpud_launch_freq_shift_stream_cuda(x, sh, n, q["inc"], q["start"], q["stream"])
            rc = rc or lib.gpud_launch_fir_v2_stream_cuda(sh, flt, q["taps"].data_ptr(), n, c["taps"], q["stream"])
            rc = rc or lib.gpud_launch_decimate_stream_cuda(flt, dec, n // c["decim"], c["decim"], q["stream"])
            if rc != 0:
                raise RuntimeError("slot: %d" % rc)
        for q in s["slots"]:
            if lib.gpud_stream_sync(q["stream"]) != 0:
                raise RuntimeError("slot sync")
        return [q["dec"] for q in s["slots"]]
    if kind == "pilot":
        got = s["det"].run(s["iq"], s["rates"])
        return {"present": np.array([g["present"] for g in got], np.int64),
                "bin": np.array([g["best_bin"] for g in got], np.int64),
                "ratio": np.array([g["ratio"] for g in got]), "median": np.array([g["median"] for g in got])}
    if kind == "rds":
        got = s["dec"].run(s["jobs"])
        return {"counts": np.array([(g["groups"], g["groups_total"], g["status"], g["pi"]) for g in got], np.int64),
                "text": np.frombuffer("".join(g["ps"].ljust(8) + g["rt"].ljust(64) for g in got).encode(), np.uint8)}
    if kind == "welch":
        return s["sp"].welch(s["iq"], s["case"]["fft"])
    c = s["case"]
    if c["mode"] == "BATCH":
        return G.wfm_batch_audio(s["iq"], c["fs"], s["off"], s["bw"])[0]
    return G.demod_audio_segment(G.MODE_BY_NAME[c["mode"]], s["iq"], c["fs"], s["off"], s["bw"])[0]


# --------------------------------------------------------------------------
# work
# --------------------------------------------------------------------------

def _channel_work(kind, T, D, n, fs, pcm, emit):
    m = n // D
    flops = 4.0 * T * m + min(6.0 * n, 4.0 * T * m) + 6.0 * m
    out = 8.0 * m if emit else 0.0
    rate, ch = fs / D, 1
    if kind == "WFM":
        dr = max(1, int(rate) // 19_000)
        ch = 2
        flops += (4 * 202 + 36 + 2) * m + 404.0 * (m // dr)
        out += 8.0 * (m // dr)
    if pcm:
        frames = m * 48_000 / rate
        flops += frames * ch * 70
        out += frames * ch * (2 if pcm == 1 else 4)
    else:
        out += 4.0 * ch * m
    return flops, out + 8.0 * T


def work(case):
    k = case["kind"]
    if k == "runner":
        f = b = 0.0
        for c in _population(case):
            df, db = _channel_work(c["kind"], c["T"], c["D"], case["block"], case["fs"], case["pcm"], case["emit_iq"])
            f, b = f + df, b + db
        return {"bytes": 8.0 * case["block"] + b, "flops": f}
    if k == "extract":
        f = b = 0.0
        for i in range(case["jobs"]):
            m, T = case["n"] // (8 if i % 4 == 0 else 20), case["taps"]
            f, b = f + 4.0 * T * m + min(6.0 * case["n"], 4.0 * T * m), b + 8.0 * m + 16.0 * T
        return {"bytes": 8.0 * case["n"] + b, "flops": f}
    if k == "launcher":
        m = case["n"] // case["decim"]
        return {"bytes": 8.0 * (case["n"] + m + 2 * case["taps"]), "flops": 4.0 * case["taps"] * m + 6.0 * case["n"]}
    if k == "slots":
        # the shifted and the filtered block are outputs of their calls
        m = case["n"] // case["decim"]
        return {"bytes": case["jobs"] * 8.0 * (5 * case["n"] + m), "flops": case["jobs"] * case["n"] * (6.0 + 4.0 * case["taps"])}
    if k == "pilot":
        n = min(case["n"], case["fs"] // 2)
        return {"bytes": case["stations"] * 8.0 * n,
                "flops": case["stations"] * (40.0 * n + 201 * 4.0 * min(n, case["fs"] // math.gcd(case["fs"], 10)))}
    if k == "rds":
        return {"bytes": case["stations"] * 8.0 * case["n"], "flops": case["stations"] * case["n"] * 1187.5 / case["fs"] * 200}
    if k == "welch":
        n = case["fft"]
        return {"bytes": 8.0 * (n + (case["segs"] - 1) * (n // 2)) + 8.0 * n, "flops": case["segs"] * 5.0 * n * math.log2(n)}
    m = case["n"] / _factor(case["fs"], 192_000 if case["mode"] in ("BATCH", "WFM_STEREO") else 48_000)
    return {"bytes": 8.0 * case["n"] + 8.0 * m * 0.25, "flops": m * (8.0 * 101 + 1000.0)}


# --------------------------------------------------------------------------
# the same in 64 bits
# --------------------------------------------------------------------------

def _lowpass(cutoff, fs, taps):
    """Hann-windowed sinc of odd length, float64."""
    taps |= 1
    fc, m = cutoff / fs, (taps - 1) / 2.0
    i = np.arange(taps)
    x = i - m
    with np.errstate(invalid="ignore", divide="ignore"):
        sinc = np.where(x == 0, 2 * fc, np.sin(TWO_PI * fc * x) / (math.pi * x))
    return sinc * 0.5 * (1 - np.cos(TWO_PI * i / (taps - 1)))


def _taps32(bw, fs, T):
    """The extraction filter: designed in 64 bits, defined by its 32-bit taps."""
    return _lowpass(max(bw / 2, 200.0), fs, T).astype(np.float32)[:T]


def _extract64(x, fs, offs, h, D, n0, count, first=0.0):
    """Rows of outputs for the offsets: sum_k h[k] s(n0 + j D - k), s the input
    (zero before it begins) turned by -2 pi off (n + first) / fs."""
    T = len(h)
    pad = torch.cat([torch.zeros(T, dtype=torch.complex128, device=DEV), x.to(torch.complex128)])
    k = torch.arange(T, dtype=torch.float64, device=DEV)
    hd = torch.as_tensor(np.asarray(h, np.float64), device=DEV)
    w = torch.as_tensor([o / fs for o in offs], dtype=torch.float64, device=DEV)

    def turn(n):
        ph = torch.outer(w, n)
        return torch.exp(-1j * TWO_PI * (ph - torch.floor(ph)))

    g = (hd * turn(-k)).flip(1).T.contiguous()  # oldest sample first
    out, step = [], max(1, (1 << 24) // T)
    for j in range(0, count, step):
        m = min(step, count - j)
        win = pad.as_strided((m, T), (D, 1), n0 + j * D - (T - 1) + T)
        n = n0 + (j + torch.arange(m, dtype=torch.float64, device=DEV)) * D
        out.append((win @ g).T * turn(n + first))
    return torch.cat(out, 1) if out else torch.zeros(len(offs), 0, dtype=torch.complex128, device=DEV)


def _fir64(x, taps):
    """Rows of x (zero before they begin) through the taps."""
    t = torch.as_tensor(np.ascontiguousarray(taps[::-1]), dtype=torch.float64, device=DEV)
    pad = torch.cat([torch.zeros(x.shape[0], len(taps) - 1, dtype=x.dtype, device=DEV), x], 1)
    return torch.stack([r.unfold(0, len(taps), 1) @ t.to(x.dtype) for r in pad])


def _disc64(iq):
    return torch.angle(iq[:, 1:] * iq[:, :-1].conj())


class _Loop64:
    """Pilot loops of several channels, serial, with the lock decision."""

    def __init__(self, count, rate):
        theta = (50.0 / rate) / (0.707 + 0.25 / 0.707)
        d = 1 + 2 * 0.707 * theta + theta * theta
        self.rate, self.a, self.b = rate, 4 * 0.707 * theta / d, 4 * theta * theta / d
        self.lpa = 1 - math.exp(-TWO_PI * 200 / rate)
        self.ph, self.fq = np.zeros(count), np.full(count, TWO_PI * 19_000 / rate)
        self.I, self.Q, self.ea = np.zeros(count), np.zeros(count), np.zeros(count)
        self.on, self.off = np.zeros(count, int), np.zeros(count, int)
        self.enabled = np.zeros(count, bool)

    def block(self, pilot):
        p = np.ascontiguousarray(pilot.cpu().numpy().T)
        if p.shape[1] == 1:
            return self._one(p[:, 0].tolist())
        n, lo, hi = p.shape[0], TWO_PI * 17_000 / self.rate, TWO_PI * 21_000 / self.rate
        ph, fq, I, Q, es = self.ph, self.fq, self.I, self.Q, np.zeros_like(self.ph)
        a, b, lpa = self.a, self.b, self.lpa
        track = np.empty_like(p)
        for i in range(n):
            z = p[i]
            I = I + lpa * (z * np.cos(ph) - I)
            Q = Q + lpa * (-z * np.sin(ph) - Q)
            e = np.arctan2(Q, I)
            fq = np.minimum(np.maximum(fq + b * e, lo), hi)
            ph = ph + fq + a * e
            ph -= TWO_PI * (ph > TWO_PI)
            es += np.abs(e)
            track[i] = ph
        self.ph, self.fq, self.I, self.Q = ph, fq, I, Q
        self.es, self.pp, self.n = es, (p * p).sum(0), n
        return torch.from_numpy(np.ascontiguousarray(track.T)).to(DEV)

    def _one(self, p):
        """block() of a single channel, in plain floats."""
        lo, hi = TWO_PI * 17_000 / self.rate, TWO_PI * 21_000 / self.rate
        ph, fq, I, Q = (float(v[0]) for v in (self.ph, self.fq, self.I, self.Q))
        a, b, lpa, es, track = self.a, self.b, self.lpa, 0.0, []
        for z in p:
            I += lpa * (z * math.cos(ph) - I)
            Q += lpa * (-z * math.sin(ph) - Q)
            e = math.atan2(Q, I)
            fq = min(max(fq + b * e, lo), hi)
            ph += fq + a * e
            if ph > TWO_PI:
                ph -= TWO_PI
            es += abs(e)
            track.append(ph)
        self.ph, self.fq, self.I, self.Q, self.es = (np.array([v]) for v in (ph, fq, I, Q, es))
        self.pp, self.n = np.array([sum(z * z for z in p)]), len(p)
        return torch.tensor(track, dtype=torch.float64, device=DEV)[None]

    def decide(self):
        self.ea = 0.9 * self.ea + 0.1 * self.es / self.n
        coh = (self.I ** 2 + self.Q ** 2) * self.n / np.maximum(self.pp, 1e-12)
        lock = (coh > 0.15) & (np.abs(self.fq * self.rate / TWO_PI - 19_000) < 250) & (self.ea < 0.35)
        self.on = np.where(lock, self.on + 1, 0)
        self.off = np.where(lock, 0, self.off + 1)
        self.enabled = (self.enabled | (self.on >= 4)) & ~(self.off >= 10)


def _resampler(rate):
    g = math.gcd(rate, 48_000)
    L, M = 48_000 // g, rate // g
    plen = (L * 32) | 1
    K = -(-plen // L)
    mid, fc = (plen - 1) / 2.0, 0.90 / max(L, M)
    n = np.arange(L * K)
    x = n - mid
    sn = np.where(x == 0, TWO_PI * fc, np.sin(TWO_PI * fc * x) / np.where(x == 0, 1, x))
    arm = np.where(n < plen, sn * np.i0(6.0 * np.sqrt(np.maximum(0.0, 1 - (x / mid) ** 2))) / np.i0(6.0) * L, 0.0)
    return L, M, K, arm.reshape(K, L).T.copy()


def _resample_plan(L, M, sizes):
    """(start counter, frames) of every call of the stateful resampler."""
    t, plan = 0, []
    for n in sizes:
        if L == M:
            plan.append((0, n))
            continue
        top = -(-((n + 1) * L - t) // M) - 1
        last = max(0, min(top, -(-(n * L - t) // M))) if top >= 0 else -1
        used = (t + last * M) // L if last >= 0 else 0
        plan.append((t, last + 1))
        t = t + (last + 1) * M - n * L - (L if used < n else 0)
    return plan


def _audio48(x, sizes, rate, wide, tau=50e-6, gain=0.35):
    """48 kHz audio of the last of the calls of `sizes` frames: rows of x hold
    the demodulated stream of one audio channel each."""
    L, M, K, arm = _resampler(rate)
    plan = _resample_plan(L, M, sizes)
    if not wide:  # no recursion behind it: the last call alone
        at, calls = sum(sizes[:-1]), [(plan[-1], sizes[-1])]
    else:
        at, calls = 0, list(zip(plan, sizes))
    pad = torch.cat([torch.zeros(x.shape[0], K, dtype=torch.float64, device=DEV), x], 1)
    a = math.exp(-1.0 / (48_000 * tau)) if wide and tau else 0.0
    y = np.zeros(x.shape[0])
    for (t, frames), n in calls:
        pos = t + torch.arange(frames, dtype=torch.int64, device=DEV) * M
        c = torch.div(pos, L, rounding_mode="floor")
        if L == M:
            z = x[:, at:at + frames].clone()
        else:
            taps = torch.as_tensor(arm, device=DEV)[pos - c * L]
            idx = (at + c - 1 + K)[:, None] - torch.arange(K, device=DEV)[None, :]
            z = torch.stack([(r[idx] * taps).sum(1) for r in pad])
        at += n
        if a:
            u = z.cpu().numpy().T
            v = np.empty_like(u)
            for i in range(frames):
                y = a * y + (1 - a) * u[i]
                v[i] = y
            z = torch.from_numpy(v.T.copy()).to(DEV)
    return z * gain if wide else z


def _wide64(iq, sizes, rate, pcm):
    """(audio of the last call, RDS baseband of the last call) of broadcast
    channels: rows of iq hold the extracted stream, sizes the calls' counts."""
    d = _disc64(iq)
    sizes = [sizes[0] - 1] + list(sizes[1:])
    last = sizes[-1]
    t15 = _lowpass(15_000, rate, 101)
    lpr, bpf = _fir64(d, t15), _fir64(d, _lowpass(53_000, rate, 101) - _lowpass(23_000, rate, 101))
    pil = _fir64(d, _lowpass(21_000, rate, 101) - _lowpass(17_000, rate, 101))
    loop, at, lr, left, right = _Loop64(d.shape[0], rate), 0, torch.zeros_like(d), [], []
    mono_hist = torch.zeros(d.shape[0], 100, dtype=torch.float64, device=DEV)
    for n in sizes:
        s = slice(at, at + n)
        lr[:, s] = bpf[:, s] * 2 * torch.sin(2 * loop.block(pil[:, s]))
        loop.decide()
        lo = max(0, at - 100)
        diff = _fir64(lr[:, lo:at + n], t15)[:, at - lo:]
        mono = _fir64(torch.cat([mono_hist, d[:, s]], 1), t15)[:, 100:]
        on = torch.from_numpy(loop.enabled).to(DEV)[:, None]
        mono_hist = torch.where(on, mono_hist, torch.cat([mono_hist, d[:, s]], 1)[:, -100:])
        left.append(torch.where(on, 0.5 * (lpr[:, s] + diff), mono))
        right.append(torch.where(on, 0.5 * (lpr[:, s] - diff), mono))
        at += n
    left, right = torch.cat(left, 1), torch.cat(right, 1)
    if pcm:
        z = [_audio48(v, sizes, rate, True) for v in (left, right)]
    else:
        z = [v[:, -last:] for v in (left, right)]
    audio = torch.stack(z, 2).reshape(d.shape[0], -1)
    # RDS: the reference adds its phase step one sample at a time
    total = d.shape[1]
    ph = torch.from_numpy(np.cumsum(np.full(total, TWO_PI * 57_000.0 / rate))).to(DEV)
    dr = max(1, rate // 19_000)
    keep = [i for i in range(0, total, dr) if i >= total - last]
    lo = max(0, keep[0] - 100) if keep else 0
    c = d[:, lo:] * torch.exp(1j * ph[lo:])
    rds = _fir64(c, _lowpass(7_500, rate, 101))[:, torch.as_tensor(keep, device=DEV).long() - lo] if keep else None
    return audio, rds


def _narrow64(kind, iq, sizes, rate, pcm):
    """Audio of the last call of narrow channels; iq: rows of the last calls'
    extracted samples with one sample before them for the discriminator."""
    out, at = [], 1
    for n in sizes:
        z = iq[:, at:at + n]
        if kind == "NFM":
            out.append(_disc64(iq[:, at - 1:at + n]))
        elif kind == "AM":
            out.append(z.abs() - z.abs().mean(1, keepdim=True))
        else:
            ph = (torch.arange(n, dtype=torch.float64, device=DEV) + 1) * (TWO_PI * (-700.0 if kind == "LSB" else 700.0) / rate)
            out.append(z.real * torch.cos(ph) - (0 if kind == "CW" else 1) * z.imag * torch.sin(ph))
        at += n
    return out


def _exact_runner(case, seed):
    if case["pcm"] == 1:
        return None  # whole numbers
    x, chans = _scene(case, seed)
    fs, n, total = case["fs"], case["block"], WARM_BLOCKS + 1
    x = torch.cat([x] * -(-total // PERIOD[case["mix"]]))[:total * n]
    groups = {}
    for c in chans:
        groups.setdefault((c["kind"], c["T"], c["D"]), []).append(c)
    headroom, out, flat = case["mix"] == "headroom", {}, {}
    wide = {}
    for i, ((kind, T, D), cs) in enumerate(groups.items()):
        rate, h = fs // D, _taps32(cs[0]["bw"], fs, T)
        ends = [(b + 1) * n // D for b in range(total)]
        sizes = [e - s for e, s in zip(ends, [0] + ends[:-1])]
        offs = [c["off"] for c in cs]
        name = "%d_%s" % (i, kind)
        if kind == "WFM":
            iq = torch.cat([_extract64(x, fs, offs[j:j + 64], h, D, D - 1, ends[-1]) for j in range(0, len(offs), 64)])
            wide.setdefault((D, rate), []).append((name, iq, sizes))
            continue
        # narrow: enough calls before the last one for the resampler's memory
        back = total - 1
        while back > 1 and ends[-2] - ends[back - 1] < 64:
            back -= 1
        back = max(1, back if case["pcm"] else total - 1)
        start = ends[back - 1] - 1
        iq = _extract64(x, fs, offs, h, D, D - 1 + start * D, ends[-1] - start)
        audio = _narrow64(kind, iq, sizes[back:], rate, case["pcm"])
        if case["pcm"]:
            # the resampler's counter runs over all calls, its memory over the last ones
            before = sum(sizes[:back]) - (1 if kind == "NFM" else 0)
            z = torch.cat([torch.zeros(len(cs), before, dtype=torch.float64, device=DEV)] + audio, 1)
            calls = [sizes[0] - (1 if kind == "NFM" else 0)] + sizes[1:]
            got = {"pcm": _audio48(z, calls, rate, False)}
        else:
            got = {"audio": audio[-1]}
        if case["emit_iq"]:
            got["iq"] = iq[:, -sizes[-1]:]
        out[name] = got
        if headroom:
            flat.setdefault(kind + "_audio", []).append(got["audio"].reshape(-1))
    for (D, rate), parts in wide.items():
        iq = torch.cat([p[1] for p in parts])
        audio, rds = _wide64(iq, parts[0][2], rate, case["pcm"])
        at = 0
        for name, p, sizes in parts:
            rows = slice(at, at + p.shape[0])
            out[name] = {("pcm" if case["pcm"] else "audio"): audio[rows], "rds": None if rds is None else rds[rows]}
            if case["emit_iq"]:
                out[name]["iq"] = p[:, -sizes[-1]:]
            at += p.shape[0]
        if headroom:
            flat.setdefault("WFM_audio", []).append(audio.reshape(-1))
            flat.setdefault("WFM_rds", []).append(rds.reshape(-1))
    return {k: torch.cat(v) for k, v in flat.items()} if headroom else out


def _exact_pilot(case, seed):
    n, fs = min(case["n"], case["fs"]), case["fs"]
    ratio, median = [], []
    for z in _baseband(seed, case["stations"], n, fs):
        z = z[max(0, n - fs // 2):].to(torch.complex128)
        d = torch.angle(z[1:] * z[:-1].conj())
        i = torch.arange(d.numel(), dtype=torch.int64, device=DEV)
        mags = []
        for b in range(201):
            ph = torch.remainder(i * (18_000 + 10 * b), fs).to(torch.float64) * (TWO_PI / fs)
            mags.append(torch.hypot((d * torch.cos(ph)).sum(), (d * torch.sin(ph)).sum()))
        m = torch.stack(mags).sort().values
        ratio.append(float(m[-1] / m[100]))
        median.append(float(m[100]))
    return {"present": None, "bin": None, "ratio": np.array(ratio), "median": np.array(median)}


def _exact_event(case, seed):
    off, bw, x = _event_setup(case, seed)
    fs, mode = case["fs"], case["mode"]
    wide = mode in ("BATCH", "WFM_STEREO")
    D = _factor(fs, 192_000 if wide else 48_000)
    rate = fs // D
    cut = max(bw / 2, 75_000.0) if wide else max(bw / 2, 200.0)
    h = _lowpass(cut, fs, 101).astype(np.float32)
    # the shift turns before it is used, the first output is input 0
    iq = _extract64(x, fs, [off], h, D, 0, -(-case["n"] // D), first=1.0)
    if mode == "BATCH":
        # one call: the lock by the pilot band's share of the power, the
        # discriminator output itself on both channels without it
        d = _disc64(iq)
        t15, loop = _lowpass(15_000, rate, 101), _Loop64(1, rate)
        lpr, bpf = _fir64(d, t15), _fir64(d, _lowpass(53_000, rate, 101) - _lowpass(23_000, rate, 101))
        pil = _fir64(d, _lowpass(21_000, rate, 101) - _lowpass(17_000, rate, 101))
        diff = _fir64(bpf * 2 * torch.sin(2 * loop.block(pil)), t15)
        n = d.shape[1]
        if loop.pp[0] / float((d * d).sum()) > 0.003 and abs(loop.fq[0] * rate / TWO_PI - 19_000) < 250 \
                and loop.es[0] / n < 0.35:
            d = torch.cat([0.5 * (lpr + diff), 0.5 * (lpr - diff)])
        else:
            d = torch.cat([d, d])
        return _audio48(d, [n], rate, True).T.reshape(-1)
    if not wide:
        pad = torch.cat([torch.zeros(1, 1, dtype=torch.complex128, device=DEV), iq], 1)
        z = _narrow64(mode, pad, [iq.shape[1]], rate, 0)[0] if mode != "NFM" else _disc64(iq)
    else:
        d = _disc64(iq)
        t15 = _lowpass(15_000, rate, 101)
        ph = torch.from_numpy(np.cumsum(np.full(d.shape[1], TWO_PI * 38_000.0 / rate))).to(DEV)
        lr = _fir64(d, _lowpass(53_000, rate, 101) - _lowpass(23_000, rate, 101)) * 2 * torch.cos(ph)
        lpr, diff = _fir64(d, t15), _fir64(lr, t15)
        z = torch.cat([0.5 * (lpr + diff), 0.5 * (lpr - diff)])
    if rate > 48_000:
        d2 = _factor(rate, 48_000)
        frames = z.shape[1] // d2 if wide else -(-z.shape[1] // d2)
        z = _fir64(z, _lowpass(0.9 * 24_000, rate, 63))[:, ::d2][:, :frames]
    return z.T.reshape(-1)


def exact(case, seed):
    kind, seed = case["kind"], int(seed)
    if kind == "runner":
        return _exact_runner(case, seed)
    if kind == "extract":
        x = _live(case, seed, case["n"])
        out = []
        for j in _jobs(case, _rng(seed, 22)):
            D = case["fs"] // j.OutRate
            out.append(_extract64(x, case["fs"], [j.OffsetHz], _taps32(j.Bandwidth, case["fs"], case["taps"]), D, D - 1,
                                  case["n"] // D)[0])
        return out
    if kind == "launcher":
        off, h, x = _launcher_setup(case, seed)
        D, T, n = case["decim"], case["taps"], case["n"]
        one = np.ones(1)
        hist = _extract64(x, case["fs"], [off], one, 1, n - (T - 1), T - 1)[0]
        return (_extract64(x, case["fs"], [off], h, D, D - 1, n // D)[0], hist, None, None)
    if kind == "slots":
        offs, starts, h, x = _slot_setup(case, seed)
        D, fs = case["decim"], case["fs"]
        return [_extract64(x, fs, [o], h, D, 0, case["n"] // D)[0] * complex(math.cos(p), math.sin(p))
                for o, p in zip(offs, starts)]
    if kind == "pilot":
        return _exact_pilot(case, seed)
    if kind == "rds":
        return None
    if kind == "welch":
        n = case["fft"]
        x = _live({"fs": 4_096_000}, seed, n + (case["segs"] - 1) * (n // 2)).to(torch.complex128)
        w = 0.5 * (1 - torch.cos(TWO_PI * torch.arange(n, dtype=torch.float64, device=DEV) / (n - 1)))
        p = torch.stack([(torch.fft.fft(x[s * (n // 2):s * (n // 2) + n] * w).abs() / n) ** 2
                         for s in range(case["segs"])]).mean(0)
        return torch.fft.fftshift(10 * torch.log10(p + 1e-24))
    return _exact_event(case, seed)
