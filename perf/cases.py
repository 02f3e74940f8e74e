"""The conversions that a user of this framework runs, as measured cases.

Each case goes through a public entry point of the package (Encoder,
BatchPlan, DiffEngine, FirChain, TrellisSdm) with the parameters of the
package's own configurations and tests.  A pass converts one whole input: a
track, a player's block, a batch of tracks or a training step.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from foo_dsd_trellis_gb300 import _lib, ntf, signals
from foo_dsd_trellis_gb300.batch import OUT_DOP, BatchPlan, StreamSpec
from foo_dsd_trellis_gb300.diff import DiffConfig, DiffEngine
from foo_dsd_trellis_gb300.fir import FirChain
from foo_dsd_trellis_gb300.pipeline import (FULL_PARALLEL, OUT_BITS, PCM_FIR_GAIN, SEG0_FIRST,
                                            Encoder)
from foo_dsd_trellis_gb300.sdm import TrellisSdm

DEV = "cuda:0"
PATH_GAIN = float(np.float32(0.708))    # the gain of the engine's DSD -> DSD rows
DSD64 = 2822400


def listed():
    return [
        # a stereo track offline at the highest quality: PCM 48 kHz -> DSD128,
        # K = 32, depth 64 (the package's headline configuration)
        dict(name="encode_dsd128_k32", kind="encode", fs_in=48000, fs_out=6144000, ch=2,
             frames=480000, ntf="clans-7", cands=32, depth=64, lat=128, seg=65536, nsegs=0,
             seed_mode="parallel", conv=0),
        # a track at the engine's default for paths that its table does not
        # list: PCM 44.1 kHz -> DSD64, K = 4, depth 8, lat 32
        dict(name="encode_dsd64_k4", kind="encode", fs_in=44100, fs_out=2822400, ch=2,
             frames=220500, ntf="auto", cands=4, depth=8, lat=32, seg=65536, nsegs=0,
             seed_mode="parallel", conv=0),
        # 5.1 with room correction: 48 kHz -> DSD512, a 65,536-tap response per
        # channel, K = 16, depth 48
        dict(name="encode_dsd512_conv_6ch", kind="encode", fs_in=48000, fs_out=24576000, ch=6,
             frames=48000, ntf="auto", cands=16, depth=48, lat=32, seg=262144, nsegs=0,
             seed_mode="parallel", conv=65536),
        # one 200 ms batch of a player below DSD512, in the reference's own
        # seeding order (segment 0 first, then the 16-level estimator), 8 segments
        dict(name="player_batch_seg0first", kind="encode", fs_in=44100, fs_out=2822400, ch=2,
             frames=8820, ntf="auto", cands=4, depth=8, lat=32, seg=0, nsegs=8,
             seed_mode="seg0", conv=0),
        # a DSD128 track re-encoded at its own rate: the path table's row
        # CLANS-6, K = 2, depth 4, boxcar pre-filter
        dict(name="redsd_same128_k2", kind="redsd", fs_in=5644800, fs_out=5644800, ch=2,
             frames=3528000, ntf="clans-6", cands=2, depth=4, lat=128, seg=65536, lowpass=False),
        # a DSD128 track decimated to 44.1 kHz PCM
        dict(name="dsd2pcm_track", kind="dsd2pcm", fs_in=5644800, fs_out=44100, ch=2,
             frames=3528000),
        # a player's 10 ms block of DSD64 decimated to 176.4 kHz PCM: launches
        # and host work count
        dict(name="dsd2pcm_block", kind="dsd2pcm", fs_in=2822400, fs_out=176400, ch=2,
             frames=1764),
        # a second of PCM 44.1 kHz -> DSD128 with the greedy PreCorr modulator
        dict(name="precorr_dsd128", kind="precorr", fs_in=44100, fs_out=5644800, ch=2,
             frames=44100, limit=12.0),
        # a library conversion: many stereo streams of mixed rates and lengths
        # in one plan, DSD128 and DSD256, K = 32, depth 64
        dict(name="batch_mixed_k32", kind="batch", streams=16, scale=0.06, cands=32, depth=64,
             seg=65536),
        # a training step of the pre-emphasis taps and the loop filter: exact
        # forward and adjoint over 16 clips
        dict(name="train_step", kind="train", clips=16, frames=512, cands=32, depth=64, lat=128),
        # the offline encoder's filter stage alone: 44.1 kHz -> DSD256, stereo
        dict(name="fir_dsd256", kind="fir", fs_in=44100, fs_out=11289600, ch=2, frames=88200,
             boxcar=0, clip=False),
        # a block through the sequential modulator (no segments) with the
        # command-line encoder's defaults K = 8, depth 4, lat 256
        dict(name="sdm_block_k8", kind="sdm", order_of="auto", rate=2822400, ch=2, count=4096,
             cands=8, depth=4, lat=256),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["encode", "encode", "seg0", "redsd", "redsd", "dsd2pcm", "dsd2pcm",
                       "precorr", "batch", "train", "fir", "sdm"])
    ch = rng.choice([1, 2, 2, 2, 3, 6])
    if kind == "encode":
        fs, mult = rng.choice([(44100, 64), (48000, 64), (44100, 128), (48000, 128), (88200, 64),
                               (44100, 256), (96000, 128)])
        k, depth = rng.choice([(2, 4), (3, 8), (4, 8), (6, 16), (8, 32), (12, 32), (16, 48),
                               (24, 64), (32, 64), (32, 64)])
        # samples over all channels: at most the headline's
        total = _log_int(rng, 2.0e6, 6.0e7)
        return dict(kind="encode", fs_in=fs, fs_out=fs * mult, ch=ch,
                    frames=max(64, total // (mult * ch)), ntf=rng.choice(["auto", "clans-7", "sdm-6"]),
                    cands=k, depth=depth, lat=rng.choice([32, 100, 128, 256]),
                    seg=rng.choice([32768, 65536, 50000, 131072]), nsegs=0, seed_mode="parallel",
                    conv=rng.choice([0, 0, 0, 5000, 65536]))
    if kind == "seg0":
        fs, mult = rng.choice([(44100, 64), (48000, 64), (88200, 32)])
        return dict(kind="encode", fs_in=fs, fs_out=fs * mult, ch=rng.choice([1, 2, 2, 6]),
                    frames=_log_int(rng, 100000, 700000) // mult, ntf="auto",
                    cands=rng.choice([2, 4, 8]), depth=8, lat=32, seg=0, nsegs=rng.choice([2, 4, 8]),
                    seed_mode="seg0", conv=0)
    if kind == "redsd":
        fi, fo = rng.choice([(DSD64, DSD64), (2 * DSD64, 2 * DSD64), (2 * DSD64, 2 * DSD64),
                             (4 * DSD64, 2 * DSD64), (DSD64, 2 * DSD64)])
        k, depth = rng.choice([(1, 4), (2, 4), (2, 8), (2, 8), (4, 8), (8, 16)])
        total = _log_int(rng, 2.0e6, 1.1e8)
        return dict(kind="redsd", fs_in=fi, fs_out=fo, ch=ch,
                    frames=max(4096, total * fi // fo // (16 * ch)), ntf=rng.choice(["clans-6", "sdm-6", "sdm-8"]),
                    cands=k, depth=depth, lat=rng.choice([64, 128]),
                    seg=rng.choice([32768, 65536]), lowpass=bool(fi == fo and rng.random() < 0.4))
    if kind == "dsd2pcm":
        fi = DSD64 * rng.choice([1, 2, 4])
        return dict(kind="dsd2pcm", fs_in=fi, fs_out=44100 * rng.choice([1, 2, 4, 8]), ch=ch,
                    frames=_log_int(rng, 882, 7000000 // ch))
    if kind == "precorr":
        fs, mult = rng.choice([(44100, 64), (48000, 64), (44100, 128), (96000, 64)])
        return dict(kind="precorr", fs_in=fs, fs_out=fs * mult, ch=rng.choice([1, 2, 6, 40]),
                    frames=_log_int(rng, 441, 5600000 // mult), limit=rng.choice([0.0, 12.0]))
    if kind == "batch":
        k, depth = rng.choice([(32, 64), (32, 64), (16, 32), (4, 8)])
        return dict(kind="batch", streams=rng.randint(5, 16), scale=rng.uniform(0.01, 0.05), cands=k,
                    depth=depth, seg=rng.choice([32768, 65536]))
    if kind == "train":
        return dict(kind="train", clips=rng.choice([3, 8, 16, 24]), frames=32 * rng.randint(8, 20),  # whole checkpoints
                    cands=rng.choice([8, 16, 32]), depth=rng.choice([32, 64]),
                    lat=rng.choice([64, 128]))
    if kind == "fir":
        fs, mult = rng.choice([(44100, 64), (48000, 128), (44100, 256), (88200, 64), (176400, 16),
                               (48000, 512), (192000, 32)])
        return dict(kind="fir", fs_in=fs, fs_out=fs * mult, ch=ch,
                    frames=_log_int(rng, 100, 4.4e7 / mult / ch), boxcar=rng.choice([0, 8]),
                    clip=rng.random() < 0.5)
    return dict(kind="sdm", order_of=rng.choice(["auto", "clans-7", "sdm-5"]), rate=DSD64,
                ch=rng.choice([1, 2, 6, 64]), count=_log_int(rng, 500, 40000),
                cands=rng.choice([1, 2, 4, 5, 8, 16, 32]), depth=rng.choice([4, 8, 32]),
                lat=rng.choice([32, 100, 256]))


# ---- inputs ----

def _music(ch, n, fs, seed):
    """Tones over pink noise, a few dB below full scale, float32 [ch, n]."""
    out = np.empty((ch, n), np.float32)
    for c in range(ch):
        rng = np.random.Generator(np.random.PCG64([seed, c]))
        out[c] = (signals.multitone(n, fs, rng, ntones=12, level_db=-20.0)
                  + signals.pink_noise(n, rng, signals.db_to_amp(-30.0))).astype(np.float32)
    return torch.from_numpy(out).to(DEV)


def _dop(ch, frames, rate, seed):
    """DoP frames [ch, frames] of a modulated DSD stream of this rate."""
    base = 44100
    mult = rate // base
    n = 16 * frames
    lat = 32
    pcm = _music(ch, -(-(n + 200000) // mult), base, seed)
    f = ntf.get_filter("clans-6", rate)
    enc = Encoder(base, rate, ch, f, 4, 2, lat, seg_len=32768, output_format=OUT_BITS)
    bits = torch.empty((ch, pcm.shape[1] * mult + 256), dtype=torch.uint8, device=DEV)
    ns, _ = enc.process(pcm, bits)
    enc.close()
    if ns < n:
        raise ValueError("the source came out short")
    w = (2 ** torch.arange(15, -1, -1, device=DEV, dtype=torch.int32))
    out = torch.empty((ch, frames), dtype=torch.float32, device=DEV)
    marker = torch.where(torch.arange(frames, device=DEV) % 2 == 0, 0x05, 0xFA - 256) << 16
    for c in range(ch):
        word = (bits[c, :n].reshape(frames, 16).to(torch.int32) * w).sum(1)
        out[c] = (marker + word).to(torch.float32) / 8388608.0
    return out


def _filter(name, rate):
    return ntf.auto_select(rate) if name == "auto" else ntf.get_filter(name, rate)


def _room(taps, ch, fs, seed):
    out = np.empty((ch, taps), np.float32)
    for c in range(ch):
        rng = np.random.Generator(np.random.PCG64([seed, 77, c]))
        h = rng.standard_normal(taps) * 10.0 ** (-3.0 * np.arange(taps) / (0.4 * fs))
        out[c] = h / np.abs(np.fft.rfft(h, 4 * taps)).max()
    return out


def prepare(case, seed):
    c = dict(case)
    kind = c["kind"]
    torch.cuda.set_device(0)
    st = {"case": c, "kind": kind}
    if kind in ("encode", "precorr"):
        st["x"] = _music(c["ch"], c["frames"], c["fs_in"], seed)
        st["gain"] = PCM_FIR_GAIN
        if kind == "encode":
            f = _filter(c["ntf"], c["fs_out"])
            st["enc"] = Encoder(c["fs_in"], c["fs_out"], c["ch"], f, c["depth"], c["cands"],
                                c["lat"], seg_len=c["seg"], nsegs=c["nsegs"],
                                seed_mode=SEG0_FIRST if c["seed_mode"] == "seg0" else FULL_PARALLEL)
            if c["conv"]:
                st["enc"].set_conv(_room(c["conv"], c["ch"], c["fs_out"], seed), 4096)
        else:
            f = ntf.auto_select_precorr(c["fs_out"])
            st["enc"] = Encoder(c["fs_in"], c["fs_out"], c["ch"], f, 64, 32, 128,
                                state_limit=c["limit"], soft_clip=False,
                                sdm_mode=_lib.SDM_PRECORR)
    elif kind in ("redsd", "dsd2pcm"):
        st["x"] = _dop(c["ch"], c["frames"], c["fs_in"], seed)
        if kind == "redsd":
            st["gain"] = PATH_GAIN
            f = _filter(c["ntf"], c["fs_out"])
            st["enc"] = Encoder(c["fs_in"], c["fs_out"], c["ch"], f, c["depth"], c["cands"],
                                c["lat"], seg_len=c["seg"], boxcar_taps=0, soft_clip=False,
                                samerate_filter=_lib.SAMERATE_LOWPASS if c["lowpass"]
                                else _lib.SAMERATE_BOXCAR)
        else:
            st["gain"] = 1.0
            f = ntf.get_filter("clans-7", c["fs_in"])
            st["enc"] = Encoder(c["fs_in"], c["fs_out"], c["ch"], f, 64, 32, 128,
                                output_format=_lib.OUT_PCM)
    elif kind == "batch":
        lay = signals.multistream_layout(c["streams"], scale=c["scale"])
        specs = []
        for e in lay:
            f = ntf.auto_select(e["fs_out"])
            specs.append(StreamSpec(e["fs_in"], e["fs_out"], e["channels"], e["frames"], f,
                                    cands=c["cands"], depth=c["depth"], lat=128,
                                    gain=PCM_FIR_GAIN))
        st["plan"] = BatchPlan(specs, seg_len=c["seg"], output_format=OUT_DOP)
        st["xs"] = [_music(e["channels"], e["frames"], e["fs_in"], seed * 100 + i)
                    for i, e in enumerate(lay)]
    elif kind == "train":
        cfg = DiffConfig(nclips=c["clips"], frames=c["frames"], cands=c["cands"],
                         depth=c["depth"], lat=c["lat"])
        f = ntf.get_filter("clans-7", cfg.fs_out)
        st["eng"] = DiffEngine(cfg, f, 0)
        st["x"] = _music(c["clips"], c["frames"], cfg.fs_in, seed) * 0.4
        rng = np.random.default_rng(seed)
        taps = rng.normal(0.0, 1e-3, cfg.preemph_taps)
        taps[0] += 1.0
        st["w"] = (taps, np.array(f.a[: f.order]), np.array(f.g[: f.order]))
    elif kind == "fir":
        st["x"] = _music(c["ch"], c["frames"], c["fs_in"], seed)
        st["fir"] = FirChain(c["fs_in"], c["fs_out"], boxcar_taps=c["boxcar"],
                             soft_clip=c["clip"], num_channels=c["ch"])
    else:
        f = _filter(c["order_of"], c["rate"])
        # the modulator's input as the chain gives it: music at the DSD rate
        st["x"] = torch.stack([_slow_music(c["count"], c["rate"], seed, k)
                               for k in range(c["ch"])])
        st["sdm"] = TrellisSdm(f.order, f.a, f.g, c["depth"], c["cands"], c["lat"],
                               num_contexts=c["ch"])
    return st


def _slow_music(n, rate, seed, k):
    rng = np.random.Generator(np.random.PCG64([seed, 5, k]))
    t = torch.arange(n, dtype=torch.float64, device=DEV) / rate
    x = torch.zeros(n, dtype=torch.float64, device=DEV)
    for f0, ph in zip(np.geomspace(60.0, 18000.0, 9), rng.random(9)):
        x += 0.05 * torch.sin(2 * math.pi * (f0 * t + ph))
    return x


def run(st):
    c, kind = st["case"], st["kind"]
    if kind in ("encode", "precorr", "redsd"):
        enc = st["enc"]
        enc.flush()                      # each pass is a new track
        out = torch.empty(enc.out_capacity(c["frames"]) + 64, dtype=torch.uint8, device=DEV)
        _, nb = enc.process(st["x"], out, st["gain"], st["gain"])
        return out[:nb]
    if kind == "dsd2pcm":
        enc = st["enc"]
        enc.flush()
        out = torch.empty((c["ch"], 16 * c["frames"] * c["fs_out"] // c["fs_in"] + 16),
                          dtype=torch.float32, device=DEV)
        n, _ = enc.process(st["x"], out, st["gain"], st["gain"])
        return out[:, :n]
    if kind == "batch":
        st["plan"].load(st["xs"])
        st["plan"].run()
        return [st["plan"].out_view(i).clone() for i in range(c["streams"])]
    if kind == "train":
        eng = st["eng"]
        eng.set_input(st["x"])
        loss = eng.forward(*st["w"])
        gt, ga, gg = eng.backward()
        return {"loss": loss, "taps": gt, "a": ga, "g": gg, "decisions": eng.buffers()[1]}
    if kind == "fir":
        st["fir"].reset()
        return st["fir"].process(st["x"], PCM_FIR_GAIN, PCM_FIR_GAIN)
    return st["sdm"].process_block(st["x"])


def work(case):
    """Bytes in and out once; operations of the algorithm as the reference
    defines it (the modulator's K (5N + 6) per sample, the filters' taps)."""
    c, kind = case, case["kind"]
    if kind in ("encode", "precorr", "redsd"):
        n_in = c["frames"] * c["ch"]
        n = (16 * n_in if kind == "redsd" else n_in) * c["fs_out"] // c["fs_in"]
        if kind == "precorr":
            per = 7 * 5 + 6
        else:
            per = c["cands"] * (5 * _filter(c["ntf"], c["fs_out"]).order + 6)
        return {"bytes": 4 * n_in + 3 * n // 16, "flops": n * (per + 62)}
    if kind == "dsd2pcm":
        n_in = c["frames"] * c["ch"]
        n = 16 * n_in * c["fs_out"] // c["fs_in"]
        return {"bytes": 4 * n_in + 4 * n, "flops": 16 * n_in * 66}
    if kind == "batch":
        b = f = 0
        for e in signals.multistream_layout(c["streams"], scale=c["scale"]):
            n_in = e["frames"] * e["channels"]
            n = n_in * (e["fs_out"] // e["fs_in"])
            b += 4 * n_in + 3 * n // 16
            f += n * (c["cands"] * (5 * ntf.auto_select(e["fs_out"]).order + 6) + 62)
        return {"bytes": b, "flops": f}
    if kind == "train":
        n = c["clips"] * c["frames"] * 128
        return {"bytes": 4 * c["clips"] * c["frames"] + n, "flops": n * (c["cands"] * 41 + 200)}
    if kind == "fir":
        n = c["frames"] * c["ch"] * (c["fs_out"] // c["fs_in"])
        return {"bytes": 4 * c["frames"] * c["ch"] + 8 * n, "flops": 66 * n}
    n = c["count"] * c["ch"]
    order = _filter(c["order_of"], c["rate"]).order
    return {"bytes": 9 * n, "flops": n * c["cands"] * (5 * order + 6)}


# ---- the same in plain torch, 64 bits ----

def _i0(x):
    return torch.special.i0(torch.as_tensor(x, dtype=torch.float64))


def _taps(n, quarter=False):
    """Kaiser (beta 12) windowed half- or quarter-band lowpass, unit sum."""
    c = (n - 1) // 2
    k = torch.arange(n, dtype=torch.float64) - c
    w = _i0(12.0 * torch.sqrt(torch.clamp(1.0 - (k / c) ** 2, min=0.0))) / _i0(12.0)
    h = torch.sinc(k * (0.25 if quarter else 0.5)) * w
    return h / h.sum()


def _up(x, factor, h):
    """Zero-stuffed by `factor`, filtered from rest."""
    ch, n = x.shape
    out = torch.zeros((ch, n, factor), dtype=torch.float64, device=x.device)
    for k in range(len(h)):
        r, j = k % factor, k // factor
        if j < n:
            out[:, j:, r] += float(h[k]) * factor * x[:, : n - j]
    return out.reshape(ch, n * factor)


def _down(x, h):
    """Filtered from rest, every second output kept."""
    ch, n = x.shape
    m = n // 2
    xp = torch.cat([torch.zeros((ch, len(h) - 1), dtype=torch.float64, device=x.device), x], 1)
    out = torch.zeros((ch, m), dtype=torch.float64, device=x.device)
    for k in range(len(h)):
        at = len(h) - 1 - k
        out += float(h[k]) * xp[:, at:at + 2 * m:2][:, :m]
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "dsd2pcm":
        x = prepare(case, seed)["x"]
        word = torch.round(x.double() * 8388608.0).to(torch.int64) & 0xFFFF
        sh = torch.arange(15, -1, -1, device=x.device)
        y = []
        for c in range(x.shape[0]):
            v = (((word[c].unsqueeze(1) >> sh) & 1).to(torch.float64) * 2 - 1).reshape(1, -1)
            r = case["fs_in"] // case["fs_out"]
            while r > 1:
                v = _down(v, _taps(63))
                r //= 2
            y.append(v[0])
        return torch.stack(y)
    if kind == "fir":
        x = prepare(case, seed)["x"].double()
        if case["boxcar"]:
            b = case["boxcar"]
            s = torch.cumsum(torch.cat([torch.zeros((x.shape[0], b), dtype=x.dtype,
                                                    device=x.device), x], 1), 1)
            x = (s[:, b:] - s[:, :-b]) / b
        ratio = case["fs_out"] // case["fs_in"]
        stages = ratio.bit_length() - 1
        to512 = case["fs_out"] in (22579200, 24576000)
        if ratio == 8 and to512:
            plan = [(4, 127), (2, 63)]
        else:
            plan = [(2, 127 if to512 and i == 0 and stages > 1 else 63) for i in range(stages)]
        for factor, n in plan:
            x = _up(x, factor, _taps(n, factor == 4))
        x = x * PCM_FIR_GAIN
        if case["clip"]:
            over = x.abs() > 0.95
            knee = 0.95 + 0.05 * torch.tanh((x.abs() - 0.95) / 0.05)
            x = torch.where(over, torch.sign(x) * knee, x)
        return x
    return None
