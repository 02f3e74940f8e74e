"""DSD -> PCM decimation (the reference's FIR-only engine branch): the GPU
chain against the oracle's FP64 restatement of the half-band /2 stages with
IPP FIRMR semantics (streamed, odd block lengths), and the whole DoP -> PCM
pipeline's SINAD on a DSD128 tone, which the reference's README table puts
above 120 dB for DSD128 -> 44.1 kHz (README.md:589-600)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("fs_in,fs_out", [(2822400, 44100), (5644800, 176400), (11289600, 88200)])
def test_decim_matches_oracle(oracle, fs_in, fs_out):
    from foo_dsd_trellis_gb300 import _lib
    rng = np.random.default_rng(fs_in // fs_out)
    nch, n = 2, 300000
    bits = (rng.random((nch, n)) > 0.5).astype(np.uint8)
    L = _lib.load()
    h = C.c_void_p()
    assert L.dsdgpu_create(0, C.byref(h)) == 0
    _lib.check(h, L.dsdgpu_decim_setup(h, fs_in, fs_out, nch))
    refs = [oracle.Decimator(fs_in, fs_out) for _ in range(nch)]
    got = [[] for _ in range(nch)]
    want = [[] for _ in range(nch)]
    pos = 0
    for ln, g in ((12345, 0.8), (1, 0.8), (n - 12346, 0.8)):
        blk = torch.from_numpy(np.ascontiguousarray(bits[:, pos:pos + ln])).cuda()
        out = torch.empty((nch, max(ln, 1)), dtype=torch.float32, device="cuda")
        m = C.c_size_t()
        _lib.check(h, L.dsdgpu_decim_process(h, nch, C.c_void_p(blk.data_ptr()), blk.stride(0), ln,
                                             C.c_void_p(out.data_ptr()), out.stride(0), g, g,
                                             C.byref(m)))
        for c in range(nch):
            got[c].append(out[c, : m.value].cpu().numpy())
            y = refs[c].process(bits[c, pos:pos + ln].astype(np.float64) * 2 - 1)
            want[c].append((y * g).astype(np.float32))
        pos += ln
    for c in range(nch):
        a, b = np.concatenate(got[c]), np.concatenate(want[c])
        assert a.shape == b.shape
        np.testing.assert_allclose(a, b, rtol=0, atol=2e-7 * max(1e-30, np.abs(b).max()))
    L.dsdgpu_destroy(h)


def _sinad(y, fs, f0):
    n = len(y)
    lo, hi = n // 4, n - n // 20
    t = np.arange(lo, hi) / fs
    A = np.stack([np.sin(2 * np.pi * f0 * t), np.cos(2 * np.pi * f0 * t), np.ones_like(t)], 1)
    coef, *_ = np.linalg.lstsq(A, y[lo:hi].astype(np.float64), rcond=None)
    fit = A[:, :2] @ coef[:2]
    res = y[lo:hi] - A @ coef
    return 10 * np.log10(np.sum(fit * fit) / np.sum(res * res))


def test_dsd_to_pcm_pipeline_sinad(oracle):
    """PCM 997 Hz -> DSD128 (a plain sequential trellis encode on the GPU: the
    DAS seams would cap any SINAD near 56 dB) -> DoP -> the DSD -> PCM
    pipeline -> 44.1 kHz float: SINAD equal to the oracle chain's on the same
    DSD (within 0.01 dB) and above 115 dB."""
    from foo_dsd_trellis_gb300 import _lib, ntf, signals
    from foo_dsd_trellis_gb300.fir import FirChain
    from foo_dsd_trellis_gb300.pipeline import PCM_FIR_GAIN, Encoder
    from foo_dsd_trellis_gb300.sdm import TrellisSdm
    fs_pcm, fs_dsd, nch, K, depth, lat = 44100, 5644800, 2, 16, 32, 32
    f = ntf.get_filter("clans-7", fs_dsd)
    # no dither: the -110 dBFS TPDF of the small case would floor the SINAD
    pcm = signals.sine_tpdf(0.25, fs_pcm, nch, dither_db=-300.0, seed=9)
    g = float(PCM_FIR_GAIN)
    fir = FirChain(fs_pcm, fs_dsd, boxcar_taps=8, soft_clip=True, num_channels=nch).process(
        torch.from_numpy(pcm).cuda(), g, g)
    sdm = TrellisSdm(f.order, f.a, f.g, depth, K, lat, num_contexts=nch)
    body = sdm.process_block(fir)
    tail = sdm.drain(lat, nch=nch)
    dsd = np.stack([np.concatenate([body[c].cpu().numpy(), tail[c].cpu().numpy()]) for c in range(nch)])
    ns = dsd.shape[1] - dsd.shape[1] % 128
    dsd = dsd[:, :ns]
    dop = np.stack([oracle.dop_float_frames(dsd[c], 0) for c in range(nch)])
    dec = Encoder(fs_dsd, fs_pcm, nch, f, depth, K, lat, output_format=_lib.OUT_PCM)
    out = torch.empty((nch, ns // 128 + 16), dtype=torch.float32, device="cuda")
    n_out, nbytes = dec.process(torch.from_numpy(dop).cuda(), out, 1.0, 1.0)
    assert n_out == ns // 128 and nbytes == 4 * n_out * nch
    got = out[:, :n_out].cpu().numpy()
    for c in range(nch):
        ref = oracle.Decimator(fs_dsd, fs_pcm).process(dsd[c].astype(np.float64) * 2 - 1)
        ref = ref.astype(np.float32)          # the reference narrows to float too
        s_got, s_ref = _sinad(got[c], fs_pcm, 997.0), _sinad(ref, fs_pcm, 997.0)
        assert abs(s_got - s_ref) < 0.01, (s_got, s_ref)
        assert s_got > 115.0, s_got


@pytest.mark.parametrize("fs_in,fs_out", [(2822400, 1411200), (2822400, 705600), (2822400, 352800),
                                          (2822400, 176400), (5644800, 44100), (11289600, 44100),
                                          (22579200, 44100)])
def test_decim_blocks_of_every_kind(oracle, fs_in, fs_out):
    """Streams cut into calls that continue in each of the chain's forms: whole
    blocks (one matrix product over the history), ragged ends (the next call
    starts in the stages), calls of less than a block, calls around the 64 and
    128 blocks where the forms change, and a reset; three channels whose rows
    are wider than the call."""
    from foo_dsd_trellis_gb300 import _lib
    D = fs_in // fs_out
    B = max(D, 16)
    lens = [3 * B, 2 * B, 5, 200 * B + 7, 127 * B, 129 * B, 40 * B + 1, B - 1, 131 * B + B // 2,
            64 * B, 300 * B]
    if D == 512:
        lens = lens[:8]
    nch = 3
    rng = np.random.default_rng(D)
    L = _lib.load()
    h = C.c_void_p()
    assert L.dsdgpu_create(0, C.byref(h)) == 0
    _lib.check(h, L.dsdgpu_decim_setup(h, fs_in, fs_out, nch))
    for rep in range(2):
        refs = [oracle.Decimator(fs_in, fs_out) for _ in range(nch)]
        for k, ln in enumerate(lens if rep == 0 else lens[:1] + lens[5:7]):
            bits = (rng.random((nch, ln + 5)) > 0.4).astype(np.uint8)
            blk = torch.from_numpy(bits).cuda()
            out = torch.full((nch, ln // D + 3), 9.0, dtype=torch.float32, device="cuda")
            m = C.c_size_t()
            _lib.check(h, L.dsdgpu_decim_process(h, nch, C.c_void_p(blk.data_ptr()), blk.stride(0), ln,
                                                 C.c_void_p(out.data_ptr()), out.stride(0), 1.0, 1.0,
                                                 C.byref(m)))
            got = out.cpu().numpy()
            for c in range(nch):
                want = refs[c].process(bits[c, :ln].astype(np.float64) * 2 - 1).astype(np.float32)
                assert m.value == len(want), (k, ln)
                np.testing.assert_allclose(got[c, : len(want)], want, rtol=0, atol=2e-7,
                                           err_msg=f"call {k} of {ln}")
                assert (got[c, len(want):] == 9.0).all()
        _lib.check(h, L.dsdgpu_decim_reset(h))
    L.dsdgpu_destroy(h)


def test_decim_dop_equals_bits(oracle):
    """The pipeline's DoP frames (read by the decimation itself) give what the
    same decisions give as bytes: whole blocks, ragged ends and short calls."""
    from foo_dsd_trellis_gb300 import _lib, ntf
    from foo_dsd_trellis_gb300.pipeline import Encoder
    fs_in, fs_out, nch = 5644800, 44100, 2
    rng = np.random.default_rng(8)
    enc = Encoder(fs_in, fs_out, nch, ntf.get_filter("clans-7", fs_in), 64, 32, 128,
                  output_format=_lib.OUT_PCM)
    L = _lib.load()
    h = C.c_void_p()
    assert L.dsdgpu_create(0, C.byref(h)) == 0
    _lib.check(h, L.dsdgpu_decim_setup(h, fs_in, fs_out, nch))
    for frames in (8 * 40, 8 * 3, 3, 8 * 200 + 5, 8 * 500, 8 * 130, 1, 8 * 90):
        bits = (rng.random((nch, 16 * frames)) > 0.5).astype(np.uint8)
        dop = torch.from_numpy(np.stack([oracle.dop_float_frames(bits[c], 0) for c in range(nch)])).cuda()
        a = torch.zeros((nch, frames // 8 + 4), dtype=torch.float32, device="cuda")
        b = torch.zeros_like(a)
        n, _ = enc.process(dop, a, 0.7, 0.9)
        blk = torch.from_numpy(bits).cuda()
        m = C.c_size_t()
        _lib.check(h, L.dsdgpu_decim_process(h, nch, C.c_void_p(blk.data_ptr()), blk.stride(0),
                                             16 * frames, C.c_void_p(b.data_ptr()), b.stride(0), 0.7, 0.9,
                                             C.byref(m)))
        assert n == m.value
        assert torch.equal(a, b), frames
    L.dsdgpu_destroy(h)


def test_decim_contexts_of_different_ratios(oracle):
    """A context's setup leaves the contexts that were set up before it usable:
    ratios from 512 down to 2, then all run, the widest first."""
    from foo_dsd_trellis_gb300 import _lib
    L = _lib.load()
    rng = np.random.default_rng(12)
    ratios = (512, 128, 16, 2)
    hs = []
    for D in ratios:
        h = C.c_void_p()
        assert L.dsdgpu_create(0, C.byref(h)) == 0
        _lib.check(h, L.dsdgpu_decim_setup(h, 44100 * D, 44100, 1))
        hs.append(h)
    for D, h in zip(ratios, hs):
        n = 40 * max(D, 16)
        bits = (rng.random(n) > 0.4).astype(np.uint8)
        d = torch.from_numpy(bits).cuda()
        out = torch.zeros(n // D, dtype=torch.float32, device="cuda")
        m = C.c_size_t()
        _lib.check(h, L.dsdgpu_decim_process(h, 1, C.c_void_p(d.data_ptr()), n, n,
                                             C.c_void_p(out.data_ptr()), n // D, 1.0, 1.0, C.byref(m)))
        want = oracle.Decimator(44100 * D, 44100).process(bits.astype(np.float64) * 2 - 1)
        assert m.value == len(want)
        np.testing.assert_allclose(out.cpu().numpy(), want, rtol=0, atol=2e-7, err_msg=str(D))
    for h in hs:
        L.dsdgpu_destroy(h)


@pytest.mark.parametrize("fs_in,fs_out,nch", [(2822400, 176400, 2), (5644800, 44100, 3), (2822400, 1411200, 1)])
def test_decim_in_place(oracle, fs_in, fs_out, nch):
    """An output that lies in the input's memory (DoP frames replaced by their
    PCM, decision bytes by theirs) is the same as in memory of its own: from
    fresh state, after whole blocks and after a ragged end."""
    from foo_dsd_trellis_gb300 import _lib, ntf
    from foo_dsd_trellis_gb300.pipeline import Encoder
    D = fs_in // fs_out
    rng = np.random.default_rng(D + nch)
    f = ntf.get_filter("clans-7", 5644800)
    mk = lambda: Encoder(fs_in, fs_out, nch, f, 64, 32, 128, output_format=_lib.OUT_PCM)
    L = _lib.load()
    hs = [C.c_void_p(), C.c_void_p()]
    for h in hs:
        assert L.dsdgpu_create(0, C.byref(h)) == 0
        _lib.check(h, L.dsdgpu_decim_setup(h, fs_in, fs_out, nch))
    encs = [mk(), mk()] if D >= 16 else []
    for frames in (65536, 8 * 4000 + 3, 8 * 3000):
        n = 16 * frames // D
        bits = (rng.random((nch, 16 * frames)) > 0.4).astype(np.uint8)
        if encs:   # PCM no longer than its DoP frames
            dop = torch.from_numpy(np.stack([oracle.dop_float_frames(bits[c], 0) for c in range(nch)])).cuda()
            want = torch.zeros((nch, n), dtype=torch.float32, device="cuda")
            encs[0].process(dop, want, 0.7, 0.9)
            encs[1].process(dop, dop, 0.7, 0.9)
            assert torch.equal(dop[:, :n], want), frames
        raw = torch.zeros((nch, 64 * frames), dtype=torch.uint8, device="cuda")
        raw[:, : 16 * frames] = torch.from_numpy(bits).cuda()
        want = torch.zeros((nch, n), dtype=torch.float32, device="cuda")
        m = C.c_size_t()
        torch.cuda.synchronize()
        for h, out, ostride in ((hs[0], want, n), (hs[1], raw, 16 * frames)):
            _lib.check(h, L.dsdgpu_decim_process(h, nch, raw.data_ptr(), 64 * frames, 16 * frames,
                                                 out.data_ptr(), ostride, 1.0, 1.0, C.byref(m)))
            assert m.value == n
        assert torch.equal(raw.view(torch.float32)[:, :n], want), frames
    for h in hs:
        L.dsdgpu_destroy(h)


@pytest.mark.parametrize("before", ["fresh", "blocks", "ragged", "stages"])
@pytest.mark.parametrize("live_first", [False, True])
def test_decim_captured_calls(oracle, before, live_first):
    """A captured dsdgpu_decim_process_async continues the stream at every
    replay of its graph, whatever the stream was before the capture, mixed with
    plain calls after it, and from rest after a reset."""
    from foo_dsd_trellis_gb300 import _lib
    fs_in, fs_out, nch, D = 5644800, 176400, 2, 32
    rng = np.random.default_rng(len(before))
    L, rt = _lib.load(), C.CDLL("libcudart.so.13")
    h, st = C.c_void_p(), C.c_void_p()
    assert L.dsdgpu_create(0, C.byref(h)) == 0
    _lib.check(h, L.dsdgpu_decim_setup(h, fs_in, fs_out, nch))
    _lib.check(h, L.dsdgpu_get_stream(h, C.byref(st)))
    refs = [oracle.Decimator(fs_in, fs_out) for _ in range(nch)]
    cap = 300 * D

    def bits(n):
        b = (rng.random((nch, cap)) > 0.4).astype(np.uint8)
        return b, torch.from_numpy(b).cuda()

    def check(out, b, n):
        L.dsdgpu_synchronize(h)
        for c in range(nch):
            want = refs[c].process(b[c, :n].astype(np.float64) * 2 - 1).astype(np.float32)
            np.testing.assert_allclose(out.cpu().numpy()[c, : len(want)], want, rtol=0, atol=2e-7)

    def call(d_in, d_out, n):
        m = C.c_size_t()
        torch.cuda.synchronize()
        _lib.check(h, L.dsdgpu_decim_process_async(h, nch, d_in.data_ptr(), cap, n, d_out.data_ptr(),
                                                   cap // D, 1.0, 1.0, C.byref(m)))

    out = torch.zeros((nch, cap // D), dtype=torch.float32, device="cuda")
    for n in {"fresh": [], "blocks": [200 * D, 70 * D], "ragged": [200 * D + 5], "stages": [200 * D + 5, 7]}[before]:
        b, d = bits(n)
        call(d, out, n)
        check(out, b, n)
    n_cap = 150 * D + 9
    _, d_in = bits(n_cap)
    d_out = torch.zeros_like(out)
    graph, ex = C.c_void_p(), C.c_void_p()
    torch.cuda.synchronize()
    assert rt.cudaStreamBeginCapture(st, 1) == 0
    call_rc = L.dsdgpu_decim_process_async(h, nch, d_in.data_ptr(), cap, n_cap, d_out.data_ptr(), cap // D,
                                           1.0, 1.0, C.byref(C.c_size_t()))
    assert rt.cudaStreamEndCapture(st, C.byref(graph)) == 0 and call_rc == 0
    assert rt.cudaGraphInstantiate(C.byref(ex), graph, C.c_ulonglong(0)) == 0
    for what in (["live"] if live_first else []) + ["replay", "replay", "live", "replay", "reset", "replay", "live"]:
        if what == "reset":
            _lib.check(h, L.dsdgpu_decim_reset(h))
            refs = [oracle.Decimator(fs_in, fs_out) for _ in range(nch)]
            continue
        if what == "live":
            b, d = bits(0)
            call(d, out, 290 * D)
            check(out, b, 290 * D)
        else:
            b, d = bits(0)
            d_in.copy_(d)
            torch.cuda.synchronize()
            assert rt.cudaGraphLaunch(ex, st) == 0
            check(d_out, b, n_cap)
    rt.cudaGraphExecDestroy(ex)
    rt.cudaGraphDestroy(graph)
    L.dsdgpu_destroy(h)


@pytest.mark.parametrize("fs_in,fs_out,n", [(2822400, 1411200, 60001), (2822400, 176400, 2053),
                                            (5644800, 44100, 20001), (22579200, 44100, 65537),
                                            (5644800, 44100, 400000 + 5)])
def test_decim_ragged_calls_launch_no_more_than_the_stages(oracle, fs_in, fs_out, n):
    """A stream whose every call ends inside a block, in calls long enough for
    the matrix product (128 blocks and more): from the second on a call takes at
    most the stages' launches, and the outputs stay the oracle's."""
    from foo_dsd_trellis_gb300 import _lib
    nch, S = 2, (fs_in // fs_out).bit_length() - 1
    rng = np.random.default_rng(n)
    L = _lib.load()
    h = C.c_void_p()
    assert L.dsdgpu_create(0, C.byref(h)) == 0
    _lib.check(h, L.dsdgpu_decim_setup(h, fs_in, fs_out, nch))
    refs = [oracle.Decimator(fs_in, fs_out) for _ in range(nch)]
    out = torch.zeros((nch, n), dtype=torch.float32, device="cuda")
    count = []
    for k in range(5):
        bits = (rng.random((nch, n)) > 0.4).astype(np.uint8)
        d = torch.from_numpy(bits).cuda()
        m, v0, v1 = C.c_size_t(), C.c_uint64(), C.c_uint64()
        L.dsdgpu_launch_count(h, C.byref(v0))
        _lib.check(h, L.dsdgpu_decim_process(h, nch, d.data_ptr(), n, n, out.data_ptr(), n, 1.0, 1.0,
                                             C.byref(m)))
        L.dsdgpu_launch_count(h, C.byref(v1))
        count.append(v1.value - v0.value)
        for c in range(nch):
            want = refs[c].process(bits[c].astype(np.float64) * 2 - 1)
            assert m.value == len(want)
            np.testing.assert_allclose(out[c, : m.value].cpu().numpy(), want, rtol=0, atol=2e-7)
    assert max(count[2:]) <= 2 * S + 1, count
    L.dsdgpu_destroy(h)


def test_decim_one_stage_long_and_short_calls(oracle):
    """Ratio 2, where long calls take the stages and short ones the product:
    a stream of both."""
    from foo_dsd_trellis_gb300 import _lib
    nch = 1
    L = _lib.load()
    h = C.c_void_p()
    assert L.dsdgpu_create(0, C.byref(h)) == 0
    _lib.check(h, L.dsdgpu_decim_setup(h, 2822400, 1411200, nch))
    ref = oracle.Decimator(2822400, 1411200)
    rng = np.random.default_rng(3)
    for n in (600, 16 * 33000, 600, 16 * 33000 + 3, 5000, 499984, 500000):
        bits = (rng.random(n) > 0.4).astype(np.uint8)
        d, out, m = torch.from_numpy(bits).cuda(), torch.zeros(n, device="cuda"), C.c_size_t()
        _lib.check(h, L.dsdgpu_decim_process(h, nch, d.data_ptr(), n, n, out.data_ptr(), n, 1.0, 1.0,
                                             C.byref(m)))
        want = ref.process(bits.astype(np.float64) * 2 - 1)
        assert m.value == len(want)
        np.testing.assert_allclose(out[: m.value].cpu().numpy(), want, rtol=0, atol=2e-7, err_msg=str(n))
    L.dsdgpu_destroy(h)
