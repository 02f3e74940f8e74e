"""GPU trellis SDM vs the oracle (bit-exact): the CUDA path is called through
the C ABI (libdsdgpu.so via foo_dsd_trellis_gb300.sdm) and compared decision
by decision with the CPU restatement of src/trellis.c."""
import zlib

import numpy as np
import pytest

from signals import multitone, sdm_input

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _ntf(name, rate):
    from foo_dsd_trellis_gb300 import ntf
    return ntf.get_filter(name, rate)


def _gpu_sdm(f, depth, K, lat, lim=0.0, nctx=1):
    from foo_dsd_trellis_gb300.sdm import TrellisSdm
    return TrellisSdm(f.order, f.a, f.g, depth, K, lat, lim, num_contexts=nctx)


def _ora(oracle, f, depth, K, lat, lim=0.0):
    return oracle.sdm(f.order, np.array(f.a), np.array(f.g), depth, K, lat, lim)


CASES = [
    # (ntf name, rate, depth, K, lat, limit)
    ("clans-5", 2822400, 32, 16, 32, 0.0),     # the plain DSD64 configuration
    ("clans-7", 6144000, 64, 32, 128, 0.0),    # the DSD128 DAS configuration
    ("clans-6", 5644800, 32, 32, 128, 0.0),
    ("clans-8", 11289600, 48, 16, 32, 0.0),
    ("sdm-6", 22579200, 16, 2, 32, 10.0),
    ("clans-4", 2822400, 8, 32, 64, 4.0),
    ("sdm-8", 5644800, 4, 8, 16, 0.0),
    ("clans-6", 2822400, 1, 3, 7, 0.0),
    ("sdm-5", 11289600, 33, 31, 100, 2.0),
    ("clans-6", 2822400, 32, 1, 256, 0.0),
]


@pytest.mark.parametrize("case", CASES, ids=[f"{c[0]}-d{c[2]}-K{c[3]}-lat{c[4]}" for c in CASES])
def test_process_block_bit_exact(oracle, case):
    name, rate, depth, K, lat, lim = case
    f = _ntf(name, rate)
    n = 20000
    x = sdm_input(n, seed=zlib.crc32(repr(case).encode()) & 0xffff, amp=0.45)
    ref = _ora(oracle, f, depth, K, lat, lim)
    want = oracle.sdm_bits(ref, x)
    g = _gpu_sdm(f, depth, K, lat, lim)
    got = g.process_block(torch.from_numpy(x).cuda())[0].cpu().numpy()
    assert len(got) == len(want) == n - lat
    bad = np.nonzero(got != want)[0]
    assert bad.size == 0, f"first mismatch at {bad[:5]} of {len(want)}"
    q = g.query(0)
    info = ref.info()
    assert q["num_cands"] == info["num_cands"]
    assert q["total_children"] == info["total_children"]
    assert q["next_filter_drops"] == info["next_filter_drops"]
    assert q["conv_fail"] == info["conv_fail"]
    np.testing.assert_array_equal(q["best_state"], ref.best_state())


def test_streaming_blocks_and_drain(oracle):
    f = _ntf("clans-7", 6144000)
    x = multitone(30000, seed=5)
    ref = _ora(oracle, f, 64, 32, 128)
    g = _gpu_sdm(f, 64, 32, 128)
    rng = np.random.default_rng(3)
    pos = 0
    while pos < len(x):
        b = int(rng.integers(1, 5000))
        blk = x[pos:pos + b]
        pos += b
        want = oracle.sdm_bits(ref, blk)
        got = g.process_block(torch.from_numpy(blk).cuda())[0].cpu().numpy()
        np.testing.assert_array_equal(got, want)
    want = (ref.drain(500) > 0).astype(np.uint8)
    got = g.drain(500)[0].cpu().numpy()
    np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("K,depth,lat,lim", [(32, 64, 257, 0.0), (32, 32, 2048, 0.0),
                                             (16, 48, 1000, 2.0), (2, 4, 512, 0.0),
                                             (5, 16, 300, 0.0)])
def test_long_latency_streaming_and_drain(oracle, K, depth, lat, lim):
    """Latencies above 256 (up to the reference's 2048) take the wide-ring
    kernel: ragged streamed blocks over two channels, then drain."""
    f = _ntf("clans-7", 5644800)
    nch = 2
    xs = [sdm_input(lat + 9000, seed=lat + c, amp=0.5) for c in range(nch)]
    refs = [_ora(oracle, f, depth, K, lat, lim) for _ in range(nch)]
    g = _gpu_sdm(f, depth, K, lat, lim, nctx=nch)
    rng = np.random.default_rng(lat)
    pos = 0
    n = len(xs[0])
    while pos < n:
        b = min(int(rng.integers(1, 2 * lat)), n - pos)
        blk = np.stack([x[pos:pos + b] for x in xs])
        pos += b
        got = g.process_block(torch.from_numpy(blk).cuda())
        for c in range(nch):
            np.testing.assert_array_equal(got[c].cpu().numpy(), oracle.sdm_bits(refs[c], blk[c]))
    got = g.drain(lat + 10, 0, nch)
    for c in range(nch):
        want = (refs[c].drain(lat + 10) > 0).astype(np.uint8)
        assert len(want) == lat
        np.testing.assert_array_equal(got[c].cpu().numpy(), want)
    q = g.query(1)
    np.testing.assert_array_equal(q["best_state"], refs[1].best_state())


def test_short_block_then_drain(oracle):
    """Fewer samples than the latency, then drain (test/test_trellis.c:122-140)."""
    f = _ntf("clans-5", 2822400)
    ref = _ora(oracle, f, 8, 16, 64)
    g = _gpu_sdm(f, 8, 16, 64)
    x = np.zeros(40)
    assert len(oracle.sdm_bits(ref, x)) == 0
    assert g.process_block(torch.from_numpy(x).cuda())[0].numel() == 0
    want = (ref.drain(256) > 0).astype(np.uint8)
    got = g.drain(256)[0].cpu().numpy()
    assert len(want) == 40
    np.testing.assert_array_equal(got, want)


def test_multichannel_and_host_form(oracle):
    f = _ntf("clans-6", 5644800)
    xs = np.stack([sdm_input(8000, seed=s) for s in (1, 2, 3)])
    g = _gpu_sdm(f, 32, 32, 128, nctx=3)
    got = g.process_block_host(xs)
    for c in range(3):
        ref = _ora(oracle, f, 32, 32, 128)
        want = ref.process(xs[c])
        np.testing.assert_array_equal(got[c], want)


def test_segments_copy_seed_discard(oracle):
    """DAS-style segments: copy a warmed context, seed the candidates with a
    state, run with warm-up discard (src/engine.c:915-938)."""
    f = _ntf("clans-7", 6144000)
    K, depth, lat = 32, 64, 128
    x = multitone(60000, seed=11)
    base = _ora(oracle, f, depth, K, lat)
    oracle.sdm_bits(base, x[:5000])
    g = _gpu_sdm(f, depth, K, lat, nctx=5)
    g.process_block(torch.from_numpy(x[:5000]).cuda(), first=0)
    g.copy_state(4, 0)          # snapshot: segments must not read a context that runs
    seed = np.array(base.best_state())
    from foo_dsd_trellis_gb300.sdm import SegmentSpec
    specs, wants = [], []
    for i, (a, b, disc, sd) in enumerate([(5000, 20000, 0, False), (15000, 32000, 3000, True),
                                          (28000, 45000, 8192 - lat, True),
                                          (40000, 60000, 100000, False)]):
        ctxo = oracle.sdm(f.order, np.array(f.a), np.array(f.g), depth, K, lat)
        ctxo.copy_from(base)
        if sd:
            ctxo.seed(seed)
        wants.append(oracle.segment_bits(ctxo, x[a:b], disc))
        specs.append(SegmentSpec(torch.from_numpy(x[a:b].copy()).cuda(), channel=i,
                                 discard=disc, seed_from=4,
                                 seed_state=torch.from_numpy(seed).cuda() if sd else None))
    # channel 0 is also a target: copy_state of 4 onto 0 is the seeding source
    outs = g.segments(specs)
    for got, want in zip(outs, wants):
        np.testing.assert_array_equal(got.cpu().numpy(), want)


VERIFY_CASES = CASES + [
    ("clans-7", 6144000, 64, 32, 128, 0.0),
    ("clans-7", 6144000, 32, 32, 64, 0.0),
    ("clans-6", 5644800, 16, 32, 32, 0.0),
    ("sdm-7", 5644800, 8, 32, 128, 3.0),
]


@pytest.mark.parametrize("case", VERIFY_CASES,
                         ids=[f"v-{c[0]}-d{c[2]}-K{c[3]}-lat{c[4]}-{i}" for i, c in enumerate(VERIFY_CASES)])
def test_fast_selection_verified_against_serial(oracle, case):
    """Verify mode runs the serial (reference-order) selection every sample
    and checks the parallel one against it: any disagreement in survivors,
    order, costs, hashed set or stored chain links fails the call."""
    from foo_dsd_trellis_gb300 import _lib
    name, rate, depth, K, lat, lim = case
    f = _ntf(name, rate)
    x = multitone(40000, seed=zlib.crc32(repr(case).encode()) & 0xffff) * 1.5
    g = _gpu_sdm(f, depth, K, lat, lim, nctx=2)
    g.set_select(_lib.SELECT_VERIFY)
    got = g.process_block(torch.from_numpy(x).cuda())[0].cpu().numpy()
    want = oracle.sdm_bits(_ora(oracle, f, depth, K, lat, lim), x)
    assert np.array_equal(got, want)
    # seeded segments start with equal costs everywhere (ties)
    from foo_dsd_trellis_gb300.sdm import SegmentSpec
    seed = torch.from_numpy(np.array(g.query(0)["best_state"])).cuda()
    g.segments([SegmentSpec(torch.from_numpy(x[:20000].copy()).cuda(), channel=1, discard=300,
                            seed_from=0, seed_state=seed)])


def test_exact_and_fast_modes_agree(oracle):
    from foo_dsd_trellis_gb300 import _lib
    f = _ntf("clans-7", 6144000)
    x = multitone(30000, seed=77)
    outs = []
    for mode in (_lib.SELECT_FAST, _lib.SELECT_EXACT):
        g = _gpu_sdm(f, 64, 32, 128)
        g.set_select(mode)
        outs.append(g.process_block(torch.from_numpy(x).cuda())[0].cpu().numpy())
    assert np.array_equal(outs[0], outs[1])


@pytest.mark.parametrize("K,depth,lat,lim", [(2, 4, 128, 0.0), (1, 8, 32, 0.0), (2, 2, 200, 3.0),
                                             (4, 8, 32, 0.0), (3, 6, 64, 2.0), (4, 3, 100, 0.0)])
def test_small_k_streaming_channels_and_drain(oracle, K, depth, lat, lim):
    """Small trellises (K <= 4, including the reference's default K = 4,
    depth 8, lat 32) take the lane-split kernel: streamed blocks over several
    channels, short path masks (dedup on most samples), the limiter and the
    drain, against the oracle."""
    f = _ntf("clans-6", 5644800)
    nch = 5
    x = np.stack([multitone(12000, seed=40 + c) * (0.6 + 0.1 * c) for c in range(nch)])
    refs = [_ora(oracle, f, depth, K, lat, lim) for _ in range(nch)]
    g = _gpu_sdm(f, depth, K, lat, lim, nctx=nch)
    for lo, hi in ((0, 1), (1, 77), (77, 5000), (5000, 12000)):
        got = g.process_block(torch.from_numpy(np.ascontiguousarray(x[:, lo:hi])).cuda())
        for c in range(nch):
            np.testing.assert_array_equal(got[c].cpu().numpy(), oracle.sdm_bits(refs[c], x[c, lo:hi]))
    tail = g.drain(lat + 10, 0, nch)
    for c in range(nch):
        np.testing.assert_array_equal(tail[c].cpu().numpy(), (refs[c].drain(lat + 10) > 0).astype(np.uint8))
        q, info = g.query(c), refs[c].info()
        assert (q["num_cands"], q["total_children"], q["next_filter_drops"], q["conv_fail"]) == \
            (info["num_cands"], info["total_children"], info["next_filter_drops"], info["conv_fail"])
        np.testing.assert_array_equal(q["best_state"], refs[c].best_state())


@pytest.mark.parametrize("K,depth", [(2, 4), (4, 8), (1, 6)])
def test_kernels_share_the_context_format(oracle, K, depth):
    """One context carried through every SDM kernel in turn: the per-thread
    kernel (more jobs than the split kernel's cap), the lane-split kernel (few
    jobs), the warp kernel at 2 and 32 lanes (DSDGPU_OPT_SDM_LANES), then the
    split kernel again, each call continuing the previous one's state."""
    from foo_dsd_trellis_gb300 import _lib
    f = _ntf("clans-6", 5644800)
    many = 2600          # above the split kernel's 2 x 2 x 4 x 152 jobs (K <= 2)
    g = _gpu_sdm(f, depth, K, 32, 0.0, nctx=many)
    refs = [_ora(oracle, f, depth, K, 32) for _ in range(2)]
    x = np.stack([multitone(15000, seed=90 + c) * 0.7 for c in range(2)])
    pos = 0
    for stage, ln in (("all", 3000), ("split", 2500), ("lanes2", 3100), ("lanes32", 2900),
                      ("split", 3500)):
        blk = x[:, pos:pos + ln]
        pos += ln
        if stage == "all":
            if K > 2:
                continue
            xa = np.zeros((many, ln))
            xa[:2] = blk
            got = g.process_block(torch.from_numpy(xa).cuda())[:2]
        else:
            g.set_option(_lib.OPT_SDM_LANES, {"split": 0, "lanes2": 2, "lanes32": 32}[stage])
            got = g.process_block(torch.from_numpy(np.ascontiguousarray(blk)).cuda())
        for c in range(2):
            np.testing.assert_array_equal(got[c].cpu().numpy(), oracle.sdm_bits(refs[c], blk[c]),
                                          err_msg=stage)
    g.set_option(_lib.OPT_SDM_LANES, 0)
    got = g.drain(64, 0, 2)
    for c in range(2):
        np.testing.assert_array_equal(got[c].cpu().numpy(), (refs[c].drain(64) > 0).astype(np.uint8))


def test_small_k_many_jobs_take_the_per_thread_kernel(oracle):
    """More K <= 2 jobs than the lane-split kernel keeps resident (2,600
    channels of one launch) run one job per thread; every channel equals the
    oracle."""
    f = _ntf("clans-6", 5644800)
    nch, n = 2600, 300
    rng = np.random.default_rng(77)
    x = (rng.standard_normal((nch, n)) * 0.25).astype(np.float64)
    g = _gpu_sdm(f, 4, 2, 16, 0.0, nctx=nch)
    got = g.process_block(torch.from_numpy(x).cuda())
    for c in range(0, nch, 97):
        ref = _ora(oracle, f, 4, 2, 16)
        np.testing.assert_array_equal(got[c].cpu().numpy(), oracle.sdm_bits(ref, x[c]))


@pytest.mark.parametrize("order", [2, 3, 9, 10])
@pytest.mark.parametrize("K", [2, 8])
def test_orders_outside_the_table(oracle, order, K):
    """Orders 2, 3, 9 and 10 (accepted by the ABI, absent from the NTF table;
    a real NTF truncated or zero-padded), through the small-trellis and warp
    kernels."""
    src = _ntf("clans-4", 2822400) if order <= 4 else _ntf("clans-8", 11289600)
    a, g = np.zeros(order), np.zeros(order)
    m = min(order, src.order)
    a[:m], g[:m] = np.array(src.a[:m]), np.array(src.g[:m])

    class F:
        pass
    f = F()
    f.order, f.a, f.g = order, list(a), list(g)
    x = sdm_input(6000, seed=order * 10 + K, amp=0.3)
    ref = oracle.sdm(order, a, g, 16, K, 24, 0.0)
    want = oracle.sdm_bits(ref, x)
    gpu = _gpu_sdm(f, 16, K, 24)
    got = gpu.process_block(torch.from_numpy(x).cuda())[0].cpu().numpy()
    np.testing.assert_array_equal(got, want)


def test_estimate_state_batch(oracle):
    """dsdgpu_sdm_estimate_state (sdm_estimate_state_multibit, src/trellis.c:1125-1187)
    over many inputs in one launch equals the oracle (pinned to the reference's
    compiled estimator), for orders 2..10, 2/3/16/97/2000 levels (the quantiser
    index from reciprocal products, its table, and the exact divisions), the limiter and
    counts 0, 1 and 20,000."""
    import ctypes as C
    from foo_dsd_trellis_gb300 import _lib, ntf
    from signals import multitone
    L = _lib.load()
    h = C.c_void_p()
    assert L.dsdgpu_create(0, C.byref(h)) == 0
    rng = np.random.default_rng(11)
    names = ["clans-4", "clans-5", "clans-6", "clans-7", "clans-8", "sdm-5", "sdm-8"]
    for levels in (2, 3, 16, 97, 2000):
        for lim in (0.0, 1.5):
            for name in names:
                f = ntf.get_filter(name, 5644800)
                p = _lib.SdmParams()
                p.order = f.order
                for i in range(f.order):
                    p.a[i], p.g[i] = f.a[i], f.g[i]
                p.state_limit = lim
                counts = [0, 1, 20000, 777]
                xs = [multitone(max(n, 1), int(rng.integers(1000))) * 0.5 for n in counts]
                d_x = [torch.from_numpy(x).cuda() for x in xs]
                items = (_lib.EstimateItem * len(counts))()
                inits = []
                for j, n in enumerate(counts):
                    items[j].d_in = d_x[j].data_ptr()
                    items[j].count = n
                    init = rng.standard_normal(f.order) * 0.1
                    inits.append(init)
                    for k in range(f.order):
                        items[j].init_state[k] = init[k]
                _lib.check(h, L.dsdgpu_sdm_estimate_state(h, C.byref(p), levels, items, len(counts)))
                for j, n in enumerate(counts):
                    want = oracle.estimate_state(f.order, np.array(f.a), np.array(f.g), inits[j],
                                                 xs[j][:n], lim, levels)
                    got = np.array(items[j].out_state[: f.order])
                    assert np.array_equal(got, want), (name, levels, lim, n)
    p = _lib.SdmParams()
    p.order = 1
    assert L.dsdgpu_sdm_estimate_state(h, C.byref(p), 16, None, 0) == _lib.ERR_ARG
    p.order = 7
    assert L.dsdgpu_sdm_estimate_state(h, C.byref(p), 1, None, 0) == _lib.ERR_ARG
    L.dsdgpu_destroy(h)


def test_estimate_state_level_boundaries(oracle):
    """The estimator's quantiser at its level boundaries: from a zero state
    the first output is v = x + a0 * x, so first inputs placed on, and one or
    a few ulps and 1e-12 .. 1e-9 either side of, every boundary
    (v / a0 + 1) / step + 0.5 = k (and x = 0, where u = 7.5 exactly at 16
    levels) reach the samples the warp form hands to the reference's
    divisions; the next 40 inputs continue from the state they leave.  Equal
    to the oracle for 3, 16 and 32 levels, with and without the limiter."""
    import ctypes as C
    from foo_dsd_trellis_gb300 import _lib, ntf
    L = _lib.load()
    h = C.c_void_p()
    assert L.dsdgpu_create(0, C.byref(h)) == 0
    f = ntf.get_filter("clans-7", 5644800)
    a0 = float(f.a[0])
    rng = np.random.default_rng(5)
    for levels in (3, 16, 32):
        step = 2.0 / (levels - 1)
        firsts = [0.0]
        for k in range(levels + 1):
            yi = (k - 0.5) * step - 1.0
            x0 = yi * a0 / (1.0 + a0)
            firsts.append(x0)
            for d in (1, 2, 4):
                firsts.append(float(np.nextafter(x0, np.inf) if d == 1 else x0 + d * np.spacing(x0)))
                firsts.append(float(np.nextafter(x0, -np.inf) if d == 1 else x0 - d * np.spacing(x0)))
            for rel in (1e-12, 3e-10, 1e-9, 2e-9):
                firsts.extend([x0 * (1 + rel) + rel, x0 * (1 - rel) - rel])
        for lim in (0.0, 1.5):
            p = _lib.SdmParams()
            p.order = f.order
            for i in range(f.order):
                p.a[i], p.g[i] = f.a[i], f.g[i]
            p.state_limit = lim
            xs = [np.concatenate([[x0], 0.3 * rng.standard_normal(40)]) for x0 in firsts
                  for _ in range(2)]
            d_x = [torch.from_numpy(x).cuda() for x in xs]
            items = (_lib.EstimateItem * len(xs))()
            for j, x in enumerate(xs):
                items[j].d_in = d_x[j].data_ptr()
                items[j].count = len(x) if j % 2 else 1
            _lib.check(h, L.dsdgpu_sdm_estimate_state(h, C.byref(p), levels, items, len(xs)))
            for j, x in enumerate(xs):
                n = items[j].count
                want = oracle.estimate_state(f.order, np.array(f.a), np.array(f.g),
                                             np.zeros(f.order), x[:n], lim, levels)
                got = np.array(items[j].out_state[: f.order])
                assert np.array_equal(got, want), (levels, lim, j, x[0])
    L.dsdgpu_destroy(h)


def test_state_distance(oracle):
    """dsdgpu_sdm_state_distance (src/trellis.c:1094-1109) of two contexts run on
    different inputs equals the sum of squared differences of the oracle's best
    states, added in order."""
    from foo_dsd_trellis_gb300 import ntf
    from foo_dsd_trellis_gb300.sdm import TrellisSdm
    from foo_dsd_trellis_gb300 import _lib
    import ctypes as C
    from signals import multitone
    f = ntf.get_filter("clans-7", 5644800)
    sdm = TrellisSdm(f.order, f.a, f.g, 16, 8, 32, 0.0, num_contexts=2)
    xs = [multitone(5000, 3 + c) * 0.6 for c in range(2)]
    refs = [oracle.sdm(f.order, np.array(f.a), np.array(f.g), 16, 8, 32) for _ in range(2)]
    sdm.process_block(torch.from_numpy(np.stack(xs)).cuda())
    for c in range(2):
        oracle.sdm_bits(refs[c], xs[c])
    d = C.c_double()
    _lib.check(sdm.h, sdm.L.dsdgpu_sdm_state_distance(sdm.h, 0, 1, C.byref(d)))
    sa, sb = refs[0].best_state(), refs[1].best_state()
    want = 0.0
    for i in range(f.order):
        t = sa[i] - sb[i]
        want += t * t
    assert d.value == want
    _lib.check(sdm.h, sdm.L.dsdgpu_sdm_state_distance(sdm.h, 1, 1, C.byref(d)))
    assert d.value == 0.0
    assert sdm.L.dsdgpu_sdm_state_distance(sdm.h, 0, 2, C.byref(d)) == _lib.ERR_ARG
    sdm.close()


@pytest.mark.parametrize("K,depth,lat", [(32, 64, 128), (32, 6, 33), (17, 3, 64), (16, 48, 31),
                                         (9, 32, 300), (8, 4, 256), (5, 3, 32), (4, 2, 65),
                                         (2, 1, 1)])
def test_costs_the_sort_words_do_not_tell(oracle, K, depth, lat):
    """Costs that the selection's 32-bit words leave undecided take its whole
    comparison: silence (equal costs from the first sample), a level far below
    and far above the words' range, and equal paths on most samples (short path
    masks), in blocks that end inside and at the ring's words."""
    f = _ntf("clans-7" if K > 8 else "clans-6", 5644800)
    x = np.concatenate([np.zeros(400), 1e-9 * multitone(300, seed=K), 0.5 * multitone(700, seed=K + 1),
                        np.array([1e4, -1e60, 1e120]), 0.3 * multitone(600, seed=K + 2)])
    ref = _ora(oracle, f, depth, K, lat)
    g = _gpu_sdm(f, depth, K, lat)
    for lo, hi in ((0, 1), (1, 33), (33, 640), (640, len(x))):
        got = g.process_block(torch.from_numpy(x[lo:hi].copy()).cuda())[0].cpu().numpy()
        np.testing.assert_array_equal(got, oracle.sdm_bits(ref, x[lo:hi]))
    info, q = ref.info(), g.query(0)
    assert (q["num_cands"], q["total_children"], q["next_filter_drops"], q["conv_fail"]) == \
        (info["num_cands"], info["total_children"], info["next_filter_drops"], info["conv_fail"])
    np.testing.assert_array_equal(q["best_state"], ref.best_state())


@pytest.mark.parametrize("K,depth,lat,njobs,order", [
    (2, 4, 40, 5, 6), (2, 4, 64, 900, 6), (2, 40, 9, 1900, 7), (1, 8, 33, 4000, 8),
    (4, 8, 32, 7, 6), (3, 6, 31, 700, 5), (4, 50, 65, 1400, 8), (8, 4, 256, 3, 6),
    (6, 16, 20, 700, 7), (7, 5, 32, 1300, 8), (16, 48, 32, 6, 8), (12, 5, 300, 9, 7)])
def test_uneven_segments_share_warps(oracle, K, depth, lat, njobs, order):
    """Small trellises put up to eight jobs on a warp, chosen by their number:
    segments of uneven lengths around the 32-sample blocks (none, one and
    many), with discards and seeds, each from a copied context, and the
    contexts that they leave."""
    from foo_dsd_trellis_gb300.sdm import SegmentSpec
    f = _ntf({5: "sdm-5", 6: "clans-6", 7: "clans-7", 8: "clans-8"}[order], 5644800)
    lens = [0, 1, 31, 32, 33, 63, 64, 65, 97, 400]
    x = multitone(1200, seed=K + njobs) * 0.8
    g = _gpu_sdm(f, depth, K, lat, nctx=njobs + 1)
    base = _ora(oracle, f, depth, K, lat)
    oracle.sdm_bits(base, x[:333])
    g.process_block(torch.from_numpy(x[:333].copy()).cuda(), first=njobs)
    seed = base.best_state() * 0.5
    xs, sd = torch.from_numpy(x).cuda(), torch.from_numpy(seed).cuda()
    specs = []
    for i in range(njobs):
        n, lo = lens[(i * 7 + i // 10) % len(lens)], 333 + i % 300
        specs.append(SegmentSpec(xs[lo:lo + n], channel=i, discard=[0, 5, 40][i % 3], seed_from=njobs,
                                 seed_state=sd if i % 2 and n else None))   # empty: a plain copy
    outs = g.segments(specs)
    for i in list(range(min(njobs, 24))) + list(range(24, njobs, 53)):
        ctx = _ora(oracle, f, depth, K, lat)
        ctx.copy_from(base)
        n, lo = lens[(i * 7 + i // 10) % len(lens)], 333 + i % 300
        if i % 2 and n:
            ctx.seed(seed)
        np.testing.assert_array_equal(outs[i].cpu().numpy(),
                                      oracle.segment_bits(ctx, x[lo:lo + n], [0, 5, 40][i % 3]),
                                      err_msg=str(i))
        q, info = g.query(i), ctx.info()
        assert (q["num_cands"], q["total_children"], q["next_filter_drops"], q["conv_fail"]) == \
            (info["num_cands"], info["total_children"], info["next_filter_drops"], info["conv_fail"]), i
        np.testing.assert_array_equal(q["best_state"], ctx.best_state())


@pytest.mark.parametrize("K,order,njobs", [(2, 6, 3000), (1, 5, 5000), (4, 5, 2000), (8, 7, 1300),
                                           (16, 8, 3), (9, 4, 700), (16, 6, 1300)])
def test_products_in_and_out_of_range(oracle, K, order, njobs):
    """At these numbers of jobs one lane has a child's whole state and forms its
    products on the integer pipe, except while a state of the warp is not in
    their range: fresh contexts (zero states) between running ones, silence,
    levels of 1e-290 and 1e120, and all back in range."""
    f = _ntf({4: "clans-4", 5: "sdm-5", 6: "clans-6", 7: "clans-7", 8: "clans-8"}[order],
             2822400 if order == 4 else 5644800)
    g = _gpu_sdm(f, 4, K, 40, nctx=njobs)
    tail = 0.4 * multitone(150, seed=K)
    rows = np.stack([np.concatenate([r, tail]) for r in (
        np.zeros(100), np.full(100, 1e-290), 0.6 * multitone(100, seed=K), np.full(100, 1e120))])
    refs = [_ora(oracle, f, 4, K, 40) for _ in range(8)]
    for k, n in enumerate((50, 250)):   # first: every second group of four
        lo = 0 if k else njobs // 2 // 4 * 4
        idx = np.arange(lo, njobs)
        xs = rows[idx % 4, :n]
        got = g.process_block(torch.from_numpy(xs).cuda(), first=lo)
        half = njobs // 2 // 4 * 4
        for c in range(8):
            fresh, row = c < 4, c % 4
            if fresh and k == 0:
                continue
            want = oracle.sdm_bits(refs[c], rows[row, :n])
            for i in np.flatnonzero(((idx < half) == fresh) & (idx % 4 == row))[::29]:
                np.testing.assert_array_equal(got[i].cpu().numpy(), want, err_msg=f"{c} {n} {i}")


def _filter(kind, order):
    """A filter of the table; "odd": the table's odd orders above DSD512, whose
    odd g are zero; "g0": every resonator at 0; "trained": every g nonzero;
    "cut": a table filter truncated or zero-padded to `order`."""
    if kind == "odd":
        return _ntf({5: "sdm-5", 7: "sdm-7"}[order], 45158400)
    src = (_ntf("clans-4", 2822400) if order <= 4 else _ntf("clans-8", 11289600)) if kind == "cut" else \
        _ntf({5: "clans-5", 6: "clans-6", 7: "clans-7", 8: "clans-8"}[order], 5644800)

    class F:
        pass
    f = F()
    f.order, f.a, f.g = order, [0.0] * order, [0.0] * order
    m = min(order, src.order)
    f.a[:m], f.g[:m] = list(src.a[:m]), list(src.g[:m])
    if kind == "g0":
        f.g = [0.0] * order
    if kind == "trained":
        f.g = [v + 1e-5 * (i + 1) for i, v in enumerate(f.g)]
    return f


@pytest.mark.parametrize("kind,order", [("odd", 7), ("odd", 5), ("g0", 6), ("g0", 7), ("trained", 7),
                                        ("trained", 8), ("cut", 2), ("cut", 3), ("cut", 9), ("cut", 10)])
@pytest.mark.parametrize("K,lanes", [(32, 0), (19, 0), (16, 16), (7, 8)])
def test_warp_kernel_filters(oracle, kind, order, K, lanes):
    """The warp kernels with filters whose coefficients the integer products do
    not take (a zero a, a zero g where the table has none), with the other
    pattern of zero g and with none: streamed, equal to the oracle."""
    from foo_dsd_trellis_gb300 import _lib
    f = _filter(kind, order)
    depth, lat = 40, 48
    n = 2600
    x = 0.5 * multitone(n, seed=order + K)
    x[700:900] = 0.0
    ref = _ora(oracle, f, depth, K, lat)
    g = _gpu_sdm(f, depth, K, lat)
    if lanes:
        g.set_option(_lib.OPT_SDM_LANES, lanes)
    for lo, hi in ((0, 31), (31, 1500), (1500, n)):
        got = g.process_block(torch.from_numpy(x[lo:hi].copy()).cuda())[0].cpu().numpy()
        np.testing.assert_array_equal(got, oracle.sdm_bits(ref, x[lo:hi]))
    assert g.last_sdm_kernel() == f"sdm_jobs_kernel<{order},{lanes or 32}>"
    info, q = ref.info(), g.query(0)
    assert (q["num_cands"], q["total_children"], q["next_filter_drops"], q["conv_fail"]) == \
        (info["num_cands"], info["total_children"], info["next_filter_drops"], info["conv_fail"])
    np.testing.assert_array_equal(q["best_state"], ref.best_state())


@pytest.mark.parametrize("kind,order", [("table", 7), ("odd", 7), ("g0", 6)])
def test_parts_kernel_filters(kind, order):
    """The balanced launch (jobs in queued parts) equals one job a warp for the
    same filters."""
    from foo_dsd_trellis_gb300 import _lib
    from foo_dsd_trellis_gb300.das import DasChannels
    f = _filter(kind, order)
    pipes = 4 * torch.cuda.get_device_properties(0).multi_processor_count
    S = (pipes + pipes // 20) // 2 + 1            # segments per channel, 2 channels
    x = np.stack([multitone(S * 9000, 30 + c) * 0.5 for c in range(2)])
    fir = torch.from_numpy(np.ascontiguousarray(x)).cuda()
    outs = []
    for balance in (1, 0):
        d = DasChannels(f.order, f.a, f.g, 16, 32, 32, num_channels=2)
        _lib.check(d.h, d.L.dsdgpu_set_option(d.h, _lib.OPT_SDM_BALANCE, balance))
        outs.append(d.process_chunk(fir, nsegs=S, seed_mode=0)[0])
        assert d.last_sdm_kernel().startswith("sdm_parts_kernel" if balance else "sdm_jobs_kernel")
        d.close()
    assert torch.equal(outs[0], outs[1])


@pytest.mark.parametrize("K,depth,lanes", [(32, 64, 0), (32, 6, 0), (18, 48, 0), (16, 8, 16), (8, 8, 8), (4, 8, 4),
                                           (2, 4, 2)])
@pytest.mark.parametrize("name,rate,amp,odd", [("clans-7", 5644800, 4.0, 0.0), ("sdm-8", 45158400, 0.4, 0.0),
                                               ("clans-6", 5644800, 0.5, 1e300)])
def test_runaway_modulator_warp_kernel(oracle, K, depth, lanes, name, rate, amp, odd):
    """A modulator that has run away (no limiter): its costs leave the range of
    the sort's words and agree to many places, or are not finite after an input
    of 1e300; the order then comes from the keys' distances or from the whole
    keys."""
    from foo_dsd_trellis_gb300 import _lib
    f = _ntf(name, rate)
    x = amp * multitone(2500, seed=K)
    x[1700] += odd
    ref = _ora(oracle, f, depth, K, 40)
    g = _gpu_sdm(f, depth, K, 40)
    if lanes:
        g.set_option(_lib.OPT_SDM_LANES, lanes)
    for lo, hi in ((0, 1000), (1000, 2500)):
        got = g.process_block(torch.from_numpy(x[lo:hi].copy()).cuda())[0].cpu().numpy()
        np.testing.assert_array_equal(got, oracle.sdm_bits(ref, x[lo:hi]))
    assert g.last_sdm_kernel().startswith("sdm_jobs_kernel")
    info, q = ref.info(), g.query(0)
    assert (q["num_cands"], q["total_children"], q["next_filter_drops"], q["conv_fail"]) == \
        (info["num_cands"], info["total_children"], info["next_filter_drops"], info["conv_fail"])
    np.testing.assert_array_equal(q["best_state"], ref.best_state())


@pytest.mark.parametrize("K,depth,order", [(2, 4, 6), (1, 6, 4), (2, 6, 8)])
def test_per_thread_kernel_shares_the_context_format(oracle, K, depth, order):
    """Contexts carried through the per-thread kernel (more jobs than five warps
    of eight a scheduler), the child kernel (few of them), the warp kernel at 2
    and 32 lanes, and the first two again; each call continues from the last."""
    from foo_dsd_trellis_gb300 import _lib
    f = _ntf({4: "clans-4", 6: "clans-6", 8: "clans-8"}[order], 5644800)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    many = 5 * 8 * 4 * sms + 33
    g = _gpu_sdm(f, depth, K, 32, nctx=many)
    refs = [_ora(oracle, f, depth, K, 32) for _ in range(2)]
    x = np.stack([multitone(2200, seed=90 + c) * 0.7 for c in range(2)])
    at = [0, many - 1]
    pos = 0
    for stage, ln in (("all", 333), ("few", 300), ("lanes2", 310), ("lanes32", 290), ("all", 400), ("few", 350)):
        blk = x[:, pos:pos + ln]
        pos += ln
        g.set_option(_lib.OPT_SDM_LANES, {"lanes2": 2, "lanes32": 32}.get(stage, 0))
        if stage == "all":
            xa = torch.zeros((many, ln), dtype=torch.float64, device="cuda")
            for c in range(2):
                xa[at[c]] = torch.from_numpy(blk[c].copy()).cuda()
            out = g.process_block(xa)
            got = [out[i] for i in at]
        else:
            got = [g.process_block(torch.from_numpy(blk[c].copy()).cuda(), first=at[c])[0] for c in range(2)]
        want = {"all": "sdm_scalar_kernel", "few": "sdm_child_kernel"}.get(stage, "sdm_jobs_kernel")
        assert g.last_sdm_kernel().startswith(want), stage
        for c in range(2):
            np.testing.assert_array_equal(got[c].cpu().numpy(), oracle.sdm_bits(refs[c], blk[c]), err_msg=stage)
    g.set_option(_lib.OPT_SDM_LANES, 0)
    for c in range(2):
        q, info = g.query(at[c]), refs[c].info()
        assert (q["num_cands"], q["total_children"], q["next_filter_drops"], q["conv_fail"]) == \
            (info["num_cands"], info["total_children"], info["next_filter_drops"], info["conv_fail"])
        np.testing.assert_array_equal(q["best_state"], refs[c].best_state())
        got = g.drain(64, at[c], 1)[0].cpu().numpy()
        np.testing.assert_array_equal(got, (refs[c].drain(64) > 0).astype(np.uint8))


@pytest.mark.parametrize("K,depth,lat,njobs,order", [(2, 4, 70, 900, 6), (2, 6, 9, 2500, 7), (4, 8, 33, 1400, 5),
                                                     (8, 16, 100, 1300, 8), (16, 32, 65, 6, 6), (16, 9, 300, 40, 7)])
def test_contexts_of_uneven_jobs_continue(oracle, K, depth, lat, njobs, order):
    """Jobs of uneven lengths beside one another in a warp: the context that each
    leaves (its ring and place in it among the rest) goes on as the oracle's."""
    from foo_dsd_trellis_gb300.sdm import SegmentSpec
    f = _ntf({5: "clans-5", 6: "clans-6", 7: "clans-7", 8: "clans-8"}[order], 5644800)
    lens = [1, 31, 32, 33, 64, 97, 130, 400]
    x = multitone(1500, seed=K + njobs) * 0.8
    g = _gpu_sdm(f, depth, K, lat, nctx=njobs + 1)
    base = _ora(oracle, f, depth, K, lat)
    oracle.sdm_bits(base, x[:333])
    g.process_block(torch.from_numpy(x[:333].copy()).cuda(), first=njobs)
    xs = torch.from_numpy(x).cuda()
    at = lambda i: (lens[(i * 5 + i // 8) % len(lens)], 333 + i % 200)
    g.segments([SegmentSpec(xs[at(i)[1]:at(i)[1] + at(i)[0]], channel=i, seed_from=njobs) for i in range(njobs)])
    assert g.last_sdm_kernel().startswith("sdm_child_kernel")
    more = x[1000:1300]
    outs = g.process_block(torch.from_numpy(np.repeat(more[None], njobs, 0)).cuda())
    for i in list(range(min(njobs, 20))) + list(range(20, njobs, 97)):
        n, lo = at(i)
        ctx = _ora(oracle, f, depth, K, lat)
        ctx.copy_from(base)
        oracle.segment_bits(ctx, x[lo:lo + n], 0)
        np.testing.assert_array_equal(outs[i].cpu().numpy(), oracle.sdm_bits(ctx, more), err_msg=str(i))
        q, info = g.query(i), ctx.info()
        assert (q["num_cands"], q["total_children"], q["next_filter_drops"], q["conv_fail"]) == \
            (info["num_cands"], info["total_children"], info["next_filter_drops"], info["conv_fail"]), i
        np.testing.assert_array_equal(g.drain(lat + 5, i, 1)[0].cpu().numpy(),
                                      (ctx.drain(lat + 5) > 0).astype(np.uint8))


@pytest.mark.parametrize("levels", [3, 16, 32, 97])
@pytest.mark.parametrize("a0", [-0.9, 1e-120, -1e-120, 3e110])
def test_estimate_state_unusual_a0(oracle, levels, a0):
    """The estimator's thresholds with a negative a_0 (the order of the levels
    turned round), and a_0 too small or large for thresholds, where every block
    takes the reference's divisions: equal to the oracle with and without the
    limiter, over counts around the blocks of 32."""
    import ctypes as C
    from foo_dsd_trellis_gb300 import _lib
    L = _lib.load()
    h = C.c_void_p()
    assert L.dsdgpu_create(0, C.byref(h)) == 0
    f = _ntf("clans-6", 5644800)
    a = [a0] + list(f.a[1:])
    rng = np.random.default_rng(levels)
    for lim in (0.0, 1.5):
        p = _lib.SdmParams()
        p.order = f.order
        for i in range(f.order):
            p.a[i], p.g[i] = a[i], f.g[i]
        p.state_limit = lim
        counts = [1, 31, 32, 33, 500]
        xs = [0.3 * rng.standard_normal(n) for n in counts]
        d_x = [torch.from_numpy(x).cuda() for x in xs]
        items = (_lib.EstimateItem * len(counts))()
        inits = [rng.standard_normal(f.order) * 0.1 for _ in counts]
        for j, n in enumerate(counts):
            items[j].d_in, items[j].count = d_x[j].data_ptr(), n
            for k in range(f.order):
                items[j].init_state[k] = inits[j][k]
        _lib.check(h, L.dsdgpu_sdm_estimate_state(h, C.byref(p), levels, items, len(counts)))
        for j, n in enumerate(counts):
            want = oracle.estimate_state(f.order, np.array(a), np.array(f.g), inits[j], xs[j], lim, levels)
            np.testing.assert_array_equal(np.array(items[j].out_state[: f.order]), want, err_msg=f"{lim} {n}")
    L.dsdgpu_destroy(h)
