"""Each CUDA stage against the reference's intermediate arrays (through include/optflow_cuda_testing.h).

The expected values come from the committed golden vectors (written by the reference itself) and from the
CPU oracle, which tests/test_oracle.py pins to the reference.
"""
import numpy as np
import pytest
from conftest import golden

from optflow_b200.config import Config

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def T():
    from optflow_b200 import testing
    return testing


# direct plans (radices up to 31; 320 ... 2112 on plans fixed at compile time), then lengths with a larger prime factor
# (Bluestein: 37, 41 * 4, 2 * 53, 151 * 4 = the padded height of a 960 x 540 frame (inner length 1216, on a fixed
# plan), the primes 191 and 1021, and 1999 = the largest inner length here, 4096)
BLUESTEIN = [37, 164, 106, 604, 191, 1021, 1999]


@pytest.mark.parametrize("L", [2, 3, 4, 5, 7, 8, 11, 13, 17, 19, 23, 29, 31])
def test_fft_lines_one_stage(T, L):
    """Lines of one radix, a transform whose first stage is its last: within the bound of test_fft_lines_runtime_plans."""
    rng = np.random.default_rng(L)
    a = (rng.standard_normal((5, L)) + 1j * rng.standard_normal((5, L))).astype(np.complex64)
    for inv in (False, True):
        got = T.fft_lines(a, inverse=inv)
        ref = np.fft.ifft(a.astype(np.complex128), axis=1) * L if inv else np.fft.fft(a.astype(np.complex128), axis=1)
        assert np.abs(got - ref).max() < 2e-6 * np.abs(ref).max(), inv


@pytest.mark.parametrize("L,bound", [(144, 2e-6), (441, 2e-6), (650, 2e-6), (975, 2e-6), (1539, 2e-6), (2023, 2e-6),
                                      (2048, 2e-6), (253, 2e-6), (841, 2e-6), (899, 2e-6), (1564, 2e-6), (1922, 2e-6), (397, 1e-5), (433, 1e-5), (917, 1e-5), (1109, 1e-5),
                                      (1431, 1e-5), (1822, 1e-5)])
def test_fft_lines_runtime_plans(T, L, bound):
    """Runtime plans by their stages' kinds: even radices first (padded stores), odd radices only, a radix above 19 (direct
    DFT), Bluestein inner lengths of 2 and 3 stages of the large radices and of 4 stages; the bounds of
    test_fft_lines_match_numpy."""
    rng = np.random.default_rng(L)
    a = (rng.standard_normal((3, L)) + 1j * rng.standard_normal((3, L))).astype(np.complex64)
    for inv in (False, True):
        got = T.fft_lines(a, inverse=inv)
        ref = np.fft.ifft(a.astype(np.complex128), axis=1) * L if inv else np.fft.fft(a.astype(np.complex128), axis=1)
        assert np.abs(got - ref).max() < bound * np.abs(ref).max(), (L, inv)


@pytest.mark.parametrize("variant", [0, 3])
@pytest.mark.parametrize("L", [674, 705, 787, 811, 929, 958, 1099, 1214, 1241, 1328, 1437, 1606, 1637, 1791, 1821, 2047])
def test_fft_lines_compiled_inner_lengths(T, L, variant):
    """One length of each Bluestein inner length with stages of its own (1352 ... 4096), in the default factor order and
    reversed (which those stages do not serve); the Bluestein bound of test_fft_lines_match_numpy."""
    from optflow_b200 import Engine, _abi
    lib = _abi.load()

    def order(v):
        n, var = np.array([L], np.int32), np.array([v], np.int32)
        lib.ofc_fft_set_plans(n.ctypes.data_as(_abi.c_i32_p), var.ctypes.data_as(_abi.c_i32_p), 1)

    rng = np.random.default_rng(L)
    a = (rng.standard_normal((3, L)) + 1j * rng.standard_normal((3, L))).astype(np.complex64)
    fwd = np.fft.fft(a.astype(np.complex128), axis=1)
    inv = np.fft.ifft(a.astype(np.complex128), axis=1) * L
    order(variant)
    try:
        eng = Engine(0)  # a fresh engine builds its plan from the table
        for inverse, ref in ((False, fwd), (True, inv)):
            assert np.abs(T.fft_lines(a, inverse=inverse, engine=eng) - ref).max() < 1e-5 * np.abs(ref).max(), inverse
    finally:
        order(0)


@pytest.mark.parametrize("shape", [(133, 911), (40, 1367), (1367, 75), (185, 333), (40, 5936), (777, 68), (40, 777), (1977, 70)])
def test_passes_runtime_plans(T, oracle, shape):
    """The row and column passes on runtime plans (direct, Bluestein, odd pitches; 6000 padded columns, where the
    reference pack's rows have one scratch buffer): test_responses and test_reference_phase_fixed_length at these sizes."""
    test_responses_fixed_length(T, oracle, shape)
    test_reference_phase_fixed_length(T, shape)


@pytest.mark.parametrize("L", [64, 128, 160, 192, 224, 320, 576, 832, 1024, 1088, 1152, 1600, 2112, 2*3*5*7*11, 3*17*19,
                               23*29, 31*8]
                         + BLUESTEIN)
def test_fft_lines_match_numpy(T, L):
    """Line transforms against numpy in float64: 2e-6 of the largest output for the direct plans, 1e-5 for
    Bluestein's (a float32 chirp, two transforms of the inner length and a product between them)."""
    rng = np.random.default_rng(L)
    a = (rng.standard_normal((5, L)) + 1j * rng.standard_normal((5, L))).astype(np.complex64)
    for inv in (False, True):
        got = T.fft_lines(a, inverse=inv)
        ref = np.fft.ifft(a.astype(np.complex128), axis=1) * L if inv else np.fft.fft(a.astype(np.complex128), axis=1)
        err = np.abs(got - ref).max() / np.abs(ref).max()
        assert err < (1e-5 if L in BLUESTEIN else 2e-6), (L, inv, err)


def test_reference_phase(T):
    """parity_gabor.rs:40-70: per filter, response error < 1e-4 of its largest |r|; phase gradient error
    < 1e-3 rad/px on the pixels whose amplitude exceeds 5 % of the filter's largest."""
    g = golden("gabor")
    ref = T.reference_phase(g["img"])
    for k, (r, gx, gy, amp) in enumerate(ref):
        want = g["r_re"][k] + 1j * g["r_im"][k]
        max_amp = np.abs(want).max()
        assert np.abs(r - want).max() / max_amp < 1e-4
        strong = g["amp"][k] > 0.05 * max_amp
        assert strong.sum() > strong.size / 20
        assert np.abs(gx - g["gx"][k])[strong].max() < 1e-3
        assert np.abs(gy - g["gy"][k])[strong].max() < 1e-3
        assert np.abs(amp - g["amp"][k])[strong].max() < 1e-4 * max_amp
    # near the zeros of a response the gradient Im(conj r rx) / |r|^2 amplifies the float32 transforms' absolute
    # error e max|r| (e ~ 1e-6; the reference's Rust port has the same float32 transforms) by max|r|^2 / amp^2:
    # scaled by (amp / max)^2 the error stays below e times (the filter's frequency + 1) < 1e-5
    for k, (r, gx, gy, amp) in enumerate(ref):
        max_amp = np.abs(g["r_re"][k] + 1j * g["r_im"][k]).max()
        weak = g["amp"][k] > 1e-4 * max_amp
        err = np.maximum(np.abs(gx - g["gx"][k]), np.abs(gy - g["gy"][k]))
        assert (err * (g["amp"][k] / max_amp) ** 2)[weak].max() < 1e-5


def _gabor_bank_np(shape, cfg):
    """phaseflow.gabor_bank (python/optflow_ref/phaseflow.py:73-89), restated in numpy for the check."""
    h, w = shape
    fy = (np.fft.fftfreq(h) * 2 * np.pi)[:, None]
    fx = (np.fft.fftfreq(w) * 2 * np.pi)[None, :]
    s_hp = cfg.dc_cut * cfg.lam * max(cfg.scales) / (2 * np.pi)
    hp = 1.0 - np.exp(-(fx ** 2 + fy ** 2) * s_hp ** 2 / 2)
    bank = []
    for sc in cfg.scales:
        w0 = 2 * np.pi / (cfg.lam * sc)
        s = cfg.bandwidth * w0
        for k in range(cfg.n_orient):
            th = np.pi * k / cfg.n_orient
            bank.append(hp * np.exp(-((fx - w0 * np.cos(th)) ** 2 + (fy - w0 * np.sin(th)) ** 2) / (2 * s * s)))
    return bank


@pytest.mark.parametrize("shape", [(96, 128), (160, 224)])
def test_responses(T, oracle, shape):
    rng = np.random.default_rng(1)
    img = rng.random(shape).astype(np.float32)
    cfg = Config()
    got = T.responses(img, cfg)
    pad = np.pad(img.astype(np.float64), 32, mode="reflect")
    F2 = np.fft.fft2(pad)
    for k, G in enumerate(_gabor_bank_np(pad.shape, cfg)):
        r = np.fft.ifft2(F2 * G)
        want = oracle.bspline_coeffs(r.real) + 1j * oracle.bspline_coeffs(r.imag)
        err = np.abs(got[k] - want).max() / np.abs(want).max()
        assert err < 1e-4, (k, err)


@pytest.mark.parametrize("shape", [(2048, 2048), (2048, 136), (136, 2048)])
def test_responses_fixed_length(T, oracle, shape):
    """Padded length 2112 (2048-pixel sides, the benchmark's size) runs the transforms' compile-time plan and the
    staged column-pair / persistent row kernels; the mixed shapes pair it with a runtime plan on the other axis."""
    rng = np.random.default_rng(7)
    img = rng.random(shape).astype(np.float32)
    cfg = Config()
    got = T.responses(img, cfg)
    pad = np.pad(img.astype(np.float64), 32, mode="reflect")
    F2 = np.fft.fft2(pad)
    bank = _gabor_bank_np(pad.shape, cfg)
    for k in (0, 5, 11):
        r = np.fft.ifft2(F2 * bank[k])
        want = oracle.bspline_coeffs(r.real) + 1j * oracle.bspline_coeffs(r.imag)
        err = np.abs(got[k] - want).max() / np.abs(want).max()
        assert err < 1e-4, (shape, k, err)


@pytest.mark.parametrize("shape", [(2048, 2048), (136, 2048)])
def test_reference_phase_fixed_length(T, shape):
    """reference_phase (phaseflow.py:92-112) at padded length 2112 against a float64 numpy restatement: the
    response within 1e-4 of its largest |r|, the phase gradient within 1e-3 rad/px where the amplitude exceeds 5 %
    of the largest (the tolerances of parity_gabor.rs:40-70)."""
    rng = np.random.default_rng(8)
    img = rng.random(shape).astype(np.float32)
    cfg = Config()
    got = T.reference_phase(img, cfg)
    h, w = shape
    pad = np.pad(img.astype(np.float64), 32, mode="reflect")
    F2 = np.fft.fft2(pad)
    fy = (np.fft.fftfreq(pad.shape[0]) * 2 * np.pi)[:, None]
    fx = (np.fft.fftfreq(pad.shape[1]) * 2 * np.pi)[None, :]
    bank = _gabor_bank_np(pad.shape, cfg)
    crop = (slice(32, 32 + h), slice(32, 32 + w))
    for k in (0, 7):
        Z = F2 * bank[k]
        r = np.fft.ifft2(Z)[crop]
        rx = np.fft.ifft2(Z * 1j * fx)[crop]
        ry = np.fft.ifft2(Z * 1j * fy)[crop]
        a2 = np.abs(r) ** 2 + 1e-12
        gx, gy = (np.conj(r) * rx).imag / a2, (np.conj(r) * ry).imag / a2
        g_r, g_gx, g_gy, g_amp = got[k]
        max_amp = np.abs(r).max()
        assert np.abs(g_r - r).max() / max_amp < 1e-4
        strong = np.sqrt(a2) > 0.05 * max_amp
        assert strong.sum() > strong.size / 20
        assert np.abs(g_gx - gx)[strong].max() < 1e-3
        assert np.abs(g_gy - gy)[strong].max() < 1e-3
        assert np.abs(g_amp - np.sqrt(a2))[strong].max() < 1e-4 * max_amp


@pytest.mark.parametrize("order", [1, 2])
def test_local_solve(T, oracle, order):
    rng = np.random.default_rng(order)
    h, w = 70, 90
    gx, gy = rng.normal(size=(2, 12, h, w))
    wk = rng.uniform(0.1, 1.0, size=(12, h, w))
    c = rng.normal(size=(12, h, w)) + 20.0  # large right-hand sides, as with |u| ~ 25 px
    sums = [(wk * gx * gx).sum(0), (wk * gx * gy).sum(0), (wk * gy * gy).sum(0), (wk * gx * c).sum(0),
            (wk * gy * c).sum(0), (wk * c * c).sum(0), wk.sum(0)]
    sums[0][10:14, 10:14] = 0.0  # degenerate: no energy
    sums[1][10:14, 10:14] = 0.0
    sums[2][10:14, 10:14] = 0.0
    ux, uy = rng.normal(size=(2, h, w))
    got = T.local_solve(sums, ux, uy, Config(shape_order=order))
    want = oracle.local_solve(sums, ux, uy, 4.0, order)
    for a, b in zip(got, want):
        np.testing.assert_allclose(a, b, rtol=1e-7, atol=1e-9)


@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("h,w", [(3, 5), (31, 32), (33, 96), (47, 97), (48, 159), (49, 161), (97, 193)])
def test_local_solve_tile_edges(T, oracle, order, h, w):
    """The window moments and the solve at the edges of their tiles: 32 columns x 48 (order 2: 32) rows in y, 160 (96)
    pixels in x, images smaller than the window; the tolerance of test_local_solve."""
    rng = np.random.default_rng(100 * h + w + order)
    gx, gy = rng.normal(size=(2, 12, h, w))
    wk = rng.uniform(0.1, 1.0, size=(12, h, w))
    c = rng.normal(size=(12, h, w)) + 20.0
    sums = [(wk * gx * gx).sum(0), (wk * gx * gy).sum(0), (wk * gy * gy).sum(0), (wk * gx * c).sum(0),
            (wk * gy * c).sum(0), (wk * c * c).sum(0), wk.sum(0)]
    ux, uy = rng.normal(size=(2, h, w))
    got = T.local_solve(sums, ux, uy, Config(shape_order=order))
    want = oracle.local_solve(sums, ux, uy, 4.0, order)
    for a, b in zip(got, want):
        np.testing.assert_allclose(a, b, rtol=1e-7, atol=1e-9)


def test_median(T):
    rng = np.random.default_rng(5)
    for n in (1, 2, 3, 10, 1001, 4096, 100000):
        v = rng.exponential(size=n) * 1e3
        assert T.median(v) == np.median(v)
    v = np.repeat(rng.random(50), 7)
    assert T.median(v) == np.median(v)
    assert T.median(np.array([3.0, 1.0, 2.0, 2.0])) == 2.0
    # both signs; values clustered in one binade (a large bucket after two digits)
    for v in (rng.standard_normal(100001), 1.0 + rng.random(200000) * 1e-6):
        assert T.median(v) == np.median(v)
    # ties: a bucket within the candidate list, and beyond it (the remaining digits then take full passes), with
    # odd and even counts and the lower middle element inside or below the tied value
    for n_tie, n in ((30000, 100000), (150000, 200001), (150000, 200000), (60000, 120000)):
        v = rng.exponential(size=n)
        v[:n_tie] = np.median(v)
        rng.shuffle(v)
        assert T.median(v) == np.median(v), (n_tie, n)
    v = np.concatenate([np.zeros(60000), rng.random(60000)])
    assert T.median(v) == np.median(v)


@pytest.mark.parametrize("n", [1, 2, 1023, 1024, 1025, 8191, 8192, 16384, 16385, 148 * 8192 + 3, 3_000_000])
def test_median_blocks_and_special_values(T, n):
    """The cooperative median at the edges of its blocks (8192 energies a block up to one block per SM, then more per
    thread) against np.median exactly: spread values, one value throughout, infinities, subnormals, a NaN."""
    rng = np.random.default_rng(n)
    for v in (rng.exponential(size=n), np.full(n, 0.25), rng.standard_normal(n) * 10.0 ** rng.integers(-300, 300, n),
              rng.integers(0, 3, n).astype(np.float64), rng.random(n) * 1e-310):
        assert T.median(v) == np.median(v)
    v = rng.exponential(size=n)
    v[: n // 3] = np.inf
    assert T.median(v) == np.median(v)
    v[n // 2] = np.nan
    assert np.isnan(T.median(v))


@pytest.mark.parametrize("n", [1, 2, 33, 4096, 65537, 98304, 98305, 303104, 606209, 1300001])
def test_median_reset_rounds(T, n):
    """Medians and resets in sequence on the alternating halves of one state, exactly: no pixel below the threshold (the
    median needed or not), some far below it, energies over 80 decades, a NaN, ties, one value for half of them, one far
    outlier on either side. Sizes around the cluster's limit, its registers and the launches' full grid, odd and even."""
    rng = np.random.default_rng(n)
    base = rng.exponential(size=n) + 0.1
    few = base.copy()
    few[rng.random(n) < 0.1] *= 1e-12
    few[: n // 50] = 0.0
    wide = base * 10.0 ** rng.uniform(-40, 40, n)
    nan = few.copy()
    nan[n // 2] = np.nan
    ties = rng.integers(0, 3, n) * 1.0
    half = np.where(rng.random(n) < 0.55, 0.0, base)
    out1, out2 = base.copy(), base.copy()
    out1[n // 3], out2[n // 3] = 1e-300, 1e300
    rounds = [(base, 0), (few, 0), (few[::-1], 1), (base, 1), (wide, 0), (wide, 1), (nan, 0), (base, 0), (ties, 0), (half, 1),
              (out1, 0), (out2, 1), (np.full(n, 0.25), 1), (few, 0)]
    e = np.stack([v for v, _ in rounds])
    u = rng.normal(size=(2, n))
    med, planes = T.median_reset(e, [f for _, f in rounds], u)
    for k, (v, force) in enumerate(rounds):
        skip = not np.isnan(v).any() and v.min() > 1e-9 * v.max() + 1e-30
        want = np.median(v)
        if force or not skip:
            np.testing.assert_equal(med[k], want, err_msg=str(k))
        hit = np.zeros(n, bool) if skip else ~(v > 1e-9 * want + 1e-30)
        np.testing.assert_array_equal(planes[k, :2], np.where(hit, u, 0.0), err_msg=str(k))
        np.testing.assert_array_equal(planes[k, 2], np.where(hit, np.pi, 0.0), err_msg=str(k))
        np.testing.assert_array_equal(planes[k, 3:], np.broadcast_to(np.where(hit, 0.0, np.nan), (4, n)), err_msg=str(k))


def test_large_components(T, oracle):
    rng = np.random.default_rng(9)
    for p in (0.3, 0.5, 0.6):
        b = rng.random((123, 157)) < p
        for area in (5, 50, 327.68):
            np.testing.assert_array_equal(T.large_components(b, area), oracle.large_components(b, area))


@pytest.mark.parametrize("w2,h2,shift", [(260, 300, (0, 0)), (260, 300, (-7, 5)), (258, 301, (0, 0)),
                                         (64, 40, (3, -2)), (2048, 2048, (0, 0))])
def test_warp_tma_matches_gather(T, oracle, w2, h2, shift):
    """The TMA-staged warp (each 32 x 16 output tile's source box staged in shared memory) against the gather kernel
    bit for bit, and both against the oracle's B-spline sampler (interp.py:52-69): smooth fields up to 15 px, a band
    whose taps span more rows than the 64 x 40 box, positions beyond the plane (clamped, mirrored taps) and NaN
    positions. A plane whose row pitch is not a multiple of 16 bytes (258 floats) takes the gather kernel in both
    modes."""
    rng = np.random.default_rng(w2 + h2)
    c2 = rng.normal(size=(h2, w2)).astype(np.float32)
    h, w = h2 - 10, w2 + 6
    yy, xx = np.mgrid[0:h, 0:w].astype(np.float64)
    sx = 15 * np.sin(xx / 37.0) * np.cos(yy / 53.0) + rng.normal(size=(h, w)) * 0.3
    sy = 9 * np.cos(xx / 29.0 + yy / 61.0)
    sy[h // 3:h // 3 + 5] += 60
    sx[5, 7] = np.nan
    sy[20, 30] = np.nan
    g, t0 = T.warp(c2, sx, sy, shift, mode=0)
    m, t1 = T.warp(c2, sx, sy, shift, mode=1)
    assert t0 == 0 and t1 == 0
    np.testing.assert_array_equal(m.view(np.uint32), g.view(np.uint32))
    X, Y = xx + shift[0] + sx, yy + shift[1] + sy
    ok = np.isfinite(X) & np.isfinite(Y)
    assert np.isnan(g[~ok]).all() and np.isfinite(g[ok]).all()
    ref = oracle.sample(c2.astype(np.float64), np.where(ok, X, 0), np.where(ok, Y, 0))
    np.testing.assert_allclose(g[ok], ref[ok], rtol=0, atol=1e-6)


@pytest.mark.parametrize("shape,amp", [((96, 128), 2.0), ((200, 264), 12.0), ((1024, 1024), 5.0)])
def test_accumulate_tma_matches_gather(T, shape, amp):
    """The TMA-staged accumulate (each filter pair's response box and reference-pack tile staged in shared memory)
    against the gather kernel, bit for bit, on refine's first inner iteration: a smooth start field, a sharp band whose
    blocks' taps span more than the 48 x 16-node box, a jump at the left border that moves taps outside the padded
    plane (mirrored indices)."""
    from scipy.ndimage import gaussian_filter
    rng = np.random.default_rng(shape[0])
    h, w = shape
    a = gaussian_filter(rng.random((h, w)), 1.5)
    b = np.roll(a, (1, 2), axis=(0, 1)) + 0.01 * rng.random((h, w))
    yy, xx = np.mgrid[0:h, 0:w].astype(np.float64)
    ux = amp * np.sin(xx / 41.0) * np.cos(yy / 37.0)
    uy = amp * np.cos(xx / 29.0 + yy / 53.0)
    uy[h // 2:h // 2 + 3] += 40.0
    ux[:, :3] -= 80.0
    from optflow_b200.api import default_engine
    from optflow_b200.measure import Profile
    s0, t0 = T.accumulate(a, b, ux, uy, mode=0)
    prof = Profile(default_engine())
    prof.start()
    s1, t1 = T.accumulate(a, b, ux, uy, mode=1)
    assert "k_accumulate_tma" in prof.read()
    assert t0 == 0 and t1 == 0
    assert np.isfinite(s1).all()
    np.testing.assert_array_equal(s1, s0)


@pytest.mark.parametrize("shape,n_orient,scales", [((64, 65), 1, (1.0,)), ((67, 131), 3, (0.6,)), ((130, 97), 5, (0.6,)),
                                                   ((70, 64), 4, (0.6, 1.0, 1.6))])
def test_accumulate_ring_and_edges(T, shape, n_orient, scales):
    """The gather accumulate (the reference pack in a ring of two filter pairs, packed sampling, border positions out of
    line) against the TMA-staged kernel's unpacked arithmetic bit for bit: one filter, odd filter counts (the last pair
    half empty), sizes off the 32 x 4 block, positions beyond the padded plane on every side."""
    rng = np.random.default_rng(shape[1])
    h, w = shape
    a, b = rng.random((h, w)), rng.random((h, w))
    yy, xx = np.mgrid[0:h, 0:w].astype(np.float64)
    ux, uy = 3 * np.sin(xx / 17.0), 2 * np.cos(yy / 23.0)
    ux[:, :4] -= 70.0
    ux[:, -4:] += 70.0
    uy[:5] -= 70.0
    uy[-5:] += 70.0
    cfg = Config(n_orient=n_orient, scales=scales)
    s0, _ = T.accumulate(a, b, ux, uy, mode=0, cfg=cfg)
    s1, t1 = T.accumulate(a, b, ux, uy, mode=1, cfg=cfg)
    assert t1 == 0 and np.isfinite(s1).all()
    np.testing.assert_array_equal(s0, s1)


def test_accumulate_ring_cases_are_two_kernels(T):
    """The two modes that test_accumulate_ring_and_edges compares are two kernels where there are two filters or more; one
    filter has the gather kernel alone (its second slot of the ring is never filled), which test_accumulate_one_filter
    checks."""
    from optflow_b200.api import default_engine
    from optflow_b200.measure import Profile
    rng = np.random.default_rng(3)
    for shape, n_orient, scales, staged in (((64, 65), 1, (1.0,), False), ((67, 131), 3, (0.6,), True),
                                            ((130, 97), 5, (0.6,), True), ((70, 64), 4, (0.6, 1.0, 1.6), True)):
        a, b = rng.random(shape), rng.random(shape)
        u = np.zeros(shape)
        prof = Profile(default_engine())
        prof.start()
        T.accumulate(a, b, u, u, mode=1, cfg=Config(n_orient=n_orient, scales=scales))
        assert ("k_accumulate_tma" in prof.read()) == staged, shape


@pytest.mark.parametrize("shape", [(64, 65), (67, 131)])
def test_accumulate_one_filter(T, oracle, shape):
    """The accumulate of a single filter (the second slot of its ring is never filled, the packed arithmetic's second half
    works on whatever is there) against the oracle's float64 sums, positions beyond the padded plane included. Tolerance,
    from the stages' (test_responses, test_reference_phase): responses within 1e-4 of their largest |r|, the phase gradient
    within 1e-3 rad/px, where |r1| and |r2| exceed 5 % of it. So the weight |r1| |r2| within e_w = 2 * 1e-4 / 0.05 relative,
    the phase difference within the same of 1 rad, c within e_c = e_w + 1e-3 (|u| + |v|), and the sums by the product rule.
    Pixels whose phase difference may wrap (within 0.1 of pi) are left out."""
    rng = np.random.default_rng(shape[1])
    h, w = shape
    from scipy.ndimage import gaussian_filter
    a = gaussian_filter(rng.random((h, w)), 1.0).astype(np.float32)
    b = np.roll(a, (1, 2), axis=(0, 1))
    yy, xx = np.mgrid[0:h, 0:w].astype(np.float64)
    ux, uy = 2 + np.sin(xx / 17.0), 1 + 0.5 * np.cos(yy / 23.0)
    ux[:, :3] -= 70.0
    uy[-3:] += 70.0
    cfg = Config(n_orient=1, scales=(1.0,))
    got, _ = T.accumulate(a, b, ux, uy, mode=0, cfg=cfg)
    want = oracle.first_sums(a, b, ux, uy, cfg)
    r, gx, gy, _ = oracle.reference_phase(a, cfg)[0]
    wk = want[6]
    r1 = np.abs(r)
    r2 = wk / r1
    c = np.where(np.abs(gx) > np.abs(gy), want[3] / (wk * gx), want[4] / (wk * gy))
    ok = (r1 > 0.05 * r1.max()) & (r2 > 0.05 * r1.max()) & (np.abs(c - gx * ux - gy * uy) < np.pi - 0.1)
    assert ok.mean() > 0.5
    ew, eg = 2 * 1e-4 / 0.05, 1e-3
    ec = ew + eg * (np.abs(ux) + np.abs(uy))
    ax, ay, ac = np.abs(gx), np.abs(gy), np.abs(c)

    def bound(p, ep, q, eq):  # of wk p q
        return wk * ((1 + ew) * (p + ep) * (q + eq) - p * q)

    bounds = [bound(ax, eg, ax, eg), bound(ax, eg, ay, eg), bound(ay, eg, ay, eg), bound(ax, eg, ac, ec),
              bound(ay, eg, ac, ec), bound(ac, ec, ac, ec), wk * ew]
    for i in range(7):
        assert np.isfinite(got[i]).all()
        assert (np.abs(got[i] - want[i]) <= bounds[i])[ok].all(), i


@pytest.mark.parametrize("amp", [1e-30, 1e-24, 1e-18, 1e12, 1e18, 1e20, 1e22])
def test_accumulate_extreme_amplitudes(T, amp):
    """The accumulate's packed phase differences at response magnitudes beyond its fast quotient's range (products of two
    responses below 1e-30 and above 1e30, infinite and NaN ones) against the TMA-staged kernel's unpacked arithmetic: bit
    for bit but for the rounding of a quotient, at most one unit of the last place of a float32 angle (2.4e-7 of pi) in the
    sums that hold it. Finite, infinite and NaN sums in the same places."""
    rng = np.random.default_rng(11)
    h, w = 67, 70
    a, b = rng.random((h, w)), rng.random((h, w))
    ux, uy = rng.normal(size=(2, h, w))
    cfg = Config(n_orient=4, scales=(0.6,))
    s0, _ = T.accumulate(a * amp, b * amp, ux, uy, mode=0, cfg=cfg)
    s1, t1 = T.accumulate(a * amp, b * amp, ux, uy, mode=1, cfg=cfg)
    assert t1 == 0
    for i in (0, 1, 2, 6):  # no phase difference in these
        np.testing.assert_array_equal(s0[i], s1[i])
    for i in (3, 4, 5):
        np.testing.assert_array_equal(np.isnan(s0[i]), np.isnan(s1[i]))
        np.testing.assert_array_equal(np.isinf(s0[i]), np.isinf(s1[i]))
        ok = np.isfinite(s1[i])
        if ok.any():
            np.testing.assert_allclose(s0[i][ok], s1[i][ok], rtol=1e-6, atol=1e-6 * np.abs(s1[i][ok]).max())


def test_atan2_phase_exact_quotients(T):
    """Magnitudes outside the fast quotient's range take the rounded quotient: arguments whose quotient is a power of two
    give one angle, whatever their common factor (2^-120 to 2^-101 and 2^101 to 2^126, subnormal ones among them)."""
    rng = np.random.default_rng(12)
    m = rng.uniform(1, 2, 4000).astype(np.float32)
    for lo, hi in ((-120, -101), (-140, -127), (101, 126)):
        s = np.ldexp(m, rng.integers(lo, hi, m.size)).astype(np.float32)
        for k in (0, 1, 3):
            y, x = s, np.ldexp(s, -k).astype(np.float32)
            same = np.ldexp(x.astype(np.float64), k) == y  # no bits lost to a subnormal
            got = T.atan2(y[same], x[same])[0]
            assert same.sum() > 100 and np.unique(got).size == 1, (lo, k)


def test_atan2_phase(T):
    """The accumulate's float32 atan2 (common.cuh, a polynomial fit of atan on [0, 1]) within 5e-7 rad of the exact
    angle of its float32 arguments over 20 decades of magnitude and every direction, like CUDA's atan2f there; signed
    zeros and axes as atan2 gives them; NaN propagated."""
    rng = np.random.default_rng(17)
    n = 1 << 20
    mag = 10.0 ** rng.uniform(-20, 20, n)
    ang = rng.uniform(-np.pi, np.pi, n)
    x = (mag * np.cos(ang)).astype(np.float32)
    y = (mag * np.sin(ang)).astype(np.float32)
    special = np.array([(0.0, 0.0), (-0.0, 0.0), (0.0, -0.0), (-0.0, -0.0), (1, 0), (-1, 0), (0, 1), (0, -1), (1, 1),
                        (-1, 1), (1, -1), (-1, -1), (3, -0.0), (-3, -0.0), (1e-38, 1e-38), (1e-44, 2e-44),
                        (2e30, -1e30), (-5e-32, 7e-32)], np.float32)
    y = np.concatenate([y, special[:, 0]])
    x = np.concatenate([x, special[:, 1]])
    mine, cuda = T.atan2(y, x)
    exact = np.arctan2(y.astype(np.float64), x.astype(np.float64))
    assert np.abs(mine - exact).max() <= 5e-7
    assert np.abs(cuda - exact).max() <= 1e-6
    k = len(special)
    np.testing.assert_array_equal(np.signbit(mine[-k:]), np.signbit(exact[-k:]))
    m2, _ = T.atan2(np.array([np.nan, 1, np.nan], np.float32), np.array([1, np.nan, np.nan], np.float32))
    assert np.isnan(m2).all()


def test_prewarp_fill(T, oracle):
    """phaseflow.prewarp's fill (phaseflow.py:344-354) with scipy's nearest-source tie rule."""
    rng = np.random.default_rng(3)
    h, w = 90, 120
    low = np.zeros((h, w), bool)
    low[30:60, 40:80] = True
    low |= rng.random((h, w)) < 0.01
    ux, uy = rng.normal(size=(2, h, w))
    slope = rng.normal(size=(h, w, 4)) * 0.01
    R = Config().auto_edge_guard_px()
    gx, gy = T.prewarp_fill(low, ux, uy, slope, R)
    ok = oracle.edt(~low) > R
    _, (iy, ix) = oracle.edt(~ok, return_indices=True)
    yy, xx = np.mgrid[0:h, 0:w].astype(np.float64)
    dx, dy = xx - ix, yy - iy
    g = slope[iy, ix]
    ex = np.where(ok, ux, ux[iy, ix] + g[..., 0] * dx + g[..., 2] * dy)
    ey = np.where(ok, uy, uy[iy, ix] + g[..., 1] * dx + g[..., 3] * dy)
    np.testing.assert_allclose(gx, ex, rtol=0, atol=1e-12)
    np.testing.assert_allclose(gy, ey, rtol=0, atol=1e-12)


def test_render_matches_the_reference_generator(oracle):
    """ofc_synth_render against the reference's own renders (tests/golden/synth.npz) and, at 384 x 320 with a
    denser pattern, against the oracle's restatement: float64 images equal to 1e-12."""
    from optflow_b200 import synth
    from test_oracle import _synth_fields
    g = golden("synth")
    p = synth.make_pattern(64, 80, seed=3, rmin=1.5, rmax=2.5)
    for name, f in _synth_fields().items():
        assert np.abs(synth.render(p, 64, 80, f) - g[f"img_{name}"]).max() < 1e-12, name
    p = synth.make_pattern(320, 384, seed=5, rmin=1.5, rmax=4.0)
    for name, f in _synth_fields().items():
        assert np.abs(synth.render(p, 320, 384, f) - oracle.render(p, 320, 384, f)).max() < 1e-12, name


def test_render_with_grid_footing_and_bands(oracle):
    """The optional displacement terms of the renderer (a Gaussian-process grid, a footing settlement, finite shear
    bands) against the oracle's restatement, whose Newton inverse takes those terms' Jacobian by central differences:
    the two inverse maps meet at the same root, so the images agree to 1e-9."""
    from optflow_b200 import synth
    rng = np.random.default_rng(9)
    h, w = 288, 352
    grid, gx0, gy0 = synth.gp_grid(h, w, 96.0, 14.0, rng)
    f = synth.Field(grid=grid, gx0=gx0, gy0=gy0, footing=(3.0, 150.0, 140.0, 220.0, 40.0),
                    bands=[synth.Band((140.0, 40.0), (-0.7071067811865476, 0.7071067811865476), 6.0, 8.0, 180.0, 1.0),
                           synth.Band((220.0, 40.0), (0.7071067811865476, 0.7071067811865476), 6.0, 8.0, 180.0, 1.0)])
    p = synth.make_pattern(h, w, seed=4, rmin=1.5, rmax=2.5)
    assert np.abs(synth.render(p, h, w, f) - oracle.render(p, h, w, f)).max() < 1e-9


def test_fft_plan_orders_agree_and_tune():
    """Every factor order of a runtime plan computes the same transform (against numpy, as the default order), and
    the tuner returns an existing order per length."""
    from optflow_b200 import _abi, fftplan, testing
    lib = _abi.load()
    rng = np.random.default_rng(3)
    lengths = [320, 604, 1088]
    res = fftplan.tune(lengths, lines=256)
    for L in lengths:
        b, times = res[L]
        assert 0 <= b < lib.ofc_fft_plan_variants() and np.isfinite(times[b])
    x = (rng.normal(size=(8, 1088)) + 1j * rng.normal(size=(8, 1088))).astype(np.complex64)
    want = np.fft.fft(x.astype(np.complex128), axis=1)
    for v in range(lib.ofc_fft_plan_variants()):
        from optflow_b200 import Engine
        L = np.array([1088], np.int32)
        var = np.array([v], np.int32)
        lib.ofc_fft_set_plans(L.ctypes.data_as(_abi.c_i32_p), var.ctypes.data_as(_abi.c_i32_p), 1)
        got = testing.fft_lines(x, engine=Engine(0))  # a fresh engine builds its plan from the table
        assert np.abs(got - want).max() < 1e-5 * np.abs(want).max(), v
    zero = np.array([0], np.int32)
    lib.ofc_fft_set_plans(L.ctypes.data_as(_abi.c_i32_p), zero.ctypes.data_as(_abi.c_i32_p), 1)
    fftplan.install(force=True)  # the shipped table again
