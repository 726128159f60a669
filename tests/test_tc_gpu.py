"""K-d2: tcgen05 FP16 X stage.

Two bars: (1) on FP16 inputs the tensor-core result equals the FP64 product of
the same FP16 values up to FP32 accumulation (relative 1e-5); (2) through the
full FX path it is within 1e-3 relative amplitude and 0.05 degree phase of the
FP64 oracle, the precision the engine promises for the tensor-core path.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _fp64_vis(xr, xi):
    """xr, xi: [C][S][K] float64 -> V[C][P] with p = i(i+1)/2 + j."""
    X = xr + 1j * xi
    C, S, _ = X.shape
    full = np.einsum("csk,ctk->cst", X, np.conj(X))
    ii, jj = np.tril_indices(S)
    order = np.argsort(ii * (ii + 1) // 2 + jj)
    return full[:, ii[order], jj[order]]


@pytest.mark.parametrize("S,C,K", [(8, 3, 64), (128, 2, 96), (130, 2, 40), (256, 1, 128), (300, 2, 32)])
def test_xmac_f16_exact_inputs(cg, S, C, K):
    rng = np.random.default_rng(S + K)
    spec = rng.standard_normal((C, 2, S, K)).astype(np.float16)
    P = S * (S + 1) // 2
    vis = np.zeros((C, P), np.complex64)
    cg.xmac_f16(spec, S, C, K, vis)
    ref = _fp64_vis(spec[:, 0].astype(np.float64), spec[:, 1].astype(np.float64))
    err = np.linalg.norm(vis - ref) / np.linalg.norm(ref)
    assert err < 1e-5, err
    # lower triangle written, autos real
    ii = np.array([i for i in range(S) for _ in range(i + 1)])
    jj = np.array([j for i in range(S) for j in range(i + 1)])
    autos = vis[:, ii == jj]
    assert np.abs(autos.imag).max() <= 1e-5 * np.abs(autos.real).max()


@pytest.mark.parametrize("K", [8, 32, 40, 296])
@pytest.mark.parametrize("S", [1, 2, 7, 8, 9, 16, 17, 31, 32, 33, 63, 64, 65])
def test_xmac_f16_gram_sizes(cg, S, K):
    """Up to 64 inputs one Gram matrix holds every product: row counts on both sides of its operand sizes, time axes of
    part of a chunk, one and more than the ring holds; overwriting and accumulating."""
    rng = np.random.default_rng(100 * S + K)
    C = 5
    spec = rng.standard_normal((C, 2, S, K)).astype(np.float16)
    X = spec[:, 0].astype(np.float64) + 1j * spec[:, 1].astype(np.float64)
    i, j = np.tril_indices(S)
    ref = np.matmul(X, X.conj().transpose(0, 2, 1))[:, i, j]
    vis = np.full((C, i.size), np.nan, np.complex64)
    cg.xmac_f16(spec, S, C, K, vis)
    # FP16 products are exact in FP32; K-term FP32 sums without rounding to nearest
    assert np.linalg.norm(vis - ref) / np.linalg.norm(ref) < 1e-5
    cg.xmac_f16(spec, S, C, K, vis, accumulate=True)
    assert np.linalg.norm(vis - 2 * ref) / np.linalg.norm(ref) < 2e-5


@pytest.mark.parametrize("S,C,K", [(65, 400, 40), (127, 310, 264), (128, 160, 8), (129, 60, 72), (200, 52, 1528),
                                   (200, 3, 1536), (300, 60, 264), (513, 2, 1600)])
def test_xmac_f16_tile_rounds(cg, S, C, K):
    """Tiles of 128: several of them in turn on one SM and a partial last round, rows of part of a tile, time axes of
    part of a chunk and of more than the ring holds, and both sides of the line to a tile a block."""
    rng = np.random.default_rng(S + C)
    spec = rng.integers(-3, 4, (C, 2, S, K)).astype(np.float16)
    X = spec[:, 0].astype(np.float64) + 1j * spec[:, 1].astype(np.float64)
    i, j = np.tril_indices(S)
    ref = np.matmul(X, X.conj().transpose(0, 2, 1))[:, i, j]
    vis = np.full((C, i.size), np.nan, np.complex64)
    cg.xmac_f16(spec, S, C, K, vis)
    # whole numbers, sums below 2^24: exact in FP32 whatever the order
    assert np.array_equal(vis, ref)
    cg.xmac_f16(spec, S, C, K, vis, accumulate=True)
    assert np.array_equal(vis, 2 * ref)


@pytest.mark.parametrize("S", [40, 200])
def test_xmac_f16_accumulate(cg, S):
    """accumulate adds to the visibilities; S = 200 has diagonal tiles past the
    single-tile size (Im = M - M^T staged in the epilogue) and an edge tile."""
    rng = np.random.default_rng(1)
    C, K = 2, 64
    spec = rng.standard_normal((C, 2, S, K)).astype(np.float16)
    vis = np.zeros((C, S * (S + 1) // 2), np.complex64)
    cg.xmac_f16(spec, S, C, K, vis)
    v2 = vis.copy()
    cg.xmac_f16(spec, S, C, K, v2, accumulate=True)
    assert np.allclose(v2, 2 * vis, rtol=1e-6, atol=1e-4)


def test_fx_tc_accumulate_channel_grouped(cg):
    """FX with accumulate on the default N = 2048 tensor-core path (channel-grouped
    spectra, diagonal tiles past 128 inputs): a second call adds the same
    visibilities."""
    import synth

    S, N, K = 160, 2048, 64
    raw = synth.stations_offset_binary(S, N * K, rho=0.2, seed=41)
    P, C = S * (S + 1) // 2, N // 2
    vis = np.zeros((C, P), np.complex64)
    cg.fx_correlate(cg.fx_params(S, N, K, raw.shape[1], x_mode=cg.X_TC_FP16), raw, vis)
    v2 = vis.copy()
    cg.fx_correlate(cg.fx_params(S, N, K, raw.shape[1], x_mode=cg.X_TC_FP16, accumulate=True), raw, v2)
    assert np.allclose(v2, 2 * vis, rtol=1e-6, atol=1e-4)


def _fx_pair(cg, raw, S, N, K, mode, **kw):
    p = cg.fx_params(S, N, K, raw.shape[1], x_mode=mode, vis_order=cg.VIS_BASELINE_MAJOR, **kw)
    vis = np.zeros((S * (S + 1) // 2, N // 2), np.complex64)
    cg.fx_correlate(p, raw, vis, delay_poly=kw.get("delay_poly"))
    return vis


@pytest.mark.parametrize("S,N,K,rho", [(64, 2048, 256, 0.02), (32, 8192, 64, 0.5), (200, 1024, 128, 0.3)])
def test_fx_tc_vs_fp64_oracle(cg, orc, S, N, K, rho):
    import synth

    raw = synth.stations_offset_binary(S, N * K, rho=rho, seed=S * 7 + N)
    p = cg.fx_params(S, N, K, raw.shape[1], x_mode=cg.X_TC_FP16, vis_order=cg.VIS_BASELINE_MAJOR)
    vis = np.zeros((S * (S + 1) // 2, N // 2), np.complex64)
    cg.fx_correlate(p, raw, vis)
    # FP64 oracle on a seeded subset of products and channels, full K
    rng = np.random.default_rng(0)
    inputs = sorted(rng.choice(S, size=min(S, 12), replace=False))
    chans = sorted(rng.choice(N // 2, size=32, replace=False))
    X = orc.fx_spectra_f64(raw, S, N, K, inputs=inputs, channels=chans)
    pairs = [(a, b) for a in range(len(inputs)) for b in range(a + 1)]
    ref = orc.fx_vis_f64(X, pairs)
    got = np.stack([vis[orc.tri_index(inputs[a], inputs[b])][chans] for a, b in pairs])
    amp_err = np.linalg.norm(got - ref, axis=1) / np.linalg.norm(ref, axis=1)
    assert amp_err.max() < 1e-3, amp_err.max()
    # phase over channels whose |V| is above the thermal-noise floor
    # 3 sqrt(V_ii V_jj / K) (below it the phase is noise, not signal)
    auto = {a: ref[pairs.index((a, a))].real for a in range(len(inputs))}
    floor = np.stack([3 * np.sqrt(auto[a] * auto[b] / K) for a, b in pairs])
    mask = np.abs(ref) > floor
    phase_deg = np.degrees(np.abs(np.angle(got * np.conj(ref))))[mask]
    assert phase_deg.max() < 0.05, phase_deg.max()
    if rho >= 0.3:
        cross = np.array([a != b for a, b in pairs])
        assert mask[cross].mean() > 0.5      # the phase bar really covers cross products
    # and agrees with the FP32 CUDA-core path
    v32 = np.zeros_like(vis)
    cg.fx_correlate(cg.fx_params(S, N, K, raw.shape[1], x_mode=cg.X_FP32, vis_order=cg.VIS_BASELINE_MAJOR),
                    raw, v32)
    rel = np.linalg.norm(vis - v32, axis=1) / np.linalg.norm(v32, axis=1)
    assert rel.max() < 1e-3


def test_fx_tc_channel_scale(cg):
    """A per-(input, channel) scale before the FP16 cast is undone in the epilogue."""
    import synth

    S, N, K = 16, 1024, 64
    raw = synth.stations_offset_binary(S, N * K, rho=0.1, seed=3)
    base = _fx_pair(cg, raw, S, N, K, cg.X_TC_FP16)
    scale = np.random.default_rng(2).uniform(0.01, 0.05, (S, N // 2)).astype(np.float32)
    scaled = _fx_pair(cg, raw, S, N, K, cg.X_TC_FP16, channel_scale=scale)
    rel = np.linalg.norm(scaled - base) / np.linalg.norm(base)
    assert rel < 1e-3


def _tc_bars(orc, vis, X, pairs, K, sel=None, chans=None, cross_coverage=True):
    """1e-3 relative amplitude per product, 0.05 deg phase above the 3-sigma noise floor."""
    ref = orc.fx_vis_f64(X, pairs)
    got = vis if sel is None else np.stack([vis[p][chans] for p in sel])
    amp_err = np.linalg.norm(got - ref, axis=1) / np.linalg.norm(ref, axis=1)
    assert amp_err.max() < 1e-3, amp_err.max()
    auto = {a: ref[pairs.index((a, a))].real for a, b in pairs if a == b}
    floor = np.stack([3 * np.sqrt(auto[a] * auto[b] / K) for a, b in pairs])
    mask = np.abs(ref) > floor
    cross = np.array([a != b for a, b in pairs])
    if cross_coverage:
        assert mask[cross].mean() > 0.5
    phase_deg = np.degrees(np.abs(np.angle(got * np.conj(ref))))[mask]
    assert phase_deg.max() < 0.05, phase_deg.max()


@pytest.fixture(params=["0", "1"], ids=["warp-fft", "tc-fstage"])
def fstage_engine(request, monkeypatch):
    """N = 2048 FP16 spectra from the warp FFT (default) or the tensor-core F stage."""
    monkeypatch.setenv("CELLSPE_FSTAGE_TC", request.param)
    return request.param


@pytest.mark.parametrize("S,K,rho", [(24, 64, 0.5), (9, 72, 0.6), (40, 136, 0.4)])
def test_fx_tc_fstage_2048_vs_fp64(cg, orc, S, K, rho, fstage_engine):
    """N = 2048 with either F stage (tensor-core one: units of 8 segments over 9
    to 40 inputs; the X stage needs K % 8 == 0)."""
    import synth

    N = 2048
    raw = synth.stations_offset_binary(S, N * K, rho=rho, lags=np.arange(S) % 3, seed=S + K)
    p = cg.fx_params(S, N, K, raw.shape[1], x_mode=cg.X_TC_FP16, vis_order=cg.VIS_BASELINE_MAJOR)
    vis = np.zeros((S * (S + 1) // 2, N // 2), np.complex64)
    cg.fx_correlate(p, raw, vis)
    inputs = list(range(min(S, 8)))
    X = orc.fx_spectra_f64(raw, S, N, K, inputs=inputs)
    pairs = [(a, b) for a in range(len(inputs)) for b in range(a + 1)]
    sel = [orc.tri_index(inputs[a], inputs[b]) for a, b in pairs]
    _tc_bars(orc, vis, X, pairs, K, sel=sel, chans=slice(None))


def test_fx_tc_fstage_2048_delay_model(cg, orc, fstage_engine):
    """Integer shifts (start offsets at every sample alignment) and the fringe /
    fractional-delay phasor in the tensor-core F stage's epilogue."""
    import synth

    S, N, K = 5, 2048, 40
    fs, lo = 32e6, 8.4e9
    margin = 4096
    raw = synth.stations_offset_binary(S, N * K + 2 * margin, rho=0.5, seed=21)
    rng = np.random.default_rng(6)
    poly = np.zeros((S, 4))
    poly[:, 0] = rng.uniform(-40e-6, 40e-6, S)
    poly[:, 1] = rng.uniform(-2e-3, 2e-3, S)          # fast rates: the shift walks through alignments
    p = cg.fx_params(S, N, K, raw.shape[1], x_mode=cg.X_TC_FP16, vis_order=cg.VIS_BASELINE_MAJOR,
                     start_sample=margin, fs_hz=fs, lo_hz=lo)
    vis = np.zeros((S * (S + 1) // 2, N // 2), np.complex64)
    cg.fx_correlate(p, raw, vis, delay_poly=poly)
    shift, ph0, dph = orc.delay_state_f64(poly, N, K, fs, lo)
    assert len(set((shift.ravel() + margin) % 64)) > 20          # many sample alignments
    X = orc.fx_spectra_f64(raw, S, N, K, margin, shift, ph0, dph)
    pairs = [(i, j) for i in range(S) for j in range(i + 1)]
    # the random delays decorrelate the inputs: the phase bar covers the autos
    _tc_bars(orc, vis, X, pairs, K, cross_coverage=False)


@pytest.fixture(params=["0", "1", "2"], ids=["warp-fft", "tc32-fstage", "tc32-specialised"])
def fstage32(request, monkeypatch):
    """N = 2048 k-blocked FP16 spectra from the warp FFT or the 32-segment
    tensor-core F stage (real-input symmetry, k1 = 32 row via pass 2'), in its
    lockstep and its warp-specialised form."""
    monkeypatch.setenv("CELLSPE_FSTAGE_TC32", request.param)
    return request.param


@pytest.mark.parametrize("S,K,rho", [(24, 64, 0.5), (9, 96, 0.6), (40, 128, 0.4), (130, 64, 0.6)])
def test_fx_tc32_fstage_vs_fp64(cg, orc, S, K, rho, fstage32):
    """Every channel (the direct, mirrored and k1 = 32 families) of the
    tensor-core F stage through the full FX path: all products of the first 8
    inputs against the FP64 oracle, and the whole matrix against the FP32 path."""
    import synth

    N = 2048
    raw = synth.stations_offset_binary(S, N * K, rho=rho, lags=np.arange(S) % 5, seed=S * 3 + K)
    p = cg.fx_params(S, N, K, raw.shape[1], x_mode=cg.X_TC_FP16, vis_order=cg.VIS_BASELINE_MAJOR)
    vis = np.zeros((S * (S + 1) // 2, N // 2), np.complex64)
    cg.fx_correlate(p, raw, vis)
    inputs = list(range(min(S, 8)))
    X = orc.fx_spectra_f64(raw, S, N, K, inputs=inputs)
    pairs = [(a, b) for a in range(len(inputs)) for b in range(a + 1)]
    sel = [orc.tri_index(inputs[a], inputs[b]) for a, b in pairs]
    _tc_bars(orc, vis, X, pairs, K, sel=sel, chans=slice(None))
    v32 = np.zeros_like(vis)
    cg.fx_correlate(cg.fx_params(S, N, K, raw.shape[1], x_mode=cg.X_FP32, vis_order=cg.VIS_BASELINE_MAJOR),
                    raw, v32)
    rel = np.linalg.norm(vis - v32, axis=1) / np.linalg.norm(v32, axis=1)
    assert rel.max() < 1e-3


def test_fx_tc32_fstage_delay_model_and_scale(cg, orc, fstage32):
    """Integer shifts at every sample alignment, the fringe / fractional-delay
    phasor on all three channel families, and a per-(input, channel) scale."""
    import synth

    S, N, K = 5, 2048, 64
    fs, lo = 32e6, 8.4e9
    margin = 4096
    raw = synth.stations_offset_binary(S, N * K + 2 * margin, rho=0.5, seed=23)
    rng = np.random.default_rng(7)
    poly = np.zeros((S, 4))
    poly[:, 0] = rng.uniform(-40e-6, 40e-6, S)
    poly[:, 1] = rng.uniform(-2e-3, 2e-3, S)
    p = cg.fx_params(S, N, K, raw.shape[1], x_mode=cg.X_TC_FP16, vis_order=cg.VIS_BASELINE_MAJOR,
                     start_sample=margin, fs_hz=fs, lo_hz=lo)
    vis = np.zeros((S * (S + 1) // 2, N // 2), np.complex64)
    cg.fx_correlate(p, raw, vis, delay_poly=poly)
    shift, ph0, dph = orc.delay_state_f64(poly, N, K, fs, lo)
    X = orc.fx_spectra_f64(raw, S, N, K, margin, shift, ph0, dph)
    pairs = [(i, j) for i in range(S) for j in range(i + 1)]
    _tc_bars(orc, vis, X, pairs, K, cross_coverage=False)
    scale = np.random.default_rng(3).uniform(0.01, 0.05, (S, N // 2)).astype(np.float32)
    ps = cg.fx_params(S, N, K, raw.shape[1], x_mode=cg.X_TC_FP16, vis_order=cg.VIS_BASELINE_MAJOR,
                      start_sample=margin, fs_hz=fs, lo_hz=lo, channel_scale=scale)
    vs = np.zeros_like(vis)
    cg.fx_correlate(ps, raw, vs, delay_poly=poly)
    assert np.linalg.norm(vs - vis) / np.linalg.norm(vis) < 1e-3


@pytest.mark.parametrize("mode", ["tc", "fp32"])
@pytest.mark.parametrize("S,N,K", [(1, 4096, 8), (8, 4096, 72), (9, 4096, 24), (16, 8192, 136), (17, 4096, 40),
                                   (32, 4096, 264), (32, 16384, 24), (33, 4096, 40), (64, 4096, 96), (65, 4096, 32)])
def test_fx_segment_major_sizes(cg, orc, S, N, K, mode):
    """Long transforms: the X stage that reads segment-major spectra itself on both sides of its input counts, with
    time axes of part of a chunk, one chunk and more than its ring; the tensor-core form with a channel scale."""
    import synth

    raw = synth.stations_offset_binary(S, N * K, rho=0.3, seed=S + K)
    C, tc = N // 2, mode == "tc"
    scale = np.random.default_rng(S).uniform(0.5, 2.0, (S, C)).astype(np.float32) if tc else None
    p = cg.fx_params(S, N, K, raw.shape[1], x_mode=cg.X_TC_FP16 if tc else cg.X_FP32, channel_scale=scale)
    vis = np.full((C, S * (S + 1) // 2), np.nan, np.complex64)
    cg.fx_correlate(p, raw, vis)
    X = np.ascontiguousarray(orc.fx_spectra_f64(raw, S, N, K).transpose(2, 0, 1))
    i, j = np.tril_indices(S)
    ref = np.matmul(X, X.conj().transpose(0, 2, 1))[:, i, j]
    # FP16 spectra: 2^-12 per value, less over K; FP32: a few 2^-24
    assert np.linalg.norm(vis - ref) / np.linalg.norm(ref) < (1e-3 if tc else 2e-6)


@pytest.mark.parametrize("S,K", [(2, 8), (5, 64), (16, 72), (23, 128), (40, 64), (64, 136), (65, 64), (130, 64)])
@pytest.mark.parametrize("part", [0, 1])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_xmac_f16_infinite_values(cg, S, K, part, value):
    """One infinite (or NaN) Re or Im value of one input: what IEEE gives in its
    products, finite values everywhere else."""
    rng = np.random.default_rng(S + K)
    C, s = 3, S // 2
    x = rng.integers(1, 4, (C, 2, S, K)).astype(np.float16)
    x[1, part, s, K // 2] = value
    vis = np.zeros((C, S * (S + 1) // 2), np.complex64)
    cg.xmac_f16(x, S, C, K, vis)
    re, im = x[:, 0].astype(np.float64), x[:, 1].astype(np.float64)
    i, j = np.tril_indices(S)
    with np.errstate(invalid="ignore"):
        rr = (re[:, i] * re[:, j] + im[:, i] * im[:, j]).sum(-1)
        ri = (im[:, i] * re[:, j] - re[:, i] * im[:, j]).sum(-1)
    assert np.array_equal(vis.real, rr.astype(np.float32), equal_nan=True)
    assert np.array_equal(vis.imag, ri.astype(np.float32), equal_nan=True)


@pytest.mark.parametrize("S,C,K", [(129, 3, 1528), (129, 3, 1536), (192, 3, 1536), (193, 40, 1536), (193, 2, 1544), (257, 2, 2056),
                                   (300, 1, 2392), (300, 1, 2400)])
def test_xmac_f16_long_integrations(cg, S, C, K):
    """Both sides of the line in K, which moves with S, from which every tile has a block of its own."""
    test_xmac_f16_tile_rounds(cg, S, C, K)
