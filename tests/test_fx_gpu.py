"""Full FX path (K-a + K-b + K-c + K-d1) vs the oracle: FP32 CPU path and FP64 model."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = 1e-5   # FP32 GPU path vs the FP32 CPU path / FP64 model, relative L2


def _rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("S,N,K", [(3, 512, 40), (2, 1024, 64), (4, 2048, 40), (3, 4096, 9), (5, 8192, 4),
                                   (2, 32768, 2), (3, 2048, 13)])
def test_fx_fp32_vs_cpu_path(cg, orc, S, N, K):
    import synth

    raw = synth.stations_offset_binary(S, N * K, rho=0.2, lags=np.arange(S) % 4, seed=S + N)
    p = cg.fx_params(S, N, K, raw.shape[1], vis_order=cg.VIS_BASELINE_MAJOR)
    vis = np.zeros((S * (S + 1) // 2, N // 2), np.complex64)
    cg.fx_correlate(p, raw, vis)
    ref = orc.fx_fp32(raw, S, N, K)
    assert _rel(vis, ref) < TOL


def test_config1_lag_known_answer(cg, orc):
    """Config 1: 2 stations, 2^22 samples each, 1024-pt FFT, station 2 lags by 3 samples.

    V_10 = X_1 conj(X_0) with x_1(t) = c(t - 3) has phase -2 pi 3 k / N; its
    lag spectrum (inverse FFT over channels) peaks at lag +3.
    """
    import synth

    S, N, K = 2, 1024, 4096
    raw = synth.stations_offset_binary(S, N * K, rho=0.1, lags=[0, 3], seed=1)
    p = cg.fx_params(S, N, K, raw.shape[1], vis_order=cg.VIS_BASELINE_MAJOR)
    vis = np.zeros((3, N // 2), np.complex64)
    cg.fx_correlate(p, raw, vis)
    cross = vis[orc.tri_index(1, 0)].astype(np.complex128)
    k = np.arange(N // 2)
    derot = (cross * np.exp(2j * np.pi * 3 * k / N))[16:-16].reshape(-1, 16).sum(axis=1)
    assert np.abs(np.angle(derot)).max() < 0.15
    lag = np.fft.ifft(cross, n=N)
    assert int(np.argmax(np.abs(lag))) == 3
    coh = np.abs(cross) / np.sqrt(vis[0].real * vis[2].real)
    assert 0.06 < np.median(coh) < 0.12                        # 2-bit coherence ~ 0.88 rho


def test_fx_delay_model_vs_oracle(cg, orc):
    import synth

    S, N, K = 3, 2048, 24
    fs, lo = 32e6, 8.4e9
    margin = 4096
    T = N * K + 2 * margin
    raw = synth.stations_offset_binary(S, T, rho=0.3, seed=9)
    rng = np.random.default_rng(4)
    poly = np.zeros((S, 4))
    poly[:, 0] = rng.uniform(-40e-6, 40e-6, S)     # +-1280 samples
    poly[:, 1] = rng.uniform(-3e-6, 3e-6, S)
    poly[:, 2] = rng.uniform(-1e-9, 1e-9, S)
    p = cg.fx_params(S, N, K, raw.shape[1], vis_order=cg.VIS_BASELINE_MAJOR, start_sample=margin,
                     fs_hz=fs, lo_hz=lo)
    vis = np.zeros((S * (S + 1) // 2, N // 2), np.complex64)
    cg.fx_correlate(p, raw, vis, delay_poly=poly)
    shift, ph0, dph = orc.delay_state_f64(poly, N, K, fs, lo)
    c = np.arange(N // 2)
    phasor = np.exp(1j * (ph0.astype(np.float32)[:, :, None].astype(np.float64) +
                          c[None, None, :] * dph.astype(np.float32)[:, :, None].astype(np.float64))).astype(np.complex64)
    ref = orc.fx_fp32(raw, S, N, K, start_sample=margin, shift=shift, phasor=phasor)
    assert _rel(vis, ref) < TOL
    # and against the FP64 model
    X = orc.fx_spectra_f64(raw, S, N, K, margin, shift, ph0, dph)
    pairs = [(i, j) for i in range(S) for j in range(i + 1)]
    ref64 = orc.fx_vis_f64(X, pairs)
    assert _rel(vis, ref64) < TOL


def test_fx_layouts_memory_and_accumulate(cg):
    import torch

    import synth

    S, N, K = 6, 1024, 16
    raw = synth.stations_offset_binary(S, N * K, rho=0.1, seed=3)
    P, C = S * (S + 1) // 2, N // 2
    vb = np.zeros((P, C), np.complex64)
    cg.fx_correlate(cg.fx_params(S, N, K, raw.shape[1], vis_order=cg.VIS_BASELINE_MAJOR), raw, vb)
    vc = np.zeros((C, P), np.complex64)
    cg.fx_correlate(cg.fx_params(S, N, K, raw.shape[1], vis_order=cg.VIS_CHANNEL_MAJOR), raw, vc)
    assert np.array_equal(vb, vc.T)
    d_raw = torch.from_numpy(raw).cuda()
    d_vis = torch.zeros((C, P), dtype=torch.complex64, device="cuda")
    cg.fx_correlate(cg.fx_params(S, N, K, raw.shape[1]), d_raw, d_vis)
    assert np.array_equal(d_vis.cpu().numpy(), vc)
    cg.fx_correlate(cg.fx_params(S, N, K, raw.shape[1], accumulate=True), raw, vc)
    assert np.allclose(vc, 2 * d_vis.cpu().numpy(), rtol=1e-6, atol=1e-4)


def test_fx_rejects_bad_jobs(cg):
    raw = np.zeros((2, 1024), np.uint8)
    vis = np.zeros((3, 512), np.complex64)
    with pytest.raises(cg.CellspeError) as e:     # unsupported FFT size
        cg.fx_correlate(cg.fx_params(2, 1000, 1, 1024), raw, vis)
    assert e.value.code == cg.ERR_ARG
    with pytest.raises(cg.CellspeError) as e:     # segments past the end of the data
        cg.fx_correlate(cg.fx_params(2, 1024, 5, 1024), raw, vis)
    assert e.value.code == cg.ERR_ARG
    cg.lib().cellspe_set_hbm_budget(1 << 10)      # admission control
    try:
        with pytest.raises(cg.CellspeError) as e:
            cg.fx_correlate(cg.fx_params(2, 1024, 4, 1024), raw, vis)
        assert e.value.code == cg.ERR_NOMEM
    finally:
        cg.lib().cellspe_set_hbm_budget(0)


def test_xf_lags_match_backward_fft(cg, orc):
    """zerocorr lags (examples/zerocorr.c:391, 626-645): FFTW_BACKWARD of the visibilities, scaled 1/n."""
    import synth

    S, N, K = 2, 1024, 512
    raw = synth.stations_offset_binary(S, N * K, rho=0.2, lags=[0, 6], seed=21)
    vis = np.zeros((3, N // 2), np.complex64)
    cg.fx_correlate(cg.fx_params(S, N, K, raw.shape[1], vis_order=cg.VIS_BASELINE_MAJOR), raw, vis)
    lags = np.zeros_like(vis)
    cg.vis_lags(vis, lags, scale=1.0 / K)
    ref = np.fft.ifft(vis.astype(np.complex128), axis=1) * (N // 2) / K
    assert np.linalg.norm(lags - ref) / np.linalg.norm(ref) < 1e-5
    # x_1(t) = c(t - 6): V_10(k) = |C|^2 exp(-2 pi i k 6 / N) over the N/2 channels,
    # whose backward transform peaks at lag index 6 / 2 = 3 (two samples per index)
    cross = lags[orc.tri_index(1, 0)]
    assert int(np.argmax(np.abs(cross))) == 3
    assert np.abs(cross[3]) > 5 * np.abs(np.delete(cross, 3)).max()


@pytest.mark.parametrize("mode", ["tc", "fp32"])
def test_fx_host_buffers_streamed_match_device(cg, mode):
    """Host-buffer jobs of 64 MB or more move their input in blocks of inputs and
    their channel-major visibilities in blocks of channels on a copy stream,
    overlapping the F and X stages: bit-identical to the device-buffer run."""
    import torch

    import synth

    S, N, K = 128, 2048, 2048
    x_mode = cg.X_TC_FP16 if mode == "tc" else cg.X_FP32
    d_raw = synth.device_stations(S, N * K, 0.1, seed=12)
    raw = d_raw.cpu().numpy()
    assert raw.nbytes >= 64 << 20
    P, C = S * (S + 1) // 2, N // 2
    d_vis = torch.empty((C, P), dtype=torch.complex64, device="cuda")
    cg.fx_correlate(cg.fx_params(S, N, K, raw.shape[1], x_mode=x_mode), d_raw, d_vis)
    ref = d_vis.cpu().numpy()
    h_vis = np.zeros((C, P), np.complex64)
    cg.fx_correlate(cg.fx_params(S, N, K, raw.shape[1], x_mode=x_mode), raw, h_vis)
    assert np.array_equal(h_vis, ref)
    vb = np.zeros((P, C), np.complex64)              # baseline-major: streamed in only
    cg.fx_correlate(cg.fx_params(S, N, K, raw.shape[1], x_mode=x_mode, vis_order=cg.VIS_BASELINE_MAJOR), raw, vb)
    assert np.array_equal(vb, ref.T)


def test_direct_call_waits_for_prior_default_stream_work(cg):
    """A synchronous call on device buffers sees the data that work queued just
    before it on the default stream writes (the library's streams are
    non-blocking; each call first waits on the device for that stream)."""
    import torch

    import synth

    S, N, K = 64, 2048, 1024
    P, C = S * (S + 1) // 2, N // 2
    src = synth.device_stations(S, N * K, 0.1, seed=13)
    p = cg.fx_params(S, N, K, src.shape[1])
    want = torch.empty((C, P), dtype=torch.complex64, device="cuda")
    cg.fx_correlate(p, src, want)
    for _ in range(3):
        raw = torch.zeros_like(src)
        busy = torch.randn((4096, 4096), device="cuda")
        for _ in range(8):                       # keep the default stream busy for a while
            busy = busy @ busy.T / 4096.0
        raw.copy_(src)                           # queued behind the products, not yet done
        vis = torch.empty((C, P), dtype=torch.complex64, device="cuda")
        cg.fx_correlate(p, raw, vis)
        assert torch.equal(vis, want)


@pytest.mark.parametrize("mode", ["tc", "fp32"])
@pytest.mark.parametrize("K", [160, 104])
def test_fx_w2048_schedules_identical(cg, mode, K, monkeypatch):
    """The 2048-point F stage's CTA schedules, between which the autotuner
    picks by time alone, compute the same values: every forced schedule gives
    bit-identical visibilities (K = 160: whole 32-segment tiles; K = 104: a
    partial last tile and the planar layout)."""
    import torch

    import synth

    S, N = 16, 2048
    x_mode = cg.X_TC_FP16 if mode == "tc" else cg.X_FP32
    raw = synth.device_stations(S, N * K, 0.2, seed=17)
    P, C = S * (S + 1) // 2, N // 2
    outs = []
    for v in "12345":
        monkeypatch.setenv("CELLSPE_FSTAGE_VARIANT", v)
        vis = torch.empty((C, P), dtype=torch.complex64, device="cuda")
        cg.fx_correlate(cg.fx_params(S, N, K, raw.shape[1], x_mode=x_mode), raw, vis)
        outs.append(vis)
    for o in outs[1:]:
        assert torch.equal(o, outs[0])


@pytest.mark.parametrize("N,K", [(512, 40), (512, 128), (1024, 40), (1024, 128), (4096, 24), (8192, 16), (16384, 8),
                                 (32768, 8)])
def test_fx_warp_fstages_delay_model(cg, orc, N, K, monkeypatch):
    """The warp four-step F stages other than N = 2048: N = 512 and 1024 (a
    half-warp per segment, 16 or 32 points per lane; 64-segment tiles in FP16, 32
    in FP32 at N = 1024: K = 40 a partial tile, K = 128 full ones) and
    N = 4096 ... 32768 (N/2048 warps per segment, each a 1024-point transform of
    every (N/2048)-th point, then radix-N/2048 columns and the real-FFT split in
    registers).  FP32 path against the oracle's FP32 path with the same delay
    model and against the CTA-wide Stockham F stage; the tensor-core path (K a
    multiple of 8) against the same job through the Stockham F stage."""
    import synth

    S = 3
    fs, lo = 32e6, 8.4e9
    margin = 4096
    raw = synth.stations_offset_binary(S, N * K + 2 * margin, rho=0.3, seed=N + 7)
    rng = np.random.default_rng(N)
    poly = np.zeros((S, 4))
    poly[:, 0] = rng.uniform(-40e-6, 40e-6, S)
    poly[:, 1] = rng.uniform(-3e-6, 3e-6, S)
    kw = dict(vis_order=cg.VIS_BASELINE_MAJOR, start_sample=margin, fs_hz=fs, lo_hz=lo)
    P = S * (S + 1) // 2
    vis = np.zeros((P, N // 2), np.complex64)
    cg.fx_correlate(cg.fx_params(S, N, K, raw.shape[1], **kw), raw, vis, delay_poly=poly)
    shift, ph0, dph = orc.delay_state_f64(poly, N, K, fs, lo)
    c = np.arange(N // 2)
    phasor = np.exp(1j * (ph0.astype(np.float32)[:, :, None].astype(np.float64) +
                          c[None, None, :] * dph.astype(np.float32)[:, :, None].astype(np.float64))).astype(np.complex64)
    ref = orc.fx_fp32(raw, S, N, K, start_sample=margin, shift=shift, phasor=phasor)
    assert _rel(vis, ref) < TOL
    tc = np.zeros_like(vis)
    cg.fx_correlate(cg.fx_params(S, N, K, raw.shape[1], x_mode=cg.X_TC_FP16, **kw), raw, tc, delay_poly=poly)
    monkeypatch.setenv("CELLSPE_FSTAGE_GENERIC", "1")
    gen = np.zeros_like(vis)
    cg.fx_correlate(cg.fx_params(S, N, K, raw.shape[1], **kw), raw, gen, delay_poly=poly)
    assert _rel(vis, gen) < 2e-6
    gtc = np.zeros_like(vis)
    cg.fx_correlate(cg.fx_params(S, N, K, raw.shape[1], x_mode=cg.X_TC_FP16, **kw), raw, gtc, delay_poly=poly)
    assert _rel(tc, gtc) < 1e-3
    assert _rel(tc, ref) < 1e-3


def _vis_f64(orc, raw, S, N, K, start=0, state=(None, None, None), lut=None):
    """[C][P] FP64 visibilities, channel-major."""
    kw = {} if lut is None else {"lut": lut}
    X = orc.fx_spectra_f64(raw, S, N, K, start, *state, **kw)             # [S][K][C]
    A = np.ascontiguousarray(X.transpose(2, 0, 1))
    i, j = np.tril_indices(S)
    return np.matmul(A, A.conj().transpose(0, 2, 1))[:, i, j]


@pytest.mark.parametrize("S,N,K", [
    (8, 512, 96), (9, 512, 23),                      # a few inputs; fewer segments than the two-term form takes
    (9, 512, 24), (16, 512, 33), (17, 1024, 64), (32, 2048, 65),      # one row quarter, partial 32-segment blocks
    (33, 2048, 48), (64, 1024, 40), (65, 512, 100), (128, 512, 31),   # one tile of 64 and 128 rows
    (129, 512, 40), (200, 2048, 32), (257, 512, 25),                  # off-diagonal tiles, ragged last rows
    (40, 4096, 40), (12, 8192, 70), (10, 32768, 24)])                 # segment-major spectra
def test_fx_fp32_split_sizes(cg, orc, S, N, K):
    """FP32 jobs on both sides of every size the X stage's forms change at, against FP64."""
    import synth

    T = (N * K + 5 + 63) // 64 * 64
    raw = synth.stations_offset_binary(S, T, rho=0.2, seed=S + N)
    p = cg.fx_params(S, N, K, raw.shape[1], start_sample=5)
    vis = np.zeros((N // 2, S * (S + 1) // 2), np.complex64)
    cg.fx_correlate(p, raw, vis)
    # FP32 rounding of an N-point transform and of K-term sums: a few 2^-24, 2e-6 at most
    assert _rel(vis, _vis_f64(orc, raw, S, N, K, 5)) < 2e-6


@pytest.mark.parametrize("start", [4, 5])
@pytest.mark.parametrize("N", [4096, 8192, 16384, 32768])
def test_fx_long_transforms(cg, orc, N, start):
    """Long transforms at even and odd first samples against FP64, every channel; with a channel scale against without."""
    import synth

    S, K = 9, 5                                      # a remainder of the 32768-point form's four segments a block
    raw = synth.stations_offset_binary(S, (N * K + start + 63) // 64 * 64, rho=0.3, seed=N + start)
    C, P = N // 2, S * (S + 1) // 2
    vis = np.zeros((C, P), np.complex64)
    cg.fx_correlate(cg.fx_params(S, N, K, raw.shape[1], start_sample=start), raw, vis)
    ref = _vis_f64(orc, raw, S, N, K, start)
    # FP32 rounding of an N-point transform and of a few sums: a few 2^-24, 2e-6 at most
    assert _rel(vis, ref) < 2e-6
    for c in (0, 1, 512, 1024, C // 2, C // 2 + 512, C - 512, C - 1):     # the mirrored columns' special cases
        assert _rel(vis[c], ref[c]) < 1e-5, c
    # FP16 spectra under a scale of powers of two are the same but for halves too small to be normal
    raw, K8 = np.concatenate([raw, raw], axis=1), 8
    scale = np.exp2(np.random.default_rng(N).integers(-1, 2, (S, C))).astype(np.float32)
    out = []
    for sc in (None, scale):
        out.append(np.zeros((C, P), np.complex64))
        cg.fx_correlate(cg.fx_params(S, N, K8, raw.shape[1], start_sample=start, x_mode=cg.X_TC_FP16, channel_scale=sc), raw, out[-1])
    assert _rel(out[1], out[0]) < 1e-5


@pytest.mark.parametrize("N", [512, 1024, 2048, 4096])
def test_fx_fp32_split_delay_levels(cg, orc, N):
    """The same with a delay model, large custom levels and a full-scale tone (the largest spectrum value of these levels)."""
    import synth

    S, K, fs, lo, margin = 20, 70, 32e6, 1e6, 2048
    T = N * K + 2 * margin
    raw = synth.stations_offset_binary(S, T, rho=0.3, seed=N)
    raw[3] = 0b11000011                              # codes 3, 0, 0, 3: +-level square wave, one channel takes N max|level| / sqrt 2
    poly = np.zeros((S, 4))
    rng = np.random.default_rng(N)
    poly[:, 0] = rng.uniform(-30e-6, 30e-6, S)
    poly[:, 1] = rng.uniform(-3e-6, 3e-6, S)
    levels = np.array([-3.0e4, -1.1e4, 0.9e4, 3.1e4], np.float32)
    p = cg.fx_params(S, N, K, raw.shape[1], start_sample=margin, fs_hz=fs, lo_hz=lo, custom_levels=levels)
    vis = np.zeros((N // 2, S * (S + 1) // 2), np.complex64)
    cg.fx_correlate(p, raw, vis, delay_poly=poly)
    ref = _vis_f64(orc, raw, S, N, K, margin, orc.delay_state_f64(poly, N, K, fs, lo), levels)
    i, j = np.tril_indices(S)
    for q in (i != 3) & (j != 3), (i == 3) & (j != 3):        # the tone's own products do not hide the others
        # the phasor's angle is FP32: up to N/2 dphase rad, 2^-24 of a few hundred rad
        assert _rel(vis[:, q], ref[:, q]) < TOL


SPLIT_FORMS = [
    (9, 512, 64), (16, 1024, 65), (17, 2048, 160), (33, 512, 127), (64, 512, 66),     # a Gram matrix of 16, 32, 64 inputs
    (9, 4096, 64), (16, 8192, 129), (32, 4096, 95), (40, 4096, 64),                   # segment-major spectra, and 33 inputs on
    (65, 512, 64), (72, 1024, 257), (128, 512, 300), (129, 512, 64), (200, 512, 287)]     # one tile, several


@pytest.mark.parametrize("S,N,K", SPLIT_FORMS + [(16, 512, 63), (65, 512, 63)])
def test_fx_fp32_split_exact_sums(cg, S, N, K):
    """Constant inputs, whose products and sums in channel 0 are whole numbers that FP32 holds: bit for bit."""
    levels = np.array([-3, -1, 1, 3], np.float32)
    code = np.arange(S) % 4
    raw = np.repeat((code * 0b01010101).astype(np.uint8)[:, None], N * K // 4 + 16, axis=1)
    p = cg.fx_params(S, N, K, raw.shape[1], custom_levels=levels)
    vis = np.full((N // 2, S * (S + 1) // 2), np.nan, np.complex64)
    cg.fx_correlate(p, raw, vis)
    i, j = np.tril_indices(S)
    ref = (levels[code[i]] * levels[code[j]]).astype(np.float64) * K * N * N
    assert ref.max() < 2.0 ** 24 * N * N                  # multiples of N^2: exact
    assert np.array_equal(vis[0].real, ref) and not vis[0].imag.any()


@pytest.mark.parametrize("S,N,K", SPLIT_FORMS)
def test_fx_fp32_split_edges(cg, orc, S, N, K):
    """The two-term forms at their own smallest sizes and partial blocks against FP64, the autos by themselves too."""
    import synth

    raw = synth.stations_offset_binary(S, (N * K + 63) // 64 * 64, rho=0.2, seed=S + N + 1)
    vis = np.zeros((N // 2, S * (S + 1) // 2), np.complex64)
    cg.fx_correlate(cg.fx_params(S, N, K, raw.shape[1]), raw, vis)
    ref = _vis_f64(orc, raw, S, N, K)
    # FP32 rounding of an N-point transform and of K-term sums: a few 2^-24, 2e-6 at most
    assert _rel(vis, ref) < 2e-6
    i, j = np.tril_indices(S)
    assert _rel(vis[:, i == j], ref[:, i == j]) < 2e-6
    assert not vis[:, i == j].imag.any()


@pytest.mark.parametrize("S,N,K,levels", [
    (20, 2048, 70, (-1e6, -1, 1, 1e6)), (70, 512, 80, (-1e4, -1, 1, 1e4)), (12, 4096, 64, (-1, 1e-5, -1e-5, 1)),
    (20, 1024, 64, (-1e5, 0, 1, 1e5))])
def test_fx_fp32_levels_rarely_taken(cg, orc, S, N, K, levels):
    """Custom levels of which the data never takes the large ones: FP32 spectra do not depend on those."""
    rng = np.random.default_rng(N)
    codes = rng.integers(1, 3, (S, (N * K + 63) // 64 * 64)).astype(np.uint8).reshape(S, -1, 4)
    raw = np.ascontiguousarray(codes[..., 0] | codes[..., 1] << 2 | codes[..., 2] << 4 | codes[..., 3] << 6)
    levels = np.array(levels, np.float32)
    vis = np.zeros((N // 2, S * (S + 1) // 2), np.complex64)
    cg.fx_correlate(cg.fx_params(S, N, K, raw.shape[1], custom_levels=levels), raw, vis)
    ref = _vis_f64(orc, raw, S, N, K, lut=levels)
    # FP32 rounding of an N-point transform and of K-term sums: a few 2^-24, 2e-6 at most
    # (channel 0 holds the mean of levels that have one: it does not hide the others)
    assert _rel(vis[1:], ref[1:]) < 2e-6


def test_stage_times_are_the_last_good_jobs(cg):
    """A job that fails after its F stage (the FP16 X stage takes K in multiples of 8) leaves the times of the one before."""
    import torch

    import synth

    S, N, K = 8, 512, 512
    raw = synth.device_stations(S, N * K, 0.1, seed=1)
    vis = torch.zeros((N // 2, S * (S + 1) // 2), dtype=torch.complex64, device="cuda")
    good = cg.fx_params(S, N, K, raw.shape[1], x_mode=cg.X_TC_FP16)
    bad = cg.fx_params(S, N, 7, raw.shape[1], x_mode=cg.X_TC_FP16)

    def fail():
        with pytest.raises(cg.CellspeError):
            cg.fx_correlate(bad, raw, vis)

    cg.fx_correlate(good, raw, vis)                  # first use: kernels are loaded
    cg.fx_correlate(good, raw, vis)
    before = cg.stage_times()
    assert min(before) >= 0 and before[1] > 0
    fail()
    assert cg.stage_times() == before                # read before the failing job
    cg.fx_correlate(good, raw, vis)
    cg.fx_correlate(good, raw, vis)
    fail()
    fail()
    t = cg.stage_times()                             # and read only after it
    assert min(t) >= 0 and t[1] > 0.5 * before[1] and t[2] > 0.5 * before[2]


def test_fx_baseline_major_into_any_address(cg):
    """Baseline-major visibilities into a device buffer that is no multiple of 8 bytes: by a copy."""
    import torch

    import synth

    S, N, K = 5, 512, 64
    raw = synth.device_stations(S, N * K, 0.1, seed=2)
    n = S * (S + 1) // 2 * (N // 2)
    p = cg.fx_params(S, N, K, raw.shape[1], vis_order=cg.VIS_BASELINE_MAJOR, memory=cg.MEM_DEVICE)
    ref = torch.zeros(2 * n, device="cuda")
    buf = torch.zeros(2 * n + 2, device="cuda")
    torch.cuda.synchronize()
    for dst in (ref, buf[1:]):
        assert cg.lib().cellspe_fx_correlate(ctypes.byref(p), raw.data_ptr(), None, dst.data_ptr()) == 0
    assert torch.equal(buf[1:-1], ref) and ref.any() and buf[0] == 0 and buf[-1] == 0


@pytest.mark.parametrize("S,N,K", [(4, 512, 64), (8, 1024, 100), (24, 2048, 96), (24, 4096, 32), (32, 8192, 64), (33, 4096, 64),
                                   (40, 8192, 24)])
@pytest.mark.parametrize("mode", [0, 1, 2])
def test_fx_workspace_estimate_is_what_a_job_takes(cg, mode, S, N, K):
    """cellspe_fx_workspace_bytes (which counts a delay model) against the scratch
    that jobs took: host and device buffers, both orders, accumulation, delays, scale."""
    import torch

    if mode == cg.X_INT8 and K % 16:
        pytest.skip("the INT8 X stage takes segments in multiples of 16")
    if mode == cg.X_TC_FP16 and K % 8:
        K -= K % 8
    C, P, margin = N // 2, S * (S + 1) // 2, 4096
    a256 = lambda n: (n + 255) // 256 * 256
    raw = torch.randint(0, 256, (S, (N * K + 2 * margin) // 4), dtype=torch.uint8)
    poly = np.zeros((S, 4))
    poly[:, 0] = np.linspace(-20e-6, 20e-6, S)
    scale = np.ones((S, C), np.float32) if mode == cg.X_TC_FP16 else None
    for dev in (False, True):
        x = raw.cuda() if dev else raw.numpy()
        for order in (cg.VIS_CHANNEL_MAJOR, cg.VIS_BASELINE_MAJOR):
            for acc, delays, sc in ((False, False, None), (True, False, None), (False, True, None), (False, False, scale)):
                shape = (P, C) if order == cg.VIS_BASELINE_MAJOR else (C, P)
                vis = torch.zeros(shape, dtype=torch.complex64, device="cuda") if dev else np.zeros(shape, np.complex64)
                if sc is not None and dev:
                    sc = torch.from_numpy(sc).cuda()
                p = cg.fx_params(S, N, K, raw.shape[1], x_mode=mode, vis_order=order, start_sample=margin, fs_hz=32e6,
                                 accumulate=acc, memory=cg.MEM_DEVICE if dev else cg.MEM_HOST, channel_scale=sc)
                pl = (torch.from_numpy(poly).cuda() if dev else poly) if delays else None
                cg.fx_correlate(p, x, vis, delay_poly=pl)
                need = cg.lib().cellspe_fx_workspace_bytes(ctypes.byref(p))
                if not delays:
                    need -= 3 * a256(S * K * 4) + (0 if dev else a256(S * 32))
                assert cg.lib().cellspe_debug_workspace_taken() == need, (dev, order, acc, delays, sc is not None)
