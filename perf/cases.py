"""Performance cases: the engine's main calls over the range they are used on.

FX correlation jobs (2-bit samples to visibilities) from the smallest job of
the serving mix to the 512-input array, with the tensor-core and the FP32 X
stage, with and without the delay model; spectrometer jobs (power spectra and
phase-cal) of interleaved, plane and framed VDIF input; batched real FFTs.
Inputs and outputs are device buffers that the caller owns.

A case is a dict of plain values; ``listed`` gives the fixed ones, ``draw``
one more from the same ranges, ``prepare`` the buffers and parameters that a
program holds before the call, ``run`` one call, ``work`` the bytes and
operations a call cannot do without, ``exact`` the outputs in 64 bits.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cellspe-tasklib_gb300"))
import cellspe_gpu as cg  # noqa: E402

THRESH = 0.98                                        # 2-bit quantiser threshold in sigma
OFFSET_BINARY = (-3.336, -1.0, 1.0, 3.336)           # levels of codes 0..3, FX jobs
MARK5B = (-3.3359, 1.0, -1.0, 3.3359)                # spectrometer, Mark5B
VDIF = (-3.3359, -1.0, 1.0, 3.3359)                  # spectrometer, VDIF
MARGIN = 66048                                       # samples around a delayed stream (2 ms at 32 MS/s and more)
FS, LO = 32e6, 8.4e9                                 # sample rate and sky frequency of the delay-tracked jobs
VDIF_BYTES = 8000                                    # payload of a VDIF frame


def _fx(name, S, N, K, mode, delay=False, start=0, order="baseline"):
    return {"name": name, "kind": "fx", "S": S, "N": N, "K": K, "mode": mode, "delay": delay, "start": start,
            "order": order}


def _spec(name, nsub, N, overlap, window, K, nspec, layout, pcal):
    return {"name": name, "kind": "spec", "nsub": nsub, "N": N, "overlap": overlap, "window": window, "K": K,
            "nspec": nspec, "layout": layout, "pcal": pcal}


def listed():
    return [
        # the serving mix's smallest job: 4 inputs, 256 channels, 2^18 samples each; latency and launches
        _fx("fx-small-tc", 4, 512, 512, "tc"),
        # two stations, one polarisation, 1024-point transform over 2^22 samples, FP32 (the plain correlator job)
        _fx("fx-pair-fp32", 2, 1024, 4096, "fp32"),
        # a middle job of the mix with ragged sizes: 24 inputs but one, a segment count that fills no tile, an odd
        # first sample, channel-major output
        _fx("fx-ragged-tc", 23, 2048, 1928, "tc", start=5, order="channel"),
        # 16 stations, two polarisations, cubic delay models, 8192-point transforms over one second, both X stages
        _fx("fx-delay-tc", 32, 8192, 4096, "tc", delay=True),
        _fx("fx-delay-fp32", 32, 8192, 4096, "fp32", delay=True),
        # the mix's 200-input job at 1024 channels in FP32
        _fx("fx-array-fp32", 200, 2048, 4096, "fp32", order="channel"),
        # the mix's largest job: 200 inputs, 16384 channels, 2^24 samples each
        _fx("fx-wide-tc", 200, 32768, 512, "tc", order="channel"),
        # 256 stations, two polarisations, 1024 channels, 4096 spectra per integration
        _fx("fx-512-tc", 512, 2048, 4096, "tc", order="channel"),
        # one second of a 16-channel Mark5B recording at 32 MS/s, 32768 spectral channels, phase-cal at 1 MHz
        _spec("spec-mark5b-64k", 16, 65536, 2, 2, 512, 1, "interleaved", True),
        # a wide-band single channel at 1024 points, many folded transforms per spectrum (the swspectrometer's
        # benchmark shape)
        _spec("spec-plane-1k", 1, 1024, 2, 2, 8192, 16, "planes", False),
        # a framed 4-channel VDIF recording with some invalid frames, 8192 points, phase-cal
        _spec("spec-vdif-8k", 4, 8192, 2, 4, 1000, 3, "vdif", True),
        # batched real transforms of the task API's usual length
        {"name": "rfft-2k", "kind": "rfft", "n": 2048, "batch": 65536},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fx", "fx", "fx", "spec", "spec", "rfft"])
    if kind == "fx":
        mode = rng.choice(["tc", "fp32"])
        N = 1 << rng.randint(9, 15)
        S = _logint(rng, 2, 240)
        T = _logint(rng, 1 << 18, 1 << 24)
        if mode == "fp32":
            T = min(T, max(1 << 18, (200 * 200 << 23) // (S * S)))
        K = max(8, T // N)
        if rng.random() < 0.5:
            K = max(8, K // 32 * 32)                 # whole 32-segment blocks as often as not
        if mode == "tc":
            K = K // 8 * 8                           # the tensor-core X stage takes multiples of 8
        c = _fx("", S, N, K, mode, delay=rng.random() < 0.4, start=rng.choice([0, 0, 3, 16, 37]),
                order=rng.choice(["baseline", "channel"]))
    elif kind == "spec":
        layout = rng.choice(["interleaved", "planes", "vdif"])
        nsub = rng.choice([1, 4, 8, 16])
        N = 1 << rng.randint(10, 16)
        overlap = rng.choice([1, 2, 2, 4])
        total = _logint(rng, 1 << 22, 1 << 28)       # samples of all subbands
        nspec = rng.choice([1, 1, 2, 3, 5, 16])
        K = max(2, total // nsub // N // nspec)
        c = _spec("", nsub, N, overlap, rng.randint(0, 5), K, nspec, layout, rng.random() < 0.5)
    else:
        n = 1 << rng.randint(7, 15)
        c = {"kind": "rfft", "n": n, "batch": max(1, _logint(rng, 1 << 16, 1 << 27) // n)}
    c.pop("name", None)
    return c


# ---- inputs -------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    return g


def _quantise(x):
    """Offset-binary codes 0..3 (uint8) of samples in sigma."""
    return (x >= -THRESH).to(torch.uint8) + (x >= 0).to(torch.uint8) + (x >= THRESH).to(torch.uint8)


def _pack(codes):
    """uint8 codes [..., 4 n] -> bytes [..., n], first code in bits 1:0."""
    c = codes.view(*codes.shape[:-1], -1, 4)
    return c[..., 0] | (c[..., 1] << 2) | (c[..., 2] << 4) | (c[..., 3] << 6)


def _stations(S, T, rho, seed):
    """uint8 [S][T/4]: inputs that share a sky signal with correlation rho."""
    g = _gen(seed)
    raw = torch.empty((S, T // 4), dtype=torch.uint8, device="cuda")
    step = 1 << 22
    for t0 in range(0, T, step):
        n = min(step, T - t0)
        sky = torch.randn(n, generator=g, device="cuda") * math.sqrt(rho)
        for s0 in range(0, S, 64):
            s1 = min(S, s0 + 64)
            x = torch.randn((s1 - s0, n), generator=g, device="cuda").mul_(math.sqrt(1 - rho)).add_(sky)
            raw[s0:s1, t0 // 4:(t0 + n) // 4] = _pack(_quantise(x))
    return raw


def _fx_samples(case):
    """Samples per input (a multiple of 64) and the first segment's sample."""
    first = case["start"] + (MARGIN if case["delay"] else 0)
    need = first + case["N"] * case["K"] + (MARGIN if case["delay"] else 0)
    return (need + 63) // 64 * 64, first


def _delays(S, seed):
    """float64 [S][4] seconds: up to +-2 ms, +-3 us/s, small curvature."""
    r = np.random.RandomState(seed & 0x7FFFFFFF)
    return np.stack([r.uniform(-2e-3, 2e-3, S), r.uniform(-3e-6, 3e-6, S), r.uniform(-1e-9, 1e-9, S),
                     r.uniform(-1e-13, 1e-13, S)], axis=1)


def _subband_codes(c, T, seed):
    """Offset-binary codes (uint8) of one subband: noise, a 1 MHz comb at 32 MS/s and three sinusoids."""
    g = _gen(seed * 64 + c)
    r = np.random.RandomState((seed * 64 + c) & 0x7FFFFFFF)
    t = np.arange(32)
    comb = 0.05 * sum(np.cos(2 * np.pi * k * t / 32 + r.uniform(0, 2 * np.pi)) for k in range(1, 16))
    comb = torch.from_numpy(comb).float().cuda()
    freq, amp = r.uniform(0.05, 0.45, 3), 0.02
    codes = torch.empty(T, dtype=torch.uint8, device="cuda")
    step = 1 << 24
    for t0 in range(0, T, step):
        n = min(step, T - t0)
        x = torch.randn(n, generator=g, device="cuda")
        at = torch.arange(t0, t0 + n, device="cuda")
        x += comb[at & 31]
        for f in freq:
            x += amp * torch.cos((2 * math.pi * ((at * float(f)) % 1.0)).float())
        codes[t0:t0 + n] = _quantise(x)
    return codes


def _spec_samples(case):
    """Samples per subband that the input carries."""
    T = case["N"] * case["K"] * case["nspec"]
    if case["layout"] == "vdif":
        per = VDIF_BYTES * 4 // case["nsub"]
        return max(2, -(-T // per)) * per
    return (T + 63) // 64 * 64


def _invalid_frames(nframes, seed):
    """Frames marked invalid: about one in a hundred, never the first."""
    bad = np.random.RandomState((seed + 5) & 0x7FFFFFFF).rand(nframes) < 0.01
    bad[0] = False
    return bad


def _vdif(payload, nsub, bad):
    """Payload bytes [frames][VDIF_BYTES] with VDIF headers in front (bytes of the whole recording)."""
    nf = payload.shape[0]
    mbps = int(FS * 2 * nsub / 1e6)
    fps = mbps * 1000000 // (8 * VDIF_BYTES)
    n = np.arange(nf, dtype=np.int64)
    h = np.zeros((nf, 8), np.uint32)
    h[:, 0] = (7654321 + n // fps).astype(np.uint32) | (bad.astype(np.uint32) << np.uint32(31))
    h[:, 1] = (n % fps).astype(np.uint32) | np.uint32(40 << 24)
    h[:, 2] = np.uint32(((VDIF_BYTES + 32) // 8) | ((nsub.bit_length() - 1) << 24))
    h[:, 3] = np.uint32(1 << 26)
    head = torch.from_numpy(h.view(np.uint8).reshape(nf, 32)).cuda()
    return torch.cat([head, payload], dim=1).reshape(-1).contiguous()


def _spec_input(case, seed):
    nsub, T, layout = case["nsub"], _spec_samples(case), case["layout"]
    table = torch.tensor([0, 1, 2, 3] if layout == "vdif" else [0, 2, 1, 3], dtype=torch.uint8, device="cuda")
    if layout == "planes":
        return torch.cat([_pack(table[_subband_codes(c, T, seed).int()]) for c in range(nsub)])
    codes = torch.empty((T, nsub), dtype=torch.uint8, device="cuda")
    for c in range(nsub):
        codes[:, c] = table[_subband_codes(c, T, seed).int()]
    raw = _pack(codes.view(-1))
    if layout == "vdif":
        raw = raw.view(-1, VDIF_BYTES)
        raw = _vdif(raw, nsub, _invalid_frames(raw.shape[0], seed))
    return raw


def prepare(case, seed):
    seed = int(seed)
    if case["kind"] == "rfft":
        x = torch.randn((case["batch"], case["n"]), generator=_gen(seed), device="cuda")
        out = torch.empty((case["batch"], case["n"] // 2 + 1), dtype=torch.complex64, device="cuda")
        return {"kind": "rfft", "x": x, "out": out, "n": case["n"], "batch": case["batch"]}
    if case["kind"] == "spec":
        nsub, nspec, N = case["nsub"], case["nspec"], case["N"]
        raw = _spec_input(case, seed)
        layout = {"interleaved": cg.SPEC_INTERLEAVED, "planes": cg.SPEC_PLANES, "vdif": cg.SPEC_VDIF_FRAMED}[case["layout"]]
        pc = dict(tonebins=32, rotatorlen=32, ntones=16) if case["pcal"] else {}
        p = cg.spec_params(N, case["overlap"], case["window"], case["K"], nspec, nsub, raw.numel(), layout=layout,
                           levels=cg.LEVELS_VDIF if case["layout"] == "vdif" else cg.LEVELS_MARK5B, fs_hz=FS, **pc)
        st = {"kind": "spec", "p": p, "raw": raw, "bins": None, "tones": None,
              "power": torch.zeros((nsub, nspec, N // 2 + 1), device="cuda")}
        if case["pcal"]:
            st["bins"] = torch.zeros((nsub, nspec, 32), dtype=torch.complex64, device="cuda")
            st["tones"] = torch.zeros((nsub, nspec, 16), dtype=torch.complex64, device="cuda")
        return st
    S, N, K = case["S"], case["N"], case["K"]
    T, first = _fx_samples(case)
    raw = _stations(S, T, 0.1, seed)
    order = cg.VIS_CHANNEL_MAJOR if case["order"] == "channel" else cg.VIS_BASELINE_MAJOR
    P = S * (S + 1) // 2
    p = cg.fx_params(S, N, K, T // 4, x_mode=cg.X_TC_FP16 if case["mode"] == "tc" else cg.X_FP32, vis_order=order,
                     start_sample=first, fs_hz=FS if case["delay"] else 0.0, lo_hz=LO if case["delay"] else 0.0)
    vis = torch.zeros((N // 2, P) if case["order"] == "channel" else (P, N // 2), dtype=torch.complex64, device="cuda")
    poly = torch.from_numpy(_delays(S, seed)).cuda() if case["delay"] else None
    return {"kind": "fx", "p": p, "raw": raw, "vis": vis, "poly": poly}


def run(state):
    if state["kind"] == "fx":
        return cg.fx_correlate(state["p"], state["raw"], state["vis"], state["poly"])
    if state["kind"] == "spec":
        cg.spectrometer(state["p"], state["raw"], state["power"], state["bins"], state["tones"])
        out = {"power": state["power"]}
        if state["bins"] is not None:
            out.update(bins=state["bins"], tones=state["tones"])
        return out
    return cg.fft_r2c(state["x"], state["out"], state["n"], state["batch"])


def work(case):
    if case["kind"] == "rfft":
        n, b = case["n"], case["batch"]
        return {"bytes": b * (4 * n + 8 * (n // 2 + 1)), "flops": b * 2.5 * n * math.log2(n)}
    if case["kind"] == "spec":
        N, rows = case["N"], case["nsub"] * case["nspec"]
        novl = case["overlap"] * case["K"] - (case["overlap"] - 1)
        return {"bytes": rows * case["K"] * N / 4 + rows * (N // 2 + 1) * 4,
                "flops": rows * novl * (2.5 * N * math.log2(N) + N + 2 * N)}
    S, N, K = case["S"], case["N"], case["K"]
    P = S * (S + 1) // 2
    return {"bytes": S * K * N / 4 + (N // 2) * P * 8.0,
            "flops": S * K * 2.5 * N * math.log2(N) + 8.0 * (N // 2) * P * K}


# ---- 64-bit values ------------------------------------------------------------
def _decode64(raw, levels):
    """Bytes [..., n] -> float64 samples [..., 4 n]."""
    table = torch.tensor(levels, dtype=torch.float32, device="cuda").double()
    shifts = torch.tensor([0, 2, 4, 6], dtype=torch.uint8, device="cuda")
    codes = (raw.unsqueeze(-1) >> shifts) & 3
    return table[codes.reshape(*raw.shape[:-1], -1).int()]


def _exact_fx(case, seed):
    S, N, K = case["S"], case["N"], case["K"]
    C, P = N // 2, S * (S + 1) // 2
    T, first = _fx_samples(case)
    raw = _stations(S, T, 0.1, seed)
    X = torch.empty((S, K, C), dtype=torch.complex128, device="cuda")
    poly = _delays(S, seed) if case["delay"] else None
    c = torch.arange(C, dtype=torch.float64, device="cuda")
    t = (np.arange(K, dtype=np.float64) * N + N / 2) / FS
    step = max(1, (1 << 27) // N)
    for s in range(S):
        x = _decode64(raw[s], OFFSET_BINARY)
        if poly is None:
            for k0 in range(0, K, step):
                k1 = min(K, k0 + step)
                X[s, k0:k1] = torch.fft.rfft(x[first + k0 * N:first + k1 * N].view(k1 - k0, N))[:, :C]
            continue
        tau = ((poly[s, 3] * t + poly[s, 2]) * t + poly[s, 1]) * t + poly[s, 0]
        shift = np.rint(tau * FS)
        cycles = LO * tau
        phase = torch.from_numpy(2 * np.pi * (cycles - np.floor(cycles))).cuda()
        dphase = torch.from_numpy(2 * np.pi * (FS / N) * (tau - shift / FS)).cuda()
        at = torch.from_numpy(first + np.arange(K) * N + shift.astype(np.int64)).cuda()
        n = torch.arange(N, device="cuda")
        for k0 in range(0, K, step):
            k1 = min(K, k0 + step)
            Y = torch.fft.rfft(x[at[k0:k1, None] + n[None, :]])[:, :C]
            ph = phase[k0:k1, None] + c[None, :] * dphase[k0:k1, None]
            X[s, k0:k1] = Y * torch.polar(torch.ones_like(ph), ph)
    i, j = torch.tril_indices(S, S, device="cuda")
    vis = torch.empty((C, P), dtype=torch.complex128, device="cuda")
    step = max(1, (1 << 28) // (S * K + S * S))
    for c0 in range(0, C, step):
        A = X[:, :, c0:c0 + step].permute(2, 0, 1).contiguous()
        vis[c0:c0 + step] = torch.bmm(A, A.conj().transpose(1, 2))[:, i, j]
    return vis if case["order"] == "channel" else vis.t().contiguous()


def _window64(kind, N):
    i = torch.arange(N, dtype=torch.float64, device="cuda")
    c = torch.cos(math.pi * (i - 0.5 * N + 0.5) / N)
    x = 2 * math.pi * i / (N - 1)
    return {0: torch.ones_like(i), 1: c, 2: c * c, 3: 0.54 - 0.46 * torch.cos(x), 4: 0.5 - 0.5 * torch.cos(x),
            5: 0.75 - 0.5 * torch.cos(x) - 0.25 * torch.cos(2 * x)}[kind]


def _exact_spec(case, seed):
    nsub, nspec, N, K, ov = case["nsub"], case["nspec"], case["N"], case["K"], case["overlap"]
    T, layout = _spec_samples(case), case["layout"]
    table = torch.tensor(OFFSET_BINARY, device="cuda")
    table = torch.where(table.abs() > 2, table.sign() * 3.3359, table).float().double()
    w = _window64(case["window"], N)
    novl, hop = ov * K - (ov - 1), N // ov
    power = torch.zeros((nsub, nspec, N // 2 + 1), dtype=torch.float64, device="cuda")
    bins = torch.zeros((nsub, nspec, 32), dtype=torch.complex128, device="cuda")
    step = max(1, (1 << 26) // N)
    for c in range(nsub):
        x = table[_subband_codes(c, T, seed).int()]
        if layout == "vdif":
            per = VDIF_BYTES * 4 // nsub
            bad = torch.from_numpy(_invalid_frames(T // per, seed)).cuda()
            x = torch.where(bad[:, None], torch.zeros_like(x.view(-1, per)), x.view(-1, per)).view(-1)
        for s in range(nspec):
            win = x[s * K * N:(s + 1) * K * N].unfold(0, N, hop)
            for j0 in range(0, novl, step):
                X = torch.fft.rfft(win[j0:j0 + step] * w)
                power[c, s] += (X.real ** 2 + X.imag ** 2).sum(0)
            fold = [j for j in range(novl) if (s * novl + j) % ov == 0]
            if case["pcal"] and fold:
                bins[c, s] = win[fold[0]::ov][:len(fold)].sum(0).view(-1, 32).sum(0)
    power /= novl
    if not case["pcal"]:
        return {"power": power}
    k = torch.arange(32, dtype=torch.float64, device="cuda")
    W = torch.polar(torch.ones((16, 32), dtype=torch.float64, device="cuda"), -2 * math.pi * torch.outer(k[:16], k) / 32)
    return {"power": power, "bins": bins, "tones": bins @ W.t() / 32}


def exact(case, seed):
    seed = int(seed)
    if case["kind"] == "fx":
        return _exact_fx(case, seed)
    if case["kind"] == "spec":
        return _exact_spec(case, seed)
    st = prepare(case, seed)
    return torch.fft.rfft(st["x"].double())
