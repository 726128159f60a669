"""cellspe_fx_correlate_async on a caller's stream, captured into a CUDA graph.

After one call has sized the thread's workspace (and the first-use tables and
schedule choices exist), the asynchronous entry point issues only stream work,
so it can be captured and replayed; the replay must reproduce the blocking
call bit for bit.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1])
def test_fx_async_graph_replay_matches_blocking_call(cg, mode):
    import torch

    import synth

    S, N, K = 16, 2048, 64
    raw = torch.from_numpy(synth.stations_offset_binary(S, N * K, rho=0.1, seed=7)).cuda()
    P = S * (S + 1) // 2
    ref = torch.zeros((N // 2, P), dtype=torch.complex64, device="cuda")
    p = cg.fx_params(S, N, K, raw.shape[1], x_mode=mode, memory=cg.MEM_DEVICE)
    cg.fx_correlate(p, raw, ref)
    s = torch.cuda.Stream()
    vis = torch.zeros_like(ref)
    with torch.cuda.stream(s):
        cg.fx_correlate_async(p, raw, vis, s.cuda_stream)          # sizes the workspace
    torch.cuda.synchronize()
    assert torch.equal(vis, ref)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s, capture_error_mode="relaxed"):
        cg.fx_correlate_async(p, raw, vis, torch.cuda.current_stream().cuda_stream)
    vis.zero_()
    torch.cuda.synchronize()
    for _ in range(2):
        g.replay()
    torch.cuda.synchronize()
    assert torch.equal(vis, ref)


@pytest.mark.parametrize("S", [16, 24, 200])
@pytest.mark.parametrize("mode", [0, 1])
def test_fx_async_after_a_timed_out_wait(cg, mode, S):
    """A wait that ran out in an earlier asynchronous job on the stream (a kernel
    whose one wait has a short limit) costs that job alone: a job queued behind
    it and every replay of a captured one still write their visibilities."""
    import torch

    import synth

    N, K = 2048, 128
    raw = torch.from_numpy(synth.stations_offset_binary(S, N * K, rho=0.1, seed=8)).cuda()
    ref = torch.zeros((N // 2, S * (S + 1) // 2), dtype=torch.complex64, device="cuda")
    p = cg.fx_params(S, N, K, raw.shape[1], x_mode=mode, memory=cg.MEM_DEVICE)
    cg.fx_correlate(p, raw, ref)
    s = torch.cuda.Stream()
    vis = torch.zeros_like(ref)
    cg.fx_correlate_async(p, raw, vis, s.cuda_stream)              # sizes the workspace
    torch.cuda.synchronize()
    vis.zero_()
    torch.cuda.synchronize()
    assert cg.lib().cellspe_debug_wait_timeout(1, 1, s.cuda_stream) == 0
    cg.fx_correlate_async(p, raw, vis, s.cuda_stream)
    torch.cuda.synchronize()
    assert torch.equal(vis, ref)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s, capture_error_mode="relaxed"):
        cg.fx_correlate_async(p, raw, vis, torch.cuda.current_stream().cuda_stream)
    for stage in (0, 1):
        vis.zero_()
        torch.cuda.synchronize()
        assert cg.lib().cellspe_debug_wait_timeout(stage, 1, s.cuda_stream) == 0
        with torch.cuda.stream(s):
            g.replay()
        torch.cuda.synchronize()
        assert torch.equal(vis, ref)
    # and the blocking call that comes next is good too, with nothing left to report
    vis.zero_()
    cg.fx_correlate(p, raw, vis)
    assert torch.equal(vis, ref)


@pytest.mark.parametrize("stage,name", [(0, "F stage"), (1, "X stage")])
def test_timed_out_wait_is_reported_once(cg, stage, name):
    """The error record reaches the host and names its stage; the next job is clean."""
    import torch

    import synth

    S, N, K = 16, 2048, 64
    raw = torch.from_numpy(synth.stations_offset_binary(S, N * K, rho=0.1, seed=7)).cuda()
    p = cg.fx_params(S, N, K, raw.shape[1], x_mode=cg.X_TC_FP16, memory=cg.MEM_DEVICE)
    ref = torch.zeros((N // 2, S * (S + 1) // 2), dtype=torch.complex64, device="cuda")
    cg.fx_correlate(p, raw, ref)
    assert cg.lib().cellspe_debug_wait_timeout(stage, 0, None) == cg.ERR_CUDA
    assert name in cg.last_error() and "timed out" in cg.last_error()
    vis = torch.zeros_like(ref)
    cg.fx_correlate(p, raw, vis)
    assert torch.equal(vis, ref)
