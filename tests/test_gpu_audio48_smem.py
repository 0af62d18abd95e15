"""What the 48 kHz resampler reserves in shared memory: its arms in float64 and
its input window in float32, and no more than a rounding of each -- resident CTAs
hide its latencies.  Read from the launches that a profile records."""
import json
import math

import pytest

import gpudemod as G

pytestmark = pytest.mark.gpu

TAPS = 33  # per arm


@pytest.mark.parametrize("rate,decim,mode,outputs", [
    (24_000, 50, "NFM", 1024),   # four outputs per thread
    (12_500, 64, "NFM", 768),    # blocks of 4 x 96
    (312_500, 8, "WFM", 256),    # stereo, one output per thread
])
def test_shared_memory_of_a_tile(cuda, tmp_path, rate, decim, mode, outputs):
    import torch
    from torch.profiler import ProfilerActivity, profile
    n = rate * decim // 10
    r = G.ChannelRunner(rate * decim, n, max_channels=2, max_taps=256)
    try:
        m, bw, ch = (G.MODE_NFM, 0.4 * rate, 1) if mode == "NFM" else (G.MODE_WFM_STEREO, 180_000.0, 2)
        r.admit(1, 0.0, bw, rate, 65, m, G.CH_AUDIO48K)
        x = torch.randn(n, dtype=torch.complex64, device="cuda")
        torch.cuda.synchronize()
        r.process_block(x)
        with profile(activities=[ProfilerActivity.CUDA]) as p:
            for _ in range(10):  # a profile may miss launches at its start
                r.process_block(x)
            torch.cuda.synchronize()
    finally:
        r.close()
    trace = tmp_path / "trace.json"
    p.export_chrome_trace(str(trace))
    used = [e["args"]["shared memory"] for e in json.loads(trace.read_text())["traceEvents"]
            if "k_audio48_rs" in e.get("name", "") and "shared memory" in e.get("args", {})]
    assert used, "the resampler's launch is not in the profile"
    g = math.gcd(rate, 48_000)
    up, down = 48_000 // g, rate // g
    need = 8 * up * TAPS + 4 * ch * ((outputs - 1) * down // up + TAPS)
    assert max(used) <= need + 8 + 4 * ch * 4 + 1024, (used, need)  # the GPU's own 1 KB per CTA, where it is counted
