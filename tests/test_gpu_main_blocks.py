"""The main-bin kernels are launched with the number of blocks that the tuning asks for."""

import json

import pytest

from larndsim_gb300 import consts, sim, tune, workloads

pytestmark = pytest.mark.gpu


def _grid(name, tmp_path, run):
    """x extent of the grid of the kernel with that name, from a trace."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as p:
        run()
        torch.cuda.synchronize()
    p.export_chrome_trace(str(tmp_path / "t.json"))
    events = json.loads((tmp_path / "t.json").read_text())["traceEvents"]
    grids = [e["args"]["grid"][0] for e in events if e.get("cat") == "kernel" and name in e["name"]]
    return grids[0] if grids else None


@pytest.mark.parametrize("blocks,warps", [(1024, 0), (341, 0), (342, 0), (1024, 8), (2048, 4), (3, 0)])
def test_asked_for_blocks(cuda, tmp_path, blocks, warps):
    import torch
    params = consts.Params(number_pix_neighbors=4)
    lut, params = sim.load_lut(workloads.synthetic_response(seed=0), params)
    tracks, fields = workloads.batched_events(seed=3, n_events=2, min_segments=300, max_segments=400)
    t = torch.from_numpy(tracks).cuda()
    want, _ = sim.simulate_wfs(params, lut, t, fields)
    try:
        tune.set_tuning({"main_blocks": blocks, "main_block_warps": warps})
        got = []
        for _ in range(2):     # a process's first trace may hold no kernels
            grid = _grid("k_main_records", tmp_path, lambda: got.append(sim.simulate_wfs(params, lut, t, fields)[0]))
    finally:
        tune.set_tuning(None)
    n = min(got[0].shape[0], want.shape[0])
    assert torch.equal(got[0][:n], want[:n])
    if grid is None:
        pytest.skip("no kernel records in the trace")
    assert grid == blocks
