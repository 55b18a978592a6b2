"""The benchmark's host-side parts."""
import json
import os
import sys

import numpy as np
import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if REPO not in sys.path:
    sys.path.insert(0, REPO)

import bench  # noqa: E402


def test_a_missing_reference_library_does_not_cost_the_line(monkeypatch):
    """The reference's sources may not be at hand: the line then says why its CPU baseline
    is missing.  Any other failure of that baseline is still an error."""
    def missing(*args, **kwargs):
        raise OSError("libhsi_ref.so: cannot open shared object file")

    monkeypatch.setattr(bench, "cpu_reference", missing)
    cpu = bench.cpu_baseline("sam_cem")
    assert list(cpu) == ["unavailable"] and "libhsi_ref.so" in cpu["unavailable"]
    json.dumps(cpu)

    def broken(*args, **kwargs):
        raise ValueError("shape")

    monkeypatch.setattr(bench, "cpu_reference", broken)
    with pytest.raises(ValueError):
        bench.cpu_baseline("sam_cem")
    monkeypatch.setattr(bench, "cpu_reference", lambda *a, **k: (np.array([0.5, 1.5]), 4, 250000))
    cpu = bench.cpu_baseline("rx_ace", " (all of it)")
    assert cpu["value"] == 1.0 and cpu["cores"] == 4 and "(all of it)" in cpu["sample"]


def _kernels(fn):
    """Kernel nodes of one captured call."""
    import torch
    from cuda.bindings import runtime
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    fn(stream)  # one-time set-up
    stream.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph, stream=stream):
        fn(stream)
    g = runtime.cudaGraph_t(graph.raw_cuda_graph())
    err, _, n = runtime.cudaGraphGetNodes(g)
    assert err == runtime.cudaError_t.cudaSuccess
    err, nodes, n = runtime.cudaGraphGetNodes(g, n)
    assert err == runtime.cudaError_t.cudaSuccess and len(nodes) >= n
    kinds = [runtime.cudaGraphNodeGetType(node) for node in nodes[:n]]
    assert all(k[0] == runtime.cudaError_t.cudaSuccess for k in kinds)
    return sum(k[1] == runtime.cudaGraphNodeType.cudaGraphNodeTypeKernel for k in kinds)


@pytest.mark.gpu
@pytest.mark.parametrize("bands", [16, 127, 128, 224, 252, 253, 254, 255])
@pytest.mark.parametrize("side", [180, 200])
def test_launch_counts_of_moments(hsi, bands, side):
    import torch
    cube = torch.rand((bands, hsi.plane_stride(side, side)), device="cuda")
    out = torch.empty(hsi.moments_elements(bands), dtype=torch.float64, device="cuda")
    ws = torch.empty(hsi.stats_workspace_bytes(side, side, bands), dtype=torch.uint8, device="cuda")
    n = _kernels(lambda s: hsi.scene_moments(cube, side, side, bands, out=out, workspace=ws, stream=s))
    assert n == bench.moments_launches([(side * side, bands)])


@pytest.mark.gpu
@pytest.mark.parametrize("bands, targets", [(113, 8), (113, 16), (127, 3), (16, 16), (113, 0)])
def test_launch_counts_of_rx_ace(hsi, bands, targets):
    import torch
    P = 4096
    cube = torch.rand((bands, P), device="cuda")
    out = torch.empty(P, device="cuda")
    stats = torch.zeros(hsi.statistics_elements(bands, targets), dtype=torch.float64, device="cuda")
    for plain in (False, True):
        size = hsi.lib().hsi_rx_ace_simt_workspace_bytes if plain else hsi.lib().hsi_rx_ace_workspace_bytes
        ws = torch.empty(size(bands, targets), dtype=torch.uint8, device="cuda")
        n = _kernels(lambda s: hsi.rx_ace(cube, 64, 64, bands, stats, targets, rx=out, simt=plain, workspace=ws,
                                          stream=s))
        assert n == bench.rx_ace_launches(bands, targets, not plain)


@pytest.mark.gpu
def test_launch_counts_of_the_batch_runner(hsi):
    """Mosaics, both moments routes, several target passes and more than 64 lists."""
    import torch
    specs = [(200, 256, (16, 113, 224)[k % 3], 1 + 15 * (k % 2), k % 3 == 0) for k in range(24)]
    gen = torch.Generator(device="cuda").manual_seed(1)
    frames = []
    for h, w, b, t, mosaic in specs:
        targets = np.random.default_rng(b).random((t, b)).astype(np.float32)
        if mosaic:
            raw = torch.rand((4 * h, 4 * w), generator=gen, device="cuda")
            frames.append(dict(raw=raw, period=4, bands=b, targets=targets))
        else:
            cube = torch.rand((b, hsi.plane_stride(h, w)), generator=gen, device="cuda")
            frames.append(dict(cube=cube, height=h, width=w, bands=b, dtype=hsi.F32, targets=targets))
    batch = hsi.Batch(frames, autotune=False)
    n = _kernels(batch.run)
    batch.close()
    assert n == bench.batch_launches(specs)
