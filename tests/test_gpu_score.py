"""GPU parity: SAM / CEM filter-bank scoring against the FP64 oracle.

Cubes are generated on the device and read back, so both sides see the same
bits.  Tolerances (stated here, checked below):
  SAM angle  : |gpu - oracle| <= 2e-3 rad everywhere (the reference's own GPU
               gate, bench/bench_sam.cu:56) and <= 1e-4 rad where the angle is
               >= 0.02 rad (acos is ill-conditioned at 0);
  SAM label  : a different best target is allowed only where the oracle's
               angles of the two targets are within 2e-3 rad
               (bench/bench_sam.cu:156-183);
  CEM        : |gpu - oracle| <= 1e-5 * sum_b |w_b x_b| + 1e-6.
"""
import re

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SAM_TOL = 2e-3
SAM_TOL_TIGHT = 1e-4


def _download(cube, B, P):
    return cube[:, :P].float().cpu().numpy().reshape(B, P)


def _check_sam(orc, host, targets, gpu_best, gpu_target, gpu_maps=None):
    T = targets.shape[0]
    allm = orc.sam_all(host, targets)
    best, which = orc.sam_best(host, targets)
    err = np.abs(gpu_best - best)
    assert err.max() <= SAM_TOL, f"max angle error {err.max()}"
    far = best >= 0.02
    if far.any():
        assert err[far].max() <= SAM_TOL_TIGHT, f"max angle error away from 0: {err[far].max()}"
    mism = np.nonzero(gpu_target != which)[0]
    for p in mism:
        g = gpu_target[p]
        assert 0 <= g < T
        assert abs(allm[g, p] - best[p]) <= SAM_TOL
    if gpu_maps is not None:
        merr = np.abs(gpu_maps - allm)
        assert merr.max() <= SAM_TOL
        if far.any():
            farm = allm >= 0.02
            assert merr[farm].max() <= SAM_TOL_TIGHT
    return err.max()


def _run(hsi, cube, H, W, B, dtype, sam=None, cem=None, maps=True):
    P = H * W
    dev = cube.device
    out = {}
    kw = {}
    if sam is not None:
        kw["sam_targets"] = torch.from_numpy(np.ascontiguousarray(sam, np.float32)).to(dev)
        kw["sam_norms"] = torch.from_numpy(hsi.target_norms(sam)).to(dev)
        out["sam_best"] = torch.full((P,), -7.0, device=dev)
        out["sam_best_target"] = torch.full((P,), -7, dtype=torch.int32, device=dev)
        if maps:
            out["sam_maps"] = torch.full((sam.shape[0], P), -7.0, device=dev)
    if cem is not None:
        kw["cem_weights"] = torch.from_numpy(np.ascontiguousarray(cem, np.float32)).to(dev)
        out["cem_best"] = torch.full((P,), -7.0, device=dev)
        out["cem_best_target"] = torch.full((P,), -7, dtype=torch.int32, device=dev)
        if maps:
            out["cem_maps"] = torch.full((cem.shape[0], P), -7.0, device=dev)
    f = hsi.make_frame(cube, H, W, B, dtype, map_stride=P, **kw, **out)
    hsi.score_frames([f])
    torch.cuda.synchronize()
    return {k: v.cpu().numpy() for k, v in out.items()}


@pytest.mark.parametrize("dtype", [0, 1])
@pytest.mark.parametrize("T", [1, 4, 8])
def test_sam_generated_scene(hsi, orc, dtype, T):
    H, W, B = 52, 70, 113
    sc = hsi.scene(B, n_targets=T, target_frac=0.01, frame_seed=0x5EED0000 + T)
    cube, _ = hsi.generate(sc, H, W, dtype=dtype)
    host = _download(cube, B, H * W)
    targets = hsi.scene_targets(sc)
    r = _run(hsi, cube, H, W, B, dtype, sam=targets)
    _check_sam(orc, host, targets, r["sam_best"], r["sam_best_target"], r["sam_maps"])


@pytest.mark.parametrize("B", [1, 3, 16, 113, 127, 224, 256])
@pytest.mark.parametrize("shape", [(1, 1), (7, 13), (33, 17), (64, 64)])
def test_sam_shapes_and_band_counts(hsi, orc, B, shape):
    H, W = shape
    sc = hsi.scene(B, n_targets=3, target_frac=0.05, frame_seed=B * 1000 + H)
    cube, _ = hsi.generate(sc, H, W)
    host = _download(cube, B, H * W)
    targets = hsi.scene_targets(sc)
    r = _run(hsi, cube, H, W, B, 0, sam=targets)
    _check_sam(orc, host, targets, r["sam_best"], r["sam_best_target"], r["sam_maps"])


def test_sam_reference_cases(hsi, orc, golden):
    for name in ("identical", "zero", "best"):
        host = golden[f"case_{name}_cube"]
        targets = golden[f"case_{name}_targets"]
        B, H, W = host.shape
        stride = hsi.plane_stride(H, W)
        cube = torch.zeros((B, stride), device="cuda")
        cube[:, : H * W] = torch.from_numpy(host.reshape(B, -1)).cuda()
        r = _run(hsi, cube, H, W, B, 0, sam=targets)
        np.testing.assert_array_equal(r["sam_best_target"], golden[f"case_{name}_target"])
        assert np.max(np.abs(r["sam_best"] - golden[f"case_{name}_score"])) <= SAM_TOL
        assert not np.isnan(r["sam_best"]).any()
    # the orthogonal and the all-zero pixel are exactly pi/2 (no NaN)
    host = golden["case_zero_cube"]
    cube = torch.zeros((4, 32), device="cuda")
    cube[:, :2] = torch.from_numpy(host.reshape(4, -1)).cuda()
    r = _run(hsi, cube, 1, 2, 4, 0, sam=golden["case_zero_targets"])
    np.testing.assert_allclose(r["sam_best"], np.float32(np.pi / 2), atol=1e-6)


def test_sam_scale_invariance(hsi):
    rng = np.random.default_rng(7)
    t = rng.uniform(0.05, 1.0, (1, 16)).astype(np.float32)
    px = rng.uniform(0.05, 1.0, 16).astype(np.float32)
    gains = np.array([1.0, 0.01, 0.5, 3.0, 250.0], np.float32)
    host = (px[:, None] * gains[None, :]).astype(np.float32)
    cube = torch.zeros((16, 32), device="cuda")
    cube[:, :5] = torch.from_numpy(host).cuda()
    r = _run(hsi, cube, 1, 5, 16, 0, sam=t)
    assert np.max(np.abs(r["sam_best"] - r["sam_best"][0])) < 1e-4


def test_multi_pass_library(hsi, orc):
    """More than 16 targets: several passes, best carried through the outputs."""
    H, W, B = 40, 50, 64
    sc = hsi.scene(B, n_targets=20, target_frac=0.01, frame_seed=4)
    cube, _ = hsi.generate(sc, H, W)
    host = _download(cube, B, H * W)
    targets = hsi.scene_targets(sc)
    rng = np.random.default_rng(1)
    cem = rng.standard_normal((37, B)).astype(np.float32) * 0.1
    r = _run(hsi, cube, H, W, B, 0, sam=targets, cem=cem)
    _check_sam(orc, host, targets, r["sam_best"], r["sam_best_target"], r["sam_maps"])
    _check_cem(orc, host, cem, r)


def _check_cem(orc, host, cem, r):
    w64 = cem.astype(np.float64)
    stats = {"cem_weight": w64}
    best, which, allm = orc.cem(host, stats)
    mag = np.abs(w64) @ np.abs(host.astype(np.float64))
    tol = 1e-5 * mag + 1e-6
    assert (np.abs(r["cem_maps"] - allm) <= tol).all()
    assert (np.abs(r["cem_best"] - best) <= tol.max(axis=0)).all()
    mism = np.nonzero(r["cem_best_target"] != which)[0]
    for p in mism:
        g = r["cem_best_target"][p]
        assert abs(allm[g, p] - best[p]) <= 2 * tol[:, p].max()


@pytest.mark.parametrize("dtype", [0, 1])
def test_cem_with_scene_statistics(hsi, orc, dtype):
    H, W, B = 64, 64, 113
    sc = hsi.scene(B, n_targets=8, target_frac=0.002, frame_seed=0x5EED1001)
    cube, _ = hsi.generate(sc, H, W, dtype=dtype)
    host = _download(cube, B, H * W)
    targets = hsi.scene_targets(sc)
    s, o, n = orc.moments(host)
    st, S = orc.build_statistics(s, o, n, targets, 1e-6)
    assert st == 0
    cem = S["cem_weight"].astype(np.float32)
    r = _run(hsi, cube, H, W, B, dtype, sam=targets, cem=cem)
    _check_sam(orc, host, targets, r["sam_best"], r["sam_best_target"], r["sam_maps"])
    _check_cem(orc, host, cem, r)
    # against the FP64 weights themselves (what the statistics say the response is)
    best64, _, all64 = orc.cem(host, S)
    assert np.max(np.abs(r["cem_maps"] - all64)) < 1e-4


@pytest.mark.parametrize("max_sam,max_cem", [(4, 4), (8, 8), (8, 4)])
def test_sam_and_cem_banks_of_uneven_sizes(hsi, orc, max_sam, max_cem):
    """One device table whose frames carry fewer filters than the launch
    bounds (down to none of one kind): both banks are scored by one
    warpgroup, and empty slots must neither score nor write."""
    counts = [(max_sam, max_cem), (max_sam - 1, 0), (1, max_cem - 1), (0, max_cem)]
    frames, keep = [], []
    for i, (ns, nc) in enumerate(counts):
        H, W, B = 40 + i, 48, 113 - 20 * i
        sc = hsi.scene(B, n_targets=max(ns, nc, 1), target_frac=0.02, frame_seed=300 + i, library_seed=31 + i)
        cube, _ = hsi.generate(sc, H, W)
        lib = hsi.scene_targets(sc)
        P = H * W
        kw, out = {}, {}
        if ns:
            kw["sam_targets"] = torch.from_numpy(np.ascontiguousarray(lib[:ns])).cuda()
            kw["sam_norms"] = torch.from_numpy(hsi.target_norms(lib[:ns])).cuda()
            out["sam_best"] = torch.full((P,), -7.0, device="cuda")
            out["sam_best_target"] = torch.full((P,), -7, dtype=torch.int32, device="cuda")
            out["sam_maps"] = torch.full((ns, P), -7.0, device="cuda")
        cem = None
        if nc:
            rng = np.random.default_rng(40 + i)
            cem = (rng.standard_normal((nc, B)) / B).astype(np.float32)
            kw["cem_weights"] = torch.from_numpy(cem).cuda()
            out["cem_best"] = torch.full((P,), -7.0, device="cuda")
            out["cem_best_target"] = torch.full((P,), -7, dtype=torch.int32, device="cuda")
            out["cem_maps"] = torch.full((nc, P), -7.0, device="cuda")
        frames.append(hsi.make_frame(cube, H, W, B, 0, map_stride=P, **kw, **out))
        keep.append((cube, lib[:ns], cem, out, H, W, B, kw))
    table = hsi.frame_table(frames)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    hsi.score_frames_device(table, len(frames), max_bands=113, max_sam=max_sam, max_cem=max_cem, status=status)
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    for cube, targets, cem, out, H, W, B, _ in keep:
        host = _download(cube, B, H * W)
        r = {k: v.cpu().numpy() for k, v in out.items()}
        if targets.shape[0]:
            _check_sam(orc, host, targets, r["sam_best"], r["sam_best_target"], r["sam_maps"])
        if cem is not None:
            _check_cem(orc, host, cem, r)


@pytest.mark.parametrize("B", [16, 113, 128])
@pytest.mark.parametrize("T", [(8, 8), (3, 0), (0, 5), (16, 16), (20, 9)])
def test_fp16_tensor_core_and_fma_scorers_match_the_oracle(hsi, orc, B, T):
    """FP16 cubes of at most 128 bands with host descriptors take the
    tensor-core scorer; descriptors in device memory take the FP32-FMA scorer.
    Both must meet the same tolerances against the FP64 oracle, including
    passes of more than 16 filters of a kind (20 SAM targets: two passes that
    carry the best), CEM weights of small magnitude (the per-filter power-of-two
    scale), and a last tile shorter than 128 pixels."""
    ns, nc = T
    H, W = 37, 101
    sc = hsi.scene(B, n_targets=max(ns, nc, 1), target_frac=0.03, frame_seed=500 + B + ns, library_seed=61 + nc)
    cube, _ = hsi.generate(sc, H, W, dtype=1)
    host = _download(cube, B, H * W)
    lib = hsi.scene_targets(sc)
    rng = np.random.default_rng(B + 7 * nc)
    cem = (rng.standard_normal((nc, B)) * 1e-3).astype(np.float32) if nc else None
    P = H * W
    for tensor_cores in (True, False):
        kw, out = {}, {}
        if ns:
            kw["sam_targets"] = torch.from_numpy(np.ascontiguousarray(lib[:ns])).cuda()
            kw["sam_norms"] = torch.from_numpy(hsi.target_norms(lib[:ns])).cuda()
            out["sam_best"] = torch.full((P,), -7.0, device="cuda")
            out["sam_best_target"] = torch.full((P,), -7, dtype=torch.int32, device="cuda")
            out["sam_maps"] = torch.full((ns, P), -7.0, device="cuda")
        if nc:
            kw["cem_weights"] = torch.from_numpy(cem).cuda()
            out["cem_best"] = torch.full((P,), -7.0, device="cuda")
            out["cem_best_target"] = torch.full((P,), -7, dtype=torch.int32, device="cuda")
            out["cem_maps"] = torch.full((nc, P), -7.0, device="cuda")
        frame = hsi.make_frame(cube, H, W, B, 1, map_stride=P, **kw, **out)
        status = torch.zeros(1, dtype=torch.int32, device="cuda")
        if tensor_cores:
            hsi.score_frames_batch([frame], status=status)
        else:
            hsi.score_frames_device(hsi.frame_table([frame]), 1, max_bands=B, max_sam=ns, max_cem=nc, dtype=1,
                                    status=status)
        torch.cuda.synchronize()
        assert int(status.item()) == 0
        r = {k: v.cpu().numpy() for k, v in out.items()}
        if ns:
            _check_sam(orc, host, lib[:ns], r["sam_best"], r["sam_best_target"], r["sam_maps"])
        if nc:
            _check_cem(orc, host, cem, r)


def test_batch_entry_mixes_element_types(hsi, orc):
    """One hsi_score_frames_batch call with FP32 and FP16 frames of several band
    counts (FP16 above 128 bands falls back to the FP32-FMA scorer)."""
    specs = [(113, 0), (113, 1), (224, 1), (16, 1), (60, 0)]
    frames, keep = [], []
    for i, (B, dt) in enumerate(specs):
        H, W = 50, 70 + 3 * i
        sc = hsi.scene(B, n_targets=4, target_frac=0.02, frame_seed=900 + i, library_seed=70 + i)
        cube, _ = hsi.generate(sc, H, W, dtype=dt)
        lib = hsi.scene_targets(sc)
        P = H * W
        best = torch.full((P,), -7.0, device="cuda")
        bt = torch.full((P,), -7, dtype=torch.int32, device="cuda")
        maps = torch.full((4, P), -7.0, device="cuda")
        # descriptors hold raw pointers: every tensor they name stays referenced until the scorer is done
        d_lib = torch.from_numpy(lib).cuda()
        d_norms = torch.from_numpy(hsi.target_norms(lib)).cuda()
        frames.append(hsi.make_frame(cube, H, W, B, dt, sam_targets=d_lib, sam_norms=d_norms, sam_maps=maps,
                                     sam_best=best, sam_best_target=bt, map_stride=P))
        keep.append((cube, lib, best, bt, maps, H, W, B, d_lib, d_norms))
    hsi.score_frames_batch(frames)
    torch.cuda.synchronize()
    for cube, lib, best, bt, maps, H, W, B, _, _ in keep:
        host = _download(cube, B, H * W)
        _check_sam(orc, host, lib, best.cpu().numpy(), bt.cpu().numpy(), maps.cpu().numpy())


def test_batched_frames_inline_and_device_table(hsi, orc):
    shapes = [(30, 41, 113), (64, 32, 16), (17, 19, 224)]
    frames, keep = [], []
    for i, (H, W, B) in enumerate(shapes):
        sc = hsi.scene(B, n_targets=3 + i, target_frac=0.02, frame_seed=77 + i, library_seed=5 + i)
        cube, _ = hsi.generate(sc, H, W)
        targets = hsi.scene_targets(sc)
        P = H * W
        tg = torch.from_numpy(targets).cuda()
        nr = torch.from_numpy(hsi.target_norms(targets)).cuda()
        best = torch.zeros(P, device="cuda")
        bt = torch.zeros(P, dtype=torch.int32, device="cuda")
        maps = torch.zeros((targets.shape[0], P), device="cuda")
        frames.append(hsi.make_frame(cube, H, W, B, 0, sam_targets=tg, sam_norms=nr, sam_maps=maps,
                                     sam_best=best, sam_best_target=bt, map_stride=P))
        keep.append((cube, targets, tg, nr, best, bt, maps, H, W, B))
    hsi.score_frames(frames)
    torch.cuda.synchronize()
    for cube, targets, _, _, best, bt, maps, H, W, B in keep:
        host = _download(cube, B, H * W)
        _check_sam(orc, host, targets, best.cpu().numpy(), bt.cpu().numpy(), maps.cpu().numpy())
        best.zero_()
        bt.zero_()
        maps.zero_()
    table = hsi.frame_table(frames)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    hsi.score_frames_device(table, len(frames), max_bands=224, max_sam=5, max_cem=0, status=status)
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    for cube, targets, _, _, best, bt, maps, H, W, B in keep:
        host = _download(cube, B, H * W)
        _check_sam(orc, host, targets, best.cpu().numpy(), bt.cpu().numpy(), maps.cpu().numpy())


@pytest.mark.parametrize("ks,kc", [(8, 8), (16, 0), (0, 16), (13, 0), (5, 7)])
@pytest.mark.parametrize("shapes,B", [([(300, 300)], 113), ([(300, 300)], 1), ([(521, 695)], 8), ([(521, 695)], 9),
                                      ([(1, 132609)], 224), ([(300, 301), (7, 5), (299, 300)], 31)])
def test_wide_form_equals_narrow_form(hsi, shapes, B, ks, kc):
    """Sixteen filter slots over tiles of 896 pixels (host descriptors) and of 512 (a
    device table) run the same sums in the same order: every output bit is equal, at
    remainders of the stages' 8 bands and of the tiles, with maps on and off 16 bytes."""
    gen = torch.Generator(device="cuda").manual_seed(7 * B + 100 * ks + kc)
    out = []
    frames = ([], [])
    for n, (H, W) in enumerate(shapes):
        P = H * W
        stride = (P + 7) // 8 * 8
        cube = torch.rand((B, stride), generator=gen, device="cuda")
        sam = torch.rand((max(ks, 1), B), generator=gen, device="cuda")
        cem = torch.randn((max(kc, 1), B), generator=gen, device="cuda")
        norms = sam.double().square().sum(1).sqrt().float()
        for form in (0, 1):
            r = dict(sm=torch.full((max(ks, 1), P + n), -7.0, device="cuda"), sb=torch.full((P,), -7.0, device="cuda"),
                     st=torch.full((P,), -7, dtype=torch.int32, device="cuda"),
                     cm=torch.full((max(kc, 1), P + n), -7.0, device="cuda"), cb=torch.full((P,), -7.0, device="cuda"),
                     ct=torch.full((P,), -7, dtype=torch.int32, device="cuda"))
            frames[form].append(hsi.make_frame(
                cube, H, W, B, sam_targets=sam if ks else None, sam_norms=norms if ks else None,
                cem_weights=cem if kc else None, sam_maps=r["sm"] if ks else None, sam_best=r["sb"] if ks else None,
                sam_best_target=r["st"] if ks else None, cem_maps=r["cm"] if kc else None,
                cem_best=r["cb"] if kc else None, cem_best_target=r["ct"] if kc else None, map_stride=P + n))
            out.append((n, form, r, cube, sam, cem, norms))
    hsi.score_frames(frames[0])
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    hsi.score_frames_device(hsi.frame_table(frames[1]), len(shapes), max_bands=B, max_sam=ks, max_cem=kc, status=status)
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    for a, b in zip(out[::2], out[1::2]):
        for key in a[2]:
            assert torch.equal(a[2][key], b[2][key]), key


def _scorer_forms(fn):
    """Whether each scorer kernel that a captured call launches is the wide form
    (score_kernel's last template argument)."""
    from cuda.bindings import driver, runtime
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    fn(stream)  # one-time set-up
    stream.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph, stream=stream):
        fn(stream)
    g = runtime.cudaGraph_t(graph.raw_cuda_graph())
    _, _, n = runtime.cudaGraphGetNodes(g)
    err, nodes, n = runtime.cudaGraphGetNodes(g, n)
    assert err == runtime.cudaError_t.cudaSuccess
    forms = []
    for node in nodes[:n]:
        if runtime.cudaGraphNodeGetType(node)[1] != runtime.cudaGraphNodeType.cudaGraphNodeTypeKernel:
            continue
        err, params = driver.cuGraphKernelNodeGetParams(driver.CUgraphNode(int(node)))
        assert err == driver.CUresult.CUDA_SUCCESS
        if int(params.func):
            err, name = driver.cuFuncGetName(params.func)
        else:
            err, name = driver.cuKernelGetName(params.kern)
        assert err == driver.CUresult.CUDA_SUCCESS
        m = re.search(r"score_kernelI.*Lb([01])EE", name.decode())
        if m:
            forms.append(m.group(1) == "1")
    return forms


def _sixteen_filters(hsi, pixels, B, gen):
    """Frames of one row each, eight SAM targets and eight CEM filters."""
    frames, keep = [], []
    for P in pixels:
        cube = torch.rand((B, (P + 31) // 32 * 32), generator=gen, device="cuda")
        sam = torch.rand((8, B), generator=gen, device="cuda")
        cem = torch.randn((8, B), generator=gen, device="cuda")
        norms = sam.double().square().sum(1).sqrt().float()
        best, which = torch.empty((2, P), device="cuda"), torch.empty((2, P), dtype=torch.int32, device="cuda")
        frames.append(hsi.make_frame(cube, 1, P, B, sam_targets=sam, sam_norms=norms, cem_weights=cem,
                                     sam_best=best[0], sam_best_target=which[0], cem_best=best[1],
                                     cem_best_target=which[1], map_stride=P))
        keep.append((cube, sam, cem, norms, best, which))
    return frames, keep


@pytest.mark.parametrize("tiles, wide", [(0.3, False), (0.99, False), (1.8, True), (1.99, True), (2.02, False),
                                         (2.7, True), (2.8, False), (2.99, False), (3.9, True), (4.83, False), (7.9, True),
                                         (9.0, True), (20.5, True)])
def test_wide_form_where_its_tiles_fill_the_gpu(hsi, tiles, wide):
    """The scorer's form at so many 896-pixel tiles per SM, in one frame and in four."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    gen = torch.Generator(device="cuda").manual_seed(1)
    n = int(tiles * sms)
    for pixels in ([n * 896 - 3], [n // 4 * 896, n // 4 * 896, n // 4 * 896, (n - 3 * (n // 4)) * 896]):
        frames, keep = _sixteen_filters(hsi, pixels, 4, gen)
        assert _scorer_forms(lambda s: hsi.score_frames(frames, stream=s)) == [wide], pixels
    table = hsi.frame_table(frames)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    assert _scorer_forms(lambda s: hsi.score_frames_device(table, 4, max_bands=4, max_sam=8, max_cem=8, status=status,
                                                           stream=s)) == [False]


@pytest.mark.parametrize("specs", [
    # (height, width, bands, SAM targets, CEM filters) of each frame
    [(300, 301, 31, 8, 8), (7, 5, 113, 1, 8), (299, 399, 31, 8, 3), (1, 896, 8, 0, 5), (1, 897, 9, 8, 0), (60, 300, 113, 7, 7)],
    [(1, 260 * 896 + 1, 224, 8, 8)],
    [(257, 700, 224, 8, 8), (120, 400, 7, 8, 8)],
    [(300, 400, 17, 16, 0), (300, 400, 33, 12, 0), (31, 33, 64, 1, 0)],
    [(300, 400, 17, 0, 16), (300, 400, 33, 0, 9), (31, 33, 64, 0, 1)],
])
def test_wide_form_equals_narrow_form_over_frames(hsi, specs):
    """As above where the launch does take the wide form (checked), over frames of different
    sizes, bands and banks: the bank and the tile ring are carried from frame to frame."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert sms == 148, "the sizes put 1.1 to 2 tiles on each of 148 SMs"
    gen = torch.Generator(device="cuda").manual_seed(sum(b for _, _, b, _, _ in specs))
    frames, out, keep = ([], []), ([], []), []
    for n, (H, W, B, ks, kc) in enumerate(specs):
        P = H * W
        cube = torch.rand((B, (P + 7) // 8 * 8), generator=gen, device="cuda")
        sam = torch.rand((max(ks, 1), B), generator=gen, device="cuda")
        cem = torch.randn((max(kc, 1), B), generator=gen, device="cuda")
        norms = sam.double().square().sum(1).sqrt().float()
        keep.append((cube, sam, cem, norms))
        for form in (0, 1):
            maps = torch.full((ks + kc, P + n), -7.0, device="cuda")
            best = torch.full((2, P), -7.0, device="cuda")
            which = torch.full((2, P), -7, dtype=torch.int32, device="cuda")
            frames[form].append(hsi.make_frame(
                cube, H, W, B, map_stride=P + n,
                **(dict(sam_targets=sam, sam_norms=norms, sam_maps=maps, sam_best=best[0], sam_best_target=which[0])
                   if ks else {}),
                **(dict(cem_weights=cem, cem_maps=maps[ks:], cem_best=best[1], cem_best_target=which[1]) if kc else {})))
            out[form].extend([maps, best, which])
    assert _scorer_forms(lambda s: hsi.score_frames_batch(frames[0], stream=s)) == [True]
    hsi.score_frames_batch(frames[0])
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    hsi.score_frames_device(hsi.frame_table(frames[1]), len(specs), max_bands=max(s[2] for s in specs),
                            max_sam=max(s[3] for s in specs), max_cem=max(s[4] for s in specs), status=status)
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    for a, b in zip(*out):
        assert torch.equal(a, b)


def test_device_table_rejects_frames_outside_bounds(hsi):
    """A frame with more bands than the launch allows is skipped, not overrun."""
    H, W, B = 8, 8, 64
    sc = hsi.scene(B, n_targets=2)
    cube, _ = hsi.generate(sc, H, W)
    t = torch.from_numpy(hsi.scene_targets(sc)).cuda()
    nr = torch.from_numpy(hsi.target_norms(hsi.scene_targets(sc))).cuda()
    best = torch.full((H * W,), -7.0, device="cuda")
    f = hsi.make_frame(cube, H, W, B, 0, sam_targets=t, sam_norms=nr, sam_best=best)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    hsi.score_frames_device(hsi.frame_table([f]), 1, max_bands=32, max_sam=2, max_cem=0, status=status)
    torch.cuda.synchronize()
    assert int(status.item()) == hsi.E_INVALID
    assert (best == -7.0).all()


def test_invalid_arguments_are_rejected(hsi):
    cube = torch.zeros((4, 32), device="cuda")
    t = np.ones((1, 4), np.float32)
    tg = torch.from_numpy(t).cuda()
    nr = torch.ones(1, device="cuda")
    best = torch.zeros(16, device="cuda")
    f = hsi.make_frame(cube, 4, 4, 4, 0, stride=30, sam_targets=tg, sam_norms=nr, sam_best=best)
    with pytest.raises(hsi.HsiError) as e:
        hsi.score_frames([f])
    assert e.value.status == hsi.E_INVALID
    f = hsi.make_frame(cube, 4, 4, 300, 0, sam_targets=tg, sam_norms=nr, sam_best=best)
    with pytest.raises(hsi.HsiError):
        hsi.score_frames([f])
