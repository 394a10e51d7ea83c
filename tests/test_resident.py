"""The resident step (csrc/resident.cu): segments of small float32 grids whose
blocks keep the fields on the chip, against the float64 flat step on the same
state, tracks and steps.

Tolerance: a float32 step rounds each value about ten times against weights
that sum to one in absolute value 1.4 at most, so it is off by up to
10 * 6e-8 * 1.4 < 1e-6 of the peak a step, and the steps' errors add at worst:
1e-6 * steps, fields and tallies alike (every tally sums values of one sign)."""

import ctypes
import importlib

import numpy as np
import pytest

from goldens import make_config, pkg

# no_xy, no_z, voxels of the chamber's grid: one block and many, ragged tiles
# and k splits, a patch of every shape, the smallest and the largest that run
# resident, k rows with one and with eight padded elements
SIZES = [(3, 1), (4, 3), (5, 20), (8, 50), (11, 50), (12, 200), (13, 43), (24, 200), (25, 149), (31, 100), (48, 200),
         (53, 200), (48, 400), (59, 400), (70, 203), (76, 200)]


def _grid(native, n, no_z, wall, dtype, variant):
    g = native.PicGrid()
    g.no_xy, g.no_z, g.nze = n, no_z, 2
    g.nzb = no_z + 4
    g.kpitch = (g.nzb + 7) // 8 * 8
    g.mid_xy = n / 2
    g.scoring_radius_sq = max(1.0, (n / 2 - 3) ** 2)
    g.p_lat, g.p_zm, g.p_zp = 0.02, 0.52, -0.06
    g.n_lat, g.n_zm, g.n_zp = 0.03, 0.70, -0.05
    g.p_cen = 1 - 4 * g.p_lat - g.p_zm - g.p_zp
    g.n_cen = 1 - 4 * g.n_lat - g.n_zm - g.n_zp
    g.alpha_dt = 2e-4
    g.gaussian_factor, g.h2_over_b2, g.cutoff_voxels = 3.0, 0.11, 6.5
    g.wall, g.dtype, g.variant = wall, dtype, variant
    return g


def _segment(native, g, torch, state, xs, ys, off, parity, graph=False, workspace="pic_segment_workspace_bytes"):
    lib = native.load()
    t = torch.float64 if g.dtype == native.PIC_F64 else torch.float32
    n, kp, steps = g.no_xy, g.kpitch, len(off) - 1
    f = [torch.zeros((n, n, kp), dtype=t, device="cuda") for _ in range(4)]
    for q in range(2):
        f[2 * parity + q][:, :, : g.nzb] = torch.from_numpy(state[q]).to("cuda", t)
    dens = [torch.zeros((n, 2 * ((n + 3) // 4 * 4)), dtype=t, device="cuda") for _ in range(2)]
    counts = torch.zeros((n, n), dtype=torch.int32, device="cuda")
    tally = torch.zeros((steps, 4), dtype=torch.float64, device="cuda")
    b = ctypes.c_int64()
    native.check(getattr(lib, workspace)(ctypes.byref(g), ctypes.byref(b)), workspace)
    ws = torch.zeros(b.value, dtype=torch.uint8, device="cuda")
    x, y = torch.from_numpy(xs).cuda(), torch.from_numpy(ys).cuda()
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    args = (ctypes.byref(g), f[0].data_ptr(), f[1].data_ptr(), f[2].data_ptr(), f[3].data_ptr(), parity, steps,
            x.data_ptr(), y.data_ptr(), off.ctypes.data, dens[0].data_ptr(), dens[1].data_ptr(), parity,
            counts.data_ptr(), tally.data_ptr(), ws.data_ptr(), ws.numel(), st.cuda_stream)
    if graph:
        h = ctypes.c_void_p()
        native.check(lib.pic_graph_create(*args, ctypes.byref(h)), "pic_graph_create")
        native.check(lib.pic_graph_launch(h, st.cuda_stream), "pic_graph_launch")
    else:
        native.check(lib.pic_run_segment(*args), "pic_run_segment")
    status = ctypes.c_int32()
    native.check(lib.pic_workspace_status(ws.data_ptr(), 0, st.cuda_stream, ctypes.byref(status)), "status")
    if graph:
        native.check(lib.pic_graph_destroy(h), "pic_graph_destroy")
    assert status.value == 0
    out = (parity + steps) & 1
    return (f[2 * out][:, :, : g.nzb].double().cpu().numpy(), f[2 * out + 1][:, :, : g.nzb].double().cpu().numpy(),
            f[2 * out][:, :, g.nzb :].abs().sum().item() + f[2 * out + 1][:, :, g.nzb :].abs().sum().item(),
            tally.cpu().numpy(), counts.cpu().numpy(), [d.double().cpu().numpy() for d in dens])


def _case(n, no_z, steps, seed, most_tracks):
    rng = np.random.default_rng(seed)
    state = [np.zeros((n, n, no_z + 4)) for _ in range(2)]
    for s in state:  # every column its own, the ring's too
        s[:, :, 1:-1] = rng.uniform(0.5, 1.5, (n, n, no_z + 2))
    m = rng.integers(0, most_tracks + 1, steps) * (rng.random(steps) < 0.7)
    off = np.concatenate([[0], np.cumsum(m)]).astype(np.int64)
    return state, rng.uniform(0, n, off[-1] + 1), rng.uniform(0, n, off[-1] + 1), off


def _compare(native, got, ref, steps):
    tol = 1e-6 * steps
    for a, b in zip(got[:2], ref[:2]):
        assert np.abs(a - b).max() <= tol * np.abs(b).max()
    assert got[2] == 0.0
    for q in range(4):
        peak = np.abs(ref[3][:, q]).max()
        assert np.abs(got[3][:, q] - ref[3][:, q]).max() <= tol * peak + 1e-30
    assert np.array_equal(got[4], ref[4])
    for a, b in zip(got[5], ref[5]):  # the caller's pair buffers, as every segment leaves them
        assert np.abs(a - b).max() <= 1e-6 * max(1.0, np.abs(b).max())


@pytest.mark.gpu
@pytest.mark.parametrize("wall", [0, 1])
@pytest.mark.parametrize("n,no_z", SIZES)
def test_resident_segment_matches_the_float64_step(n, no_z, wall):
    import torch

    native = importlib.import_module(pkg().__name__ + "._native")
    steps = 9
    state, xs, ys, off = _case(n, no_z, steps, 100 * n + no_z + wall, 12)
    g = _grid(native, n, no_z, wall, native.PIC_F32, 0)
    resident = ctypes.c_int32()
    native.check(native.load().pic_segment_resident(ctypes.byref(g), ctypes.byref(resident)), "pic_segment_resident")
    assert resident.value == 1
    parity = n & 1
    before = native.load().pic_kernel_launches()
    got = _segment(native, g, torch, state, xs, ys, off, parity)
    assert native.load().pic_kernel_launches() - before <= 4  # binning, tiles, steps, tallies
    ref = _segment(native, _grid(native, n, no_z, wall, native.PIC_F64, 1), torch, state, xs, ys, off, parity)
    _compare(native, got, ref, steps)
    again = _segment(native, g, torch, state, xs, ys, off, parity, graph=True)
    for a, b in zip(got[:4], again[:4]):  # the same bits, from a replayed graph
        assert np.array_equal(a, b)


@pytest.mark.gpu
@pytest.mark.parametrize("n,no_z,steps,tracks", [(10, 50, 600, 3), (24, 100, 300, 20), (31, 60, 12, 30000)])
def test_resident_segments_of_several_launches(n, no_z, steps, tracks):
    """More steps than one launch takes, and more tracks than one deposition does."""
    import torch

    native = importlib.import_module(pkg().__name__ + "._native")
    state, xs, ys, off = _case(n, no_z, steps, n, tracks)
    for wall in (0, 1):
        g = _grid(native, n, no_z, wall, native.PIC_F32, 0)
        g64 = _grid(native, n, no_z, wall, native.PIC_F64, 1)
        g.gaussian_factor = g64.gaussian_factor = 3.0 / tracks
        got = _segment(native, g, torch, state, xs, ys, off, 0)
        ref = _segment(native, g64, torch, state, xs, ys, off, 0)
        _compare(native, got, ref, steps)


def test_what_runs_resident():
    """The choice follows the descriptor alone: AUTO float32 grids that fit,
    nothing that asks for a kernel or has truncation boxes beyond 64 cells."""
    native = importlib.import_module(pkg().__name__ + "._native")
    lib = native.load()

    def resident(**kw):
        g = _grid(native, kw.pop("n", 24), kw.pop("no_z", 200), 0, kw.pop("dtype", native.PIC_F32), kw.pop("variant", 0))
        for k, v in kw.items():
            setattr(g, k, v)
        out, seg, step = ctypes.c_int32(), ctypes.c_int64(), ctypes.c_int64()
        native.check(lib.pic_segment_resident(ctypes.byref(g), ctypes.byref(out)), "pic_segment_resident")
        native.check(lib.pic_segment_workspace_bytes(ctypes.byref(g), ctypes.byref(seg)), "pic_segment_workspace_bytes")
        native.check(lib.pic_step_workspace_bytes(ctypes.byref(g), ctypes.byref(step)), "pic_step_workspace_bytes")
        assert seg.value >= step.value
        return bool(out.value)

    assert resident()
    assert resident(deposit_variant=native.PIC_DEPOSIT_BINNED)
    assert not resident(deposit_variant=native.PIC_DEPOSIT_TRACKS)
    assert not resident(variant=1) and not resident(steps_per_launch=32) and not resident(dtype=native.PIC_F64)
    assert not resident(cutoff_voxels=31.5)
    assert not resident(n=208, no_z=400) and not resident(n=1068, no_z=400)
    engine = importlib.import_module(pkg().__name__ + ".engine")
    assert engine.runs_resident(engine.make_grid(make_config("column_10um_r008")))
    assert not engine.runs_resident(engine.make_grid(make_config("column_10um_r02", track_cutoff_sigmas=None)))


@pytest.mark.gpu
@pytest.mark.parametrize("wall", [0, 1])
@pytest.mark.parametrize("n,no_z", [(3, 1), (4, 30), (5, 20), (8, 50), (12, 200), (13, 43), (24, 200), (25, 149), (31, 100),
                                    (48, 200), (53, 200), (48, 400)])
def test_resident_reverse_sweep_matches_the_float64_one(n, no_z, wall):
    """lambda over the whole grid, ring and corners included, and the five
    derivative sums, through segments of even, odd and short lengths.

    Tolerance: lambda as the fields above; a derivative sum adds products mu Du
    (the last one p n of the scored voxels and mu p n) whose factors are each
    off by that much of their peaks, so it is off by 2e-6 * steps of the sum of
    their magnitudes at worst."""
    import torch

    native = importlib.import_module(pkg().__name__ + "._native")
    lib = native.load()
    steps, every = 17, 6 if n % 2 else 5
    rng = np.random.default_rng(7 * n + no_z + wall)
    kp = (no_z + 4 + 7) // 8 * 8
    n_seg = -(-steps // every)
    m = rng.integers(0, 2, steps)
    m[0] = 1
    off = np.concatenate([[0], np.cumsum(m)]).astype(np.int64)
    dp = (n + 3) // 4 * 4
    ckpt = np.zeros((2, n_seg, n, n, kp))
    ckpt[..., 1 : no_z + 3] = rng.uniform(0.5, 1.5, (2, n_seg, n, n, no_z + 2))
    keep = rng.uniform(0.0, 0.1, (int(m.sum()), n, dp, 2))

    def sweep(dtype, variant):
        g = _grid(native, n, no_z, wall, dtype, variant)
        t = torch.float64 if dtype == native.PIC_F64 else torch.float32
        dev = lambda a: torch.from_numpy(a).to("cuda", t)  # noqa: E731
        c, d = dev(ckpt), dev(keep)
        states = torch.zeros((2, every, n, n, kp), dtype=t, device="cuda")
        lam = torch.zeros((2, 2, n, n, kp), dtype=t, device="cuda")
        grad = torch.zeros(5, dtype=torch.float64, device="cuda")
        need = {}
        for name in ("pic_segment_workspace_bytes", "pic_adjoint_workspace_bytes"):
            b = ctypes.c_int64()
            native.check(getattr(lib, name)(ctypes.byref(g), ctypes.byref(b)), name)
            need[name] = torch.zeros(b.value, dtype=torch.uint8, device="cuda")
        ws, aws = need.values()
        st = torch.cuda.current_stream().cuda_stream
        before = lib.pic_kernel_launches()
        native.check(lib.pic_adjoint_backward(
            ctypes.byref(g), c[0].data_ptr(), c[1].data_ptr(), n * n * kp, steps, every, off.ctypes.data, d.data_ptr(),
            states[0].data_ptr(), states[1].data_ptr(), lam[0, 0].data_ptr(), lam[0, 1].data_ptr(), lam[1, 0].data_ptr(),
            lam[1, 1].data_ptr(), grad.data_ptr(), ws.data_ptr(), ws.numel(), aws.data_ptr(), aws.numel(), st),
            "pic_adjoint_backward")
        torch.cuda.synchronize()
        return lam[steps & 1].double().cpu().numpy(), grad.cpu().numpy(), lib.pic_kernel_launches() - before

    lam, grad, launches = sweep(native.PIC_F32, 0)
    ref, want, _ = sweep(native.PIC_F64, 1)
    # two a segment (a short last one step by step) and the final sum; lambda of
    # the largest does not fit the chip: its adjoint steps are launched one by one
    assert launches <= 2 * n_seg + 1 + 4 * every + (2 * steps if n * n * no_z > 800000 else 0)
    tol = 1e-6 * steps
    for a, b in zip(lam, ref):
        assert np.abs(a - b).max() <= tol * np.abs(b).max()
    voxels = steps * (n - 2) ** 2 * (no_z + 2)
    magnitude = np.array([np.abs(ref).mean() * 2.0] * 4 + [1.0 + np.abs(ref).mean() * 2.0]) * voxels
    assert (np.abs(grad - want) <= 2 * tol * magnitude).all()


@pytest.mark.gpu
@pytest.mark.parametrize("n,no_z,tracks,steps,flat", [(24, 100, 600, 4, False), (24, 100, 2000, 4, True), (24, 100, 2000, 16, False),
                                                      (18, 50, 20000, 12, True), (31, 60, 60000, 5, True)])
def test_dense_segments_step_flat(n, no_z, tracks, steps, flat):
    """Steps of so many tracks that one block's sum of them would outlast the
    per-track deposition of all (resident_steps_eligible): launched one by one."""
    import torch

    native = importlib.import_module(pkg().__name__ + "._native")
    rng = np.random.default_rng(n + tracks)
    state = _case(n, no_z, steps, n, 1)[0]
    off = np.arange(steps + 1, dtype=np.int64) * tracks
    off[2:] -= tracks  # the second step has none
    xs, ys = rng.uniform(0, n, (2, off[-1]))
    g = _grid(native, n, no_z, 0, native.PIC_F32, 0)
    g64 = _grid(native, n, no_z, 0, native.PIC_F64, 1)
    g.gaussian_factor = g64.gaussian_factor = 3.0 / tracks
    before = native.load().pic_kernel_launches()
    got = _segment(native, g, torch, state, xs, ys, off, 0)
    launches = native.load().pic_kernel_launches() - before
    assert launches == (2 * steps - 1 if flat else 4)  # a deposition and a step each; binning, tiles, steps, tallies
    ref = _segment(native, g64, torch, state, xs, ys, off, 0)
    # a cell's float32 sum of `tracks` terms of one sign, rounded at each: at
    # worst half an ulp of the sum a term, and of that a random walk's share,
    # sqrt(tracks) 3e-8 of the deposition's peak (1.5 at most) with four deviations
    tol = 1e-6 * steps + 1.5 * 4 * tracks**0.5 * 3e-8 * steps
    for a, b in zip(got[:2], ref[:2]):
        assert np.abs(a - b).max() <= tol * np.abs(b).max()
    for q in range(4):
        assert np.abs(got[3][:, q] - ref[3][:, q]).max() <= tol * np.abs(ref[3][:, q]).max() + 1e-30
    assert np.array_equal(got[4], ref[4])


@pytest.mark.gpu
@pytest.mark.parametrize("name,tuned", [("column_10um_r008", 0), ("column_5um_r05_d8p91", 1)])
def test_tuning_leaves_resident_grids_to_the_library(monkeypatch, name, tuned):
    """The autotuner names a variant, and a grid with one named does not run resident."""
    autotune = importlib.import_module(pkg().__name__ + ".autotune")
    calls = []
    monkeypatch.setattr(autotune, "tune", lambda *a, **kw: calls.append(a))
    pkg().run_simulation_b200(make_config(name), progress=False, return_fields=False, max_steps=8, tune=True)
    assert len(calls) == tuned


@pytest.mark.gpu
def test_gradient_within_the_memory_a_step_workspace_leaves():
    """A memory_limit that holds the fields, the step workspace, lambda and the
    segment schedule is enough: the resident steps' workspace is given back then."""
    import torch

    adj = importlib.import_module(pkg().__name__ + ".adjoint")
    native = importlib.import_module(pkg().__name__ + "._native")
    cfg = make_config("column_10um_r008")
    free = adj.AdjointRun(cfg, max_steps=200)
    ks = free.forward()
    grad = free.backward()
    eng, step = free._eng, ctypes.c_int64()
    native.check(native.load().pic_step_workspace_bytes(ctypes.byref(eng.grid), ctypes.byref(step)), "bytes")
    assert eng.workspace.numel() > step.value
    rest = (*eng.pos, *eng.neg, *eng.dens, eng.counts, eng.tally, eng.xs, eng.ys)
    held = sum(t.numel() * t.element_size() for t in rest) + step.value
    own = sum(t.numel() * t.element_size() for t in (free.ckpt, free.dens_keep))
    states = 2 * (free.K + 2) * free.field * 4  # the segment's states and lambda
    free.release()
    for schedule in ("segments", "auto"):
        run = adj.AdjointRun(cfg, max_steps=200, memory_limit=held + own + states, schedule=schedule)
        assert abs(run.forward() - ks) <= 1e-6 * ks and run.kind == "segments"
        np.testing.assert_allclose(run.backward(), grad, rtol=1e-4)
        run.release()
    with pytest.raises(MemoryError):
        adj.AdjointRun(cfg, max_steps=200, memory_limit=held + own + states - 4, schedule="segments").forward()
    torch.cuda.synchronize()


@pytest.mark.gpu
@pytest.mark.parametrize("variant", [0, 1])
@pytest.mark.parametrize("n,no_z", [(5, 20), (24, 200), (48, 200), (53, 200), (59, 400), (76, 200)])
def test_tallies_lose_no_bits(n, no_z, variant):
    """Beyond the four k of an item the tallies are summed in double-floats: of
    integers below 2^22, of which four add up exactly in float32, they are exact.
    A step of weight one keeps P = 2 m and halves it where it meets N = 1/2."""
    import torch

    native = importlib.import_module(pkg().__name__ + "._native")
    g = _grid(native, n, no_z, 0, native.PIC_F32, variant)
    g.p_lat = g.p_zm = g.p_zp = g.n_lat = g.n_zm = g.n_zp = 0.0
    g.p_cen = g.n_cen = g.alpha_dt = 1.0
    m = np.random.default_rng(n).integers(0, 1 << 21, (n, n, no_z + 4)).astype(np.float64)
    m[:, :, 0] = m[:, :, -1] = 0
    half = np.zeros_like(m)
    half[:, :, 1:-1] = 0.5
    tally = _segment(native, g, torch, [2 * m, half], np.zeros(1), np.zeros(1), np.zeros(5, dtype=np.int64), 0)[3][0]
    i = np.arange(1, n - 1)
    scored = (i[:, None] - g.mid_xy) ** 2 + (i[None, :] - g.mid_xy) ** 2 < g.scoring_radius_sq
    inside = m[1:-1, 1:-1, g.nze : g.nze + no_z][scored]
    assert inside.size and inside.sum() < 2**44
    assert np.array_equal(tally, [0.0, inside.sum(), inside.sum(), (0.5 - inside).sum()])


@pytest.mark.gpu
@pytest.mark.parametrize("variant", [0, 1])
@pytest.mark.parametrize("n,no_z", [(5, 20), (24, 200), (31, 100), (48, 200), (53, 200)])
def test_derivative_sums_lose_no_bits(n, no_z, variant):
    """The same of the reverse sweep: with weights of one and no recombination
    lambda stays what it is, and dR/da adds (1 - lambda+ - lambda-) p n over p = n =
    1: integers of which four add up exactly in float32, the rest in double-floats."""
    import torch

    native = importlib.import_module(pkg().__name__ + "._native")
    lib = native.load()
    steps = every = 8
    kp = (no_z + 4 + 7) // 8 * 8
    g = _grid(native, n, no_z, 0, native.PIC_F32, 0)
    g.adjoint_variant = variant
    g.p_lat = g.p_zm = g.p_zp = g.n_lat = g.n_zm = g.n_zp = g.alpha_dt = 0.0
    g.p_cen = g.n_cen = 1.0
    lam = np.zeros((2, 2, n, n, kp))
    lam[0, :, 1:-1, 1:-1, 1 : no_z + 3] = np.random.default_rng(n).integers(0, 1 << 21, (2, n - 2, n - 2, no_z + 2))
    one = np.zeros((2, 1, n, n, kp))
    one[..., 1 : no_z + 3] = 1.0
    dev = lambda a: torch.from_numpy(a).to("cuda", torch.float32)  # noqa: E731
    ckpt, L = dev(one), dev(lam)
    states = torch.zeros((2, every, n, n, kp), device="cuda")
    grad = torch.zeros(5, dtype=torch.float64, device="cuda")
    ws = []
    for name in ("pic_segment_workspace_bytes", "pic_adjoint_workspace_bytes"):
        b = ctypes.c_int64()
        native.check(getattr(lib, name)(ctypes.byref(g), ctypes.byref(b)), name)
        ws.append(torch.zeros(b.value, dtype=torch.uint8, device="cuda"))
    off = np.zeros(steps + 1, dtype=np.int64)
    before = lib.pic_kernel_launches()
    native.check(lib.pic_adjoint_backward(
        ctypes.byref(g), ckpt[0].data_ptr(), ckpt[1].data_ptr(), n * n * kp, steps, every, off.ctypes.data, None,
        states[0].data_ptr(), states[1].data_ptr(), L[0, 0].data_ptr(), L[0, 1].data_ptr(), L[1, 0].data_ptr(),
        L[1, 1].data_ptr(), grad.data_ptr(), ws[0].data_ptr(), ws[0].numel(), ws[1].data_ptr(), ws[1].numel(),
        torch.cuda.current_stream().cuda_stream), "pic_adjoint_backward")
    assert lib.pic_kernel_launches() - before == (steps if variant else 1) + 2  # and the states, the final sum
    i = np.arange(1, n - 1)
    scored = (i[:, None] - g.mid_xy) ** 2 + (i[None, :] - g.mid_xy) ** 2 < g.scoring_radius_sq
    want = steps * (scored.sum() * no_z - lam[0].sum())
    assert abs(want) < 2**44 and grad[4].item() == want
    assert np.array_equal(L[steps & 1].cpu().numpy(), lam[0])


@pytest.mark.gpu
@pytest.mark.parametrize("n,no_z,adjoint", [(24, 200, 7), (48, 200, 7), (76, 200, -1)])
def test_packets_that_never_come_end_the_launch_with_a_status(n, no_z, adjoint):
    """The resident kernels' bounded wait, with patches of one, two and six
    columns: every block leaves, the status says why, the derivative sums are NaN,
    and the context runs on."""
    import torch

    native = importlib.import_module(pkg().__name__ + "._native")
    lib = native.load()
    g = _grid(native, n, no_z, 0, native.PIC_F32, 0)
    out = [ctypes.c_int32(-5) for _ in range(3)]
    native.check(lib.pic_selftest_packets(ctypes.byref(g), *(ctypes.byref(o) for o in out),
                                          torch.cuda.current_stream().cuda_stream), "pic_selftest_packets")
    assert [o.value for o in out] == [7, adjoint, 1 if adjoint == 7 else 0]
    state, xs, ys, off = _case(n, no_z, 9, n, 12)
    got = _segment(native, g, torch, state, xs, ys, off, 0)
    ref = _segment(native, _grid(native, n, no_z, 0, native.PIC_F64, 1), torch, state, xs, ys, off, 0)
    _compare(native, got, ref, 9)


def test_the_packet_selftest_needs_blocks_that_trade():
    native = importlib.import_module(pkg().__name__ + "._native")
    out = [ctypes.c_int32() for _ in range(3)]
    for n, no_z in ((3, 1), (208, 400)):  # one block; not resident
        g = _grid(native, n, no_z, 0, native.PIC_F32, 0)
        assert native.load().pic_selftest_packets(ctypes.byref(g), *(ctypes.byref(o) for o in out), None) != native.PIC_OK
