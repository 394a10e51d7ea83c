"""The float32 flat step over eight-wide items (csrc/pic_wide.cuh) and the
tallies a segment's steps sum for one another, against the float64 step.

Tolerance as for the resident step: 1e-6 of the peak a step, steps added up."""

import importlib
import warnings
from types import SimpleNamespace

import numpy as np
import pytest

from goldens import pkg
from test_resident import _case, _compare, _grid, _segment

# no_xy, no_z (four layers more in all): one interior column; a column of one
# vector, of exactly a warp, of a warp and one vector, of many; rows with one to
# eight padded layers; a grid of one block and of every block
SIZES = [(3, 1), (3, 600), (4, 3), (5, 20), (9, 252), (9, 255), (10, 260), (33, 57), (40, 28), (57, 203), (90, 124),
         (130, 300)]


@pytest.mark.gpu
@pytest.mark.parametrize("wall", [0, 1])
@pytest.mark.parametrize("n,no_z", SIZES)
def test_flat_segment_matches_the_float64_step(n, no_z, wall):
    import torch

    native = importlib.import_module(pkg().__name__ + "._native")
    for steps in (1, 2, 9):  # a step alone, a step and its last, both partial buffers in turn
        state, xs, ys, off = _case(n, no_z, steps, 100 * n + no_z + wall, 12)
        g = _grid(native, n, no_z, wall, native.PIC_F32, native.PIC_VARIANT_FLAT)
        g64 = _grid(native, n, no_z, wall, native.PIC_F64, native.PIC_VARIANT_FLAT)
        for variant in (native.PIC_DEPOSIT_AUTO, native.PIC_DEPOSIT_TRACKS):  # pairs kept and pairs cleared
            g.deposit_variant = g64.deposit_variant = variant
            got = _segment(native, g, torch, state, xs, ys, off, n & 1)
            ref = _segment(native, g64, torch, state, xs, ys, off, n & 1)
            _compare(native, got, ref, steps)


def _thick_batch():
    kw = dict(grid_size_um=10.0, E_MeV_u=56.2, dose_rate_Gy_s=20.0, pulse_duration_s=4e-7, repetition_rate_hz=50.0)
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        return [pkg().SimulationConfig(voltage_V=v, electrode_gap_cm=gap, sampled_radius_cm=r, seed=s, **kw)
                for v, gap, r, s in ((4000.0, 1.2, 0.002, 1), (3000.0, 0.2, 0.006, 2), (3500.0, 0.1, 0.012, 3))]


@pytest.mark.gpu
def test_batched_steps_do_not_depend_on_the_blocks(monkeypatch):
    """Grids with fewer threads than vectors in a column (one block for 1206
    layers), and with one block or many: the same fields, bit for bit, and the
    same tallies to the rounding of their double-float sums (44 bits)."""
    batched = importlib.import_module(pkg().__name__ + ".batched")
    run = lambda: pkg().run_batched_b200(_thick_batch(), solo_grids=0, return_fields=True)
    many = run()
    monkeypatch.setattr(batched, "_grid_blocks", lambda items, sms: np.ones(len(items), dtype=np.int64))
    for a, b in zip(many, run()):
        assert np.array_equal(a.positive_array, b.positive_array) and np.array_equal(a.negative_array, b.negative_array)
        assert np.abs(a.positive_array).max() > 0
        np.testing.assert_allclose(a.recombination, b.recombination, rtol=1e-11, atol=0)


@pytest.mark.parametrize("seed", range(6))
def test_grid_blocks_fill_whole_waves(seed):
    batched = importlib.import_module(pkg().__name__ + ".batched")
    rng = np.random.default_rng(seed)
    items = rng.integers(300, 3_000_000, int(rng.integers(1, 64)))
    nb = batched._grid_blocks(items, 152)
    want = -(-int(items.sum()) // batched.items_per_block(int(items.sum()), 152))
    assert nb.min() >= 1 and nb.sum() <= max(want, want + (nb == 1).sum() - 1)
    if (items * want // items.sum()).min() >= 1:
        assert nb.sum() == want
        assert (items / nb).max() <= 2 * items.sum() / want


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["PIC_F32", "PIC_F64"])
@pytest.mark.parametrize("n,no_z,steps", [(20, 3, 300), (200, 3, 90)])
def test_depositing_further_ahead_changes_nothing(n, no_z, steps, dtype):
    """Segments with more depositing steps than the slots of one launch pair (256
    for one tile, 38 for sixteen), against groups of eight: the same bits."""
    import torch

    native = importlib.import_module(pkg().__name__ + "._native")
    state, xs, ys, off = _case(n, no_z, steps, n, 40)
    g = _grid(native, n, no_z, 0, getattr(native, dtype), native.PIC_VARIANT_FLAT)
    runs = [_segment(native, g, torch, state, xs, ys, off, 0, workspace=w)
            for w in ("pic_segment_workspace_bytes", "pic_step_workspace_bytes")]
    for a, b in zip(runs[0][:5], runs[1][:5]):
        assert np.array_equal(a, b)
    for a, b in zip(runs[0][5], runs[1][5]):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("n,bins", [(31, 1), (32, 1), (33, 1), (64, 1), (97, 2), (130, 3), (1025, 31), (70001, 400)])
def test_arrivals_drawn_in_blocks_equal_numpys(n, bins):
    """The histogram of a pulse drawn in blocks (from 32 draws a bin on), and the
    generator's place after it, with bins that end before, at and past the pulse."""
    pulses = importlib.import_module(pkg().__name__ + ".pulses")
    for seed, end in ((1, 0.97), (2, 1.0), (3, 1.05)):
        edges = np.linspace(0.0, 5.4e-4 * end, bins + 1)
        cfg = SimpleNamespace(number_of_tracks_per_pulse=n, pulse_duration_s=5.4e-4, pulse_time_bins=edges)
        mine, theirs = np.random.default_rng(seed), np.random.default_rng(seed)
        got = pulses.pulse_arrival_counts(cfg, mine)
        arrival = np.cumsum(theirs.random(n))
        arrival /= arrival[-1]
        arrival *= cfg.pulse_duration_s
        assert np.array_equal(got, np.histogram(arrival, edges)[0])
        assert mine.random() == theirs.random()


@pytest.mark.gpu
@pytest.mark.parametrize("wall", [0, 1])
@pytest.mark.parametrize("n,no_z", SIZES)
def test_flat_adjoint_step_matches_the_float64_one(n, no_z, wall):
    """One reverse step against the float64 kernel (which reads the state's
    neighbours where this one sums by parts). lambda: ten roundings of values
    within 2 of the peak, 1e-6 of it; each derivative: 1e-6 of the sum of
    its terms' magnitudes (twelve weights of mu u at most, (1 + mu) p n)."""
    import ctypes

    import torch

    native = importlib.import_module(pkg().__name__ + "._native")
    lib = native.load()
    rng = np.random.default_rng(n + no_z)
    nzb = no_z + 4
    kp = (nzb + 7) // 8 * 8
    fields = np.zeros((4, n, n, kp))
    fields[:2, :, :, 1 : nzb - 1] = rng.uniform(0.5, 1.5, (2, n, n, nzb - 2))
    fields[2:, :, :, 1 : nzb - 1] = rng.uniform(-1.0, 1.0, (2, n, n, nzb - 2))
    pairs = rng.uniform(0.0, 1.0, (n, (n + 3) // 4 * 4, 2))

    def step(dtype, dep):
        t = torch.float64 if dtype == native.PIC_F64 else torch.float32
        g = _grid(native, n, no_z, wall, dtype, native.PIC_VARIANT_FLAT)
        g.adjoint_variant = native.PIC_VARIANT_FLAT
        f = torch.from_numpy(fields).to("cuda", t)
        out = torch.full((2, n, n, kp), 7.0, dtype=t, device="cuda")
        d = torch.from_numpy(pairs).to("cuda", t).contiguous()
        grad = torch.zeros(5, dtype=torch.float64, device="cuda")
        b = ctypes.c_int64()
        native.check(lib.pic_adjoint_workspace_bytes(ctypes.byref(g), ctypes.byref(b)), "bytes")
        ws = torch.zeros(b.value, dtype=torch.uint8, device="cuda")
        native.check(lib.pic_adjoint_step(ctypes.byref(g), f[0].data_ptr(), f[1].data_ptr(), d.data_ptr() if dep else None,
                                          f[2].data_ptr(), f[3].data_ptr(), out[0].data_ptr(), out[1].data_ptr(),
                                          grad.data_ptr(), ws.data_ptr(), ws.numel(),
                                          torch.cuda.current_stream().cuda_stream), "pic_adjoint_step")
        return out.double().cpu().numpy(), grad.cpu().numpy()

    for dep in (True, False):
        lam, grad = step(native.PIC_F32, dep)
        ref, rgrad = step(native.PIC_F64, dep)
        assert np.abs(lam - ref).max() <= 1e-6 * max(1.0, np.abs(ref).max())
        assert not lam[:, :, :, nzb - 1 :].any() and not lam[:, :, :, 0].any()
        fold = 4 if wall else 1  # a corner column holds its own lambda and three ring columns'
        mu, u = np.abs(fields[2:]) * fold, fields[:2] + (2.0 if dep else 0.0)
        sums = [12 * (mu[q] * u[q]).sum() + 4 * mu[q].sum() for q in (0, 0, 1, 1)]
        sums.append(((1 + mu[0] + mu[1]) * u[0] * u[1]).sum())
        assert (np.abs(grad - rgrad) <= 1e-6 * np.array(sums)).all()


@pytest.mark.parametrize("seed", range(5))
def test_grids_step_alone_from_a_phase_on(seed):
    """The phases a batch steps grid by grid are the last ones: all those, and no
    more, from which on every phase is estimated faster so."""
    batched = importlib.import_module(pkg().__name__ + ".batched")
    rng = np.random.default_rng(seed)
    cells = rng.choice([0.1, 0.5, 2.0, 6.0, 20.0, 60.0], 12)
    resident = cells < 1.0
    phases = batched._phases(rng.integers(1, 40, 12))

    def alone(active):
        own = sum(batched._solo_us(cells[c], resident[c]) for c in active)
        return own < 0.9 * batched._batched_us(sum(cells[c] for c in active))

    first = batched.solo_from(phases, cells, resident)
    assert all(alone(active) for _, _, active in phases[first:])
    assert first == 0 or not alone(phases[first - 1][2])
    assert batched.solo_from([], [], []) == 0


@pytest.mark.parametrize("n,no_z,wall,expected", [(51, 600, 0, 0), (51, 600, 1, 0), (59, 400, 0, 1), (86, 200, 0, 1)])
def test_tall_grids_step_flat(n, no_z, wall, expected):
    """Grids whose resident division is estimated slower than the flat step."""
    import ctypes

    native = importlib.import_module(pkg().__name__ + "._native")
    out = ctypes.c_int32(-1)
    g = _grid(native, n, no_z, wall, native.PIC_F32, 0)
    native.check(native.load().pic_segment_resident(ctypes.byref(g), ctypes.byref(out)), "pic_segment_resident")
    assert out.value == expected


@pytest.mark.gpu
@pytest.mark.parametrize("n,no_z", [(3, 1), (5, 20), (24, 200), (61, 200)])
def test_float64_lone_steps_equal_a_segments(n, no_z):
    """A step that finishes its own tallies (blocks of 256) and a segment's steps
    (blocks of 64, summed by the next one): the same fields, bit for bit, and the
    same tallies to the rounding of a sum of 1e6 values of one sign."""
    import ctypes

    import torch

    native = importlib.import_module(pkg().__name__ + "._native")
    lib = native.load()
    steps = 3
    state, xs, ys, off = _case(n, no_z, steps, n, 0)
    for wall in (0, 1):
        g = _grid(native, n, no_z, wall, native.PIC_F64, native.PIC_VARIANT_FLAT)
        whole = _segment(native, g, torch, state, xs, ys, off, 0)
        f = [torch.zeros((n, n, g.kpitch), dtype=torch.float64, device="cuda") for _ in range(4)]
        for q in range(2):
            f[q][:, :, : g.nzb] = torch.from_numpy(state[q])
        tally = torch.zeros((steps, 4), dtype=torch.float64, device="cuda")
        b = ctypes.c_int64()
        native.check(lib.pic_step_workspace_bytes(ctypes.byref(g), ctypes.byref(b)), "pic_step_workspace_bytes")
        ws = torch.zeros(b.value, dtype=torch.uint8, device="cuda")
        for s in range(steps):
            i, o = 2 * (s & 1), 2 * (~s & 1)
            native.check(lib.pic_step(ctypes.byref(g), f[i].data_ptr(), f[i + 1].data_ptr(), f[o].data_ptr(),
                                      f[o + 1].data_ptr(), None, None, tally[s].data_ptr(), ws.data_ptr(), ws.numel(),
                                      torch.cuda.current_stream().cuda_stream), "pic_step")
        out = 2 * (steps & 1)
        for q in range(2):
            assert np.array_equal(f[out + q][:, :, : g.nzb].cpu().numpy(), whole[q])
        np.testing.assert_allclose(tally.cpu().numpy(), whole[3], rtol=1e6 * 2.0**-53, atol=0)


@pytest.mark.parametrize("n,shape,variant", [(608, {}, 1), (608, dict(tile_rows=8), 2), (608, dict(ctas_per_sm=1), 2),
                                             (330, dict(tile_rows=8), 1), (1068, {}, 2)])
def test_a_shape_asks_for_the_streaming_step(n, shape, variant):
    """AUTO of 1e8 to 2e8 cells steps flat, but not where the caller gives the
    streaming step a shape, which is checked as ever."""
    import ctypes

    native = importlib.import_module(pkg().__name__ + "._native")
    g = _grid(native, n, 400, 0, native.PIC_F32, 0)
    for k, v in shape.items():
        setattr(g, k, v)
    out = native.PicGrid()
    native.check(native.load().pic_resolve_shape(ctypes.byref(g), ctypes.byref(out)), "pic_resolve_shape")
    assert out.variant == variant
    g.consumer_warps = 99
    refused = native.load().pic_resolve_shape(ctypes.byref(g), ctypes.byref(out)) != native.PIC_OK
    assert refused == (n * n * g.kpitch >= 10**8)
