"""GPU adjoint of the advection (lm_adjoint_*, k_adjoint.cu) against its FP64 checkers.

* the tape's forward in "f32" precision is bit-identical to the fused engine's advection (lm_step,
  no kick); the default "ds" precision carries positions in double-float;
* dL/d(lon0, lat0) and dL/d(u, v) agree with an FP64 torch autograd of the same scheme
  (oracle/adjoint_ref.py) and with FP64 central finite differences of the C oracle along random
  directions (h = 1e-6 deg for positions, 1e-6 m/s for the field);
* the gradient is deterministic: bit-identical across repeated backward sweeps and across
  checkpoint intervals (the recomputed segments are bit-identical to the forward);
* microbes that leave the domain are frozen and their gradient passes through unchanged.

The loss is the differentiation benchmark's: the mean squared great-circle distance between
final positions and seeded targets (initial positions plus N(0, 20 km) offsets).
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

KM_PER_DEG = 111.32


def _case(field, n, seed, box=(199.0, 202.0, 24.0, 27.0)):
    rng = np.random.default_rng(seed)
    lon = (box[0] + (box[1] - box[0]) * rng.random(n)).astype(np.float32)
    lat = (box[2] + (box[3] - box[2]) * rng.random(n)).astype(np.float32)
    tlon = lon.astype(np.float64) + rng.normal(0, 20.0 / KM_PER_DEG, n)
    tlat = lat.astype(np.float64) + rng.normal(0, 20.0 / KM_PER_DEG, n)
    return lon, lat, tlon, tlat


def _gpu_grads(field, lon, lat, tlon, tlat, t0, dt, n_steps, k, allow_oob=False, weight=None, precision="f32"):
    from lagrangian_microbes_gb300.adjoint import AdjointTape, advect_rk4, great_circle_m
    dev = torch.device("cuda:0")
    l0 = torch.from_numpy(lon).to(dev).requires_grad_(True)
    a0 = torch.from_numpy(lat).to(dev).requires_grad_(True)
    u = torch.from_numpy(field.u).to(dev).requires_grad_(True)
    v = torch.from_numpy(field.v).to(dev).requires_grad_(True)
    tape = AdjointTape(precision=precision)
    x, y = advect_rk4(l0, a0, u, v, field.lon, field.lat, field.times, t0, dt, n_steps, checkpoint_every=k,
                      tape=tape, allow_out_of_bounds=allow_oob)
    dist = great_circle_m(x.double(), y.double(), torch.from_numpy(tlon).to(dev), torch.from_numpy(tlat).to(dev))
    w = torch.ones_like(dist) if weight is None else torch.from_numpy(np.asarray(weight, np.float64)).to(dev)
    loss = (w * dist * dist).sum() / dist.numel()  # the mean squared distance (over the weighted microbes)
    loss.backward()
    out = [t.grad.double().cpu().numpy() for t in (l0, a0, u, v)]
    sig = tape.cell_signature().cpu().numpy().view(np.uint64)
    res = (x.detach().cpu().numpy(), y.detach().cpu().numpy(), float(loss.detach()), out, sig)
    tape.close()
    tape.ctx.close()
    return res


def _fp64_grads(field, lon, lat, tlon, tlat, t0, dt, n_steps, weight=None):
    import adjoint_ref
    tl = [torch.from_numpy(np.asarray(a, np.float64).copy()).requires_grad_(True)
          for a in (lon, lat, field.u, field.v)]
    x, y = adjoint_ref.advect(field.lon, field.lat, field.times, tl[2], tl[3], tl[0], tl[1], t0, dt, n_steps,
                              checkpoint_every=16)
    dist = adjoint_ref.haversine_m(x, y, torch.from_numpy(tlon), torch.from_numpy(tlat))
    w = torch.ones_like(dist) if weight is None else torch.from_numpy(np.asarray(weight, np.float64))
    loss = (w * dist * dist).sum() / dist.numel()
    loss.backward()
    return float(loss.detach()), [t.grad.numpy() for t in tl]


def _fp64_signature(orc, f, lon, lat, t0, dt, n_steps):
    return orc.advect_f64_field64(f.u, f.v, f.lon, f.lat, f.times, np.asarray(lon, np.float64),
                                  np.asarray(lat, np.float64), t0, dt, n_steps, cell_signature=True)[3]


def central_difference(orc, f, lon, lat, tlon, tlat, t0, dt, n_steps, d, h=1e-6, path=None):
    """FP64 central difference of the loss along direction d = (d_lon0, d_lat0, d_u, d_v), over the
    microbes whose two runs sample the same grid cells at every stage (the others straddle an edge
    of the piecewise-bilinear field, where the derivative jumps) and, with `path`, the cells of the
    GPU run too. Returns (fd, keep mask)."""
    import adjoint_ref
    runs = []
    for s in (h, -h):
        x, y, _, sig = orc.advect_f64_field64(f.u.astype(np.float64) + s * d[2], f.v.astype(np.float64) + s * d[3],
                                              f.lon, f.lat, f.times, lon.astype(np.float64) + s * d[0],
                                              lat.astype(np.float64) + s * d[1], t0, dt, n_steps, cell_signature=True)
        dd = adjoint_ref.haversine_m(torch.from_numpy(x), torch.from_numpy(y), torch.from_numpy(tlon),
                                     torch.from_numpy(tlat)).numpy()
        runs.append((dd * dd, sig))
    keep = runs[0][1] == runs[1][1]
    if path is not None:
        keep &= runs[0][1] == path
    fd = float((runs[0][0] - runs[1][0])[keep].sum()) / lon.size / (2 * h)
    return fd, keep


def _rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


def test_adjoint_forward_bit_identical_to_engine_advection(lm, small_field):
    f = small_field
    lon, lat, _, _ = _case(f, 5000, 1)
    t0, dt, n_steps = float(f.times[0]), 3600.0, 40
    sim = lm.Simulation(f, lon.astype(np.float64), lat.astype(np.float64), np.ones(lon.size, np.int8), kh=0.0)
    sim.step(t0, dt, n_steps, interact=False)
    want_lon, want_lat, _, st = sim.state()
    sim.close()
    assert (st == 0).all()
    x, y, _, _, _ = _gpu_grads(f, lon, lat, lon.astype(np.float64), lat.astype(np.float64), t0, dt, n_steps, 7)
    np.testing.assert_array_equal(x, want_lon)
    np.testing.assert_array_equal(y, want_lat)


@pytest.mark.parametrize("precision", ["f32", "ds"])
def test_adjoint_matches_fp64_autograd_and_finite_differences(lm, orc, small_field, precision):
    """Gradients within 1e-4 relative of the FP64 scheme, microbe by microbe on the same cell path.

    The map is piecewise smooth: moving a start by 0.1 m moves the FP64 gradient itself by ~1e-4
    when a stage crosses a cell edge, and the float32 trajectory sits ~0.1-1 m from the FP64 one.
    The comparison therefore keeps the microbes whose GPU and FP64 runs sample the same cells (the
    GPU reports its path, lm_adjoint_cell_signature) and reports how many that is."""
    f = small_field
    lon, lat, tlon, tlat = _case(f, 3000, 2)
    t0, dt, n_steps = float(f.times[0]), 3600.0, 48
    _, _, loss32, g, sig = _gpu_grads(f, lon, lat, tlon, tlat, t0, dt, n_steps, 16, precision=precision)
    same = sig == _fp64_signature(orc, f, lon, lat, t0, dt, n_steps)
    assert same.mean() >= 0.97, same.mean()
    loss64, g64 = _fp64_grads(f, lon, lat, tlon, tlat, t0, dt, n_steps)
    assert abs(loss32 - loss64) <= 1e-5 * loss64
    errs = [_rel(a, b) for a, b in zip(g, g64)]
    assert max(errs) < 1e-3, errs  # all microbes, cell-edge crossings included
    _, _, _, gs, _ = _gpu_grads(f, lon, lat, tlon, tlat, t0, dt, n_steps, 16, weight=same, precision=precision)
    _, g64s = _fp64_grads(f, lon, lat, tlon, tlat, t0, dt, n_steps, weight=same)
    errs = [_rel(a, b) for a, b in zip(gs, g64s)]
    assert max(errs) < 1e-4, errs
    # directional derivatives vs FP64 central differences of the C oracle on a float64 field
    # (error of the vector of 16 directional derivatives: a single direction whose derivative happens
    # to be near zero would inflate a per-direction ratio without any loss of accuracy)
    rng = np.random.default_rng(5)
    ads, fds, dropped = [], [], 0
    for _ in range(16):
        d = [rng.standard_normal(a.shape) for a in (lon, lat, f.u, f.v)]
        fd, keep = central_difference(orc, f, lon, lat, tlon, tlat, t0, dt, n_steps, d, path=sig)
        dropped = max(dropped, int((~keep).sum()))
        _, _, _, gk, _ = _gpu_grads(f, lon, lat, tlon, tlat, t0, dt, n_steps, 16, weight=keep, precision=precision)
        ads.append(sum(float((gg * dd).sum()) for gg, dd in zip(gk, d)))
        fds.append(fd)
    ads, fds = np.array(ads), np.array(fds)
    assert dropped <= lon.size * 3 // 100
    assert _rel(ads, fds) < 1e-4, (ads, fds)
    assert np.median(np.abs(ads - fds) / np.abs(fds)) < 1e-4


@pytest.mark.parametrize("precision", ["f32", "ds"])
def test_adjoint_gradient_is_deterministic_across_runs_and_checkpoint_intervals(lm, small_field, precision):
    f = small_field
    lon, lat, tlon, tlat = _case(f, 20000, 3)
    t0, dt, n_steps = float(f.times[0]), 3600.0, 30
    ref = _gpu_grads(f, lon, lat, tlon, tlat, t0, dt, n_steps, 30, precision=precision)
    for k in (30, 1, 7):
        got = _gpu_grads(f, lon, lat, tlon, tlat, t0, dt, n_steps, k, precision=precision)
        np.testing.assert_array_equal(got[0], ref[0])
        for a, b in zip(got[3], ref[3]):
            np.testing.assert_array_equal(a, b)


def test_adjoint_repeated_backward_is_bit_identical(lm, small_field):
    from lagrangian_microbes_gb300.adjoint import AdjointTape
    f = small_field
    lon, lat, _, _ = _case(f, 10000, 4)
    dev = torch.device("cuda:0")
    tape = AdjointTape()
    tape.forward(torch.from_numpy(lon).to(dev), torch.from_numpy(lat).to(dev), torch.from_numpy(f.u).to(dev),
                 torch.from_numpy(f.v).to(dev), f.lon, f.lat, f.times, float(f.times[0]), 3600.0, 20, 8)
    g = torch.randn(2, lon.size, device=dev)
    first = [t.cpu().numpy() for t in tape.backward(g[0], g[1])]
    second = [t.cpu().numpy() for t in tape.backward(g[0], g[1])]
    for a, b in zip(first, second):
        np.testing.assert_array_equal(a, b)
    tape.close()


def test_adjoint_frozen_microbes_pass_their_gradient_through(lm, orc, small_field):
    f = small_field
    # a strip hugging the eastern edge: some microbes leave the grid and freeze
    lon, lat, tlon, tlat = _case(f, 2000, 6, box=(205.85, 206.0, 24.0, 27.0))
    t0, dt, n_steps = float(f.times[0]), 3600.0, 24
    _, _, st = orc.advect_f64(f, lon, lat, t0, dt, n_steps)
    assert 0 < int((st != 0).sum()) < lon.size  # some froze, some stayed
    sig64 = _fp64_signature(orc, f, lon, lat, t0, dt, n_steps)
    _, _, _, _, sig = _gpu_grads(f, lon, lat, tlon, tlat, t0, dt, n_steps, 8, allow_oob=True)
    same = sig == sig64
    assert same.mean() >= 0.97
    _, _, _, g, _ = _gpu_grads(f, lon, lat, tlon, tlat, t0, dt, n_steps, 8, allow_oob=True, weight=same)
    _, g64 = _fp64_grads(f, lon, lat, tlon, tlat, t0, dt, n_steps, weight=same)
    errs = [_rel(a, b) for a, b in zip(g, g64)]
    assert max(errs) < 1e-4, errs


def test_adjoint_time_window_outside_field_raises(lm, small_field):
    from lagrangian_microbes_gb300 import TimeRangeError
    from lagrangian_microbes_gb300.adjoint import AdjointTape
    f = small_field
    dev = torch.device("cuda:0")
    z = torch.zeros(4, device=dev) + 200.0
    tape = AdjointTape()
    with pytest.raises(TimeRangeError):
        tape.forward(z, z - 175.0, torch.from_numpy(f.u).to(dev), torch.from_numpy(f.v).to(dev), f.lon, f.lat, f.times,
                     float(f.times[-1]), 3600.0, 5)
    tape.close()


def test_adjoint_f64_trajectories_track_the_fp64_scheme(lm, orc, small_field):
    """FP64 mode: positions within 1e-9 deg of the FP64 oracle and gradients within 1e-5 of the FP64
    autograd on every microbe (no cell-path selection needed), deterministic across intervals."""
    f = small_field
    lon, lat, tlon, tlat = _case(f, 3000, 8)
    t0, dt, n_steps = float(f.times[0]), 3600.0, 48
    x, y, loss, g, sig = _gpu_grads(f, lon, lat, tlon, tlat, t0, dt, n_steps, 16, precision="f64")
    x64, y64, _, sig64 = orc.advect_f64_field64(f.u, f.v, f.lon, f.lat, f.times, lon.astype(np.float64),
                                                lat.astype(np.float64), t0, dt, n_steps, cell_signature=True)
    # final positions come back as float64 in this mode
    assert x.dtype == np.float64 and np.abs(x - x64).max() <= 1e-9 and np.abs(y - y64).max() <= 1e-9
    assert (sig == sig64).all()
    loss64, g64 = _fp64_grads(f, lon, lat, tlon, tlat, t0, dt, n_steps)
    errs = [_rel(a, b) for a, b in zip(g, g64)]
    assert max(errs) < 1e-5, errs
    again = _gpu_grads(f, lon, lat, tlon, tlat, t0, dt, n_steps, 5, precision="f64")
    for a, b in zip(again[3], g):
        np.testing.assert_array_equal(a, b)


def test_adjoint_steps_longer_than_a_cell_fall_back_to_the_record_form(lm, orc):
    """Stages that leave the 3 x 3 cells around a step's start (a fine grid, fast flow) switch the
    backward to sorting the stage records themselves; the gradient still matches the FP64 scheme
    and is deterministic."""
    f = lm.synthetic_psi_field(199.0, 203.0, 24.0, 28.0, 0.02, n_frames=8, frame_seconds=3600.0, rms_speed=2.0,
                               seed=3)
    lon, lat, tlon, tlat = _case(f, 2000, 9, box=(200.5, 201.5, 25.5, 26.5))
    t0, dt, n_steps = float(f.times[0]), 3600.0, 6
    _, _, _, g, sig = _gpu_grads(f, lon, lat, tlon, tlat, t0, dt, n_steps, 4)
    same = sig == _fp64_signature(orc, f, lon, lat, t0, dt, n_steps)
    assert same.mean() >= 0.9
    _, _, _, gs, _ = _gpu_grads(f, lon, lat, tlon, tlat, t0, dt, n_steps, 4, weight=same)
    _, g64 = _fp64_grads(f, lon, lat, tlon, tlat, t0, dt, n_steps, weight=same)
    errs = [_rel(a, b) for a, b in zip(gs, g64)]
    assert max(errs) < 1e-4, errs
    again = _gpu_grads(f, lon, lat, tlon, tlat, t0, dt, n_steps, 3)
    for a, b in zip(again[3], g):
        np.testing.assert_array_equal(a, b)


def _tape_backward(f, lon, lat, g, n_steps, k, precision, dt=3600.0):
    from lagrangian_microbes_gb300.adjoint import AdjointTape
    dev = torch.device("cuda:0")
    tape = AdjointTape(precision=precision)
    tape.forward(torch.from_numpy(lon).to(dev), torch.from_numpy(lat).to(dev), torch.from_numpy(f.u).to(dev),
                 torch.from_numpy(f.v).to(dev), f.lon, f.lat, f.times, float(f.times[0]), dt, n_steps, k)
    out = [[t.cpu().numpy() for t in tape.backward(torch.from_numpy(g[0]).to(dev), torch.from_numpy(g[1]).to(dev))]
           for _ in range(2)]
    tape.close()
    tape.ctx.close()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
    return out[0]


@pytest.mark.parametrize("precision", ["f32", "ds", "f64"])
@pytest.mark.parametrize("n", [1, 31, 127, 128, 129, 257, 5000])
def test_adjoint_field_gradient_does_not_depend_on_the_order_of_the_microbes(small_field, n, precision):
    """All microbes in one field cell (one item of its sums, several, a ragged last one) beside
    scattered ones, adjoints over twelve decades: the field's gradient is bit-identical for shuffled
    microbes (the sums are integers), and so are the microbes' own gradients."""
    f = small_field
    rng = np.random.default_rng(60 + n)
    lon = np.concatenate([200.05 + 0.15 * rng.random(n), 199 + 3 * rng.random(300)]).astype(np.float32)
    lat = np.concatenate([25.05 + 0.15 * rng.random(n), 24 + 3 * rng.random(300)]).astype(np.float32)
    g = (rng.standard_normal((2, lon.size)) * 10.0 ** rng.uniform(-6, 6, lon.size)).astype(np.float32)
    ref = _tape_backward(f, lon, lat, g, 7, 3, precision)
    p = rng.permutation(lon.size)
    got = _tape_backward(f, lon[p], lat[p], np.ascontiguousarray(g[:, p]), 7, 7, precision)
    for a, b in zip(got[:2], ref[:2]):
        np.testing.assert_array_equal(a, b[p])
    for a, b in zip(got[2:], ref[2:]):
        np.testing.assert_array_equal(a, b)


def _still_field(lm, n_frames=3):
    axis = 0.125 * np.arange(17)
    zero = np.zeros((n_frames, 17, 17), np.float32)
    return lm.VelocityField(200.0 + axis, 25.0 + axis, 3600.0 * np.arange(n_frames), zero, zero)


def _still_gradient(f, lon, lat, g, share, magnitude=False):
    """dL/dU, dL/dV per frame of one step in a field at rest, in float64: a microbe stays where it is, so a node gets its
    bilinear weight times its adjoint times the frame's share of the step, in field units. Positions are multiples of
    1/4 of a cell here, exact in every precision."""
    out = np.zeros((2, len(share), 17, 17))
    x, y = (lon.astype(np.float64) - 200.0) * 8.0, (lat.astype(np.float64) - 25.0) * 8.0
    i, j = np.minimum(x.astype(int), 15), np.minimum(y.astype(int), 15)
    a, b = x - i, y - j
    m = 1852.0 * 60.0
    per = np.stack([g[0] / (m * np.cos(np.deg2rad(lat.astype(np.float64)))), g[1] / m])
    if magnitude:
        per = np.abs(per)
    for dj, di, w in ((0, 0, (1 - a) * (1 - b)), (0, 1, a * (1 - b)), (1, 0, (1 - a) * b), (1, 1, a * b)):
        for k in range(2):
            for fr, s in enumerate(share):
                np.add.at(out[k, fr], (j + dj, i + di), w * per[k].astype(np.float64) * s)
    return out


@pytest.mark.parametrize("precision", ["f32", "ds", "f64"])
@pytest.mark.parametrize("n, large", [(3, 1e8), (3, 1e12), (200, 1e10), (700, 1e14), (4500, 1e8), (140_000, 1e12), (0, 0)])
def test_adjoint_small_terms_beside_large_ones_keep_their_digits(lm, n, large, precision):
    """A node's sum of small terms is as accurate as its own terms, whatever adjoints the field cell holds elsewhere: one
    large adjoint on a cell's corner beside n ordinary ones (no term of it at the other nodes, none in dL/dV), and
    adjoints over fourteen decades on the edges and inside of 36 cells. Bound: some 20 roundings of 2^-24 and a float32
    cosine within 2 ulp on the way from a term to the gradient, 24 x 2^-24 = 1.43e-6 of the terms' magnitude."""
    f = _still_field(lm)
    rng = np.random.default_rng(63 + n)
    if large:
        q = rng.integers(1, 4, (2, n))  # inside the cell
        lon = np.concatenate([[200.5], 200.5 + 0.03125 * q[0]]).astype(np.float32)
        lat = np.concatenate([[25.25], 25.25 + 0.03125 * q[1]]).astype(np.float32)
        g = rng.uniform(0.5, 2.0, (2, n + 1)).astype(np.float32)
        g[0, 0] = large
    else:
        lon = (200.5 + 0.03125 * rng.integers(0, 24, 500)).astype(np.float32)
        lat = (25.5 + 0.03125 * rng.integers(0, 24, 500)).astype(np.float32)
        g = (rng.standard_normal((2, 500)) * 10.0 ** rng.uniform(-7, 7, 500)).astype(np.float32)
    got = _tape_backward(f, lon, lat, g, 1, 1, precision)
    share = (1800.0, 1800.0, 0.0)  # of 3,600 s: stage 1 at frame 0, stages 2 and 3 between the frames, stage 4 at frame 1
    want, size = (_still_gradient(f, lon, lat, g, share, m) for m in (False, True))
    for k in range(2):
        err = np.abs(got[2 + k].astype(np.float64) - want[k])
        assert (err <= 1.5e-6 * size[k]).all(), (k, (err / np.maximum(size[k], 1e-300)).max())


@pytest.mark.parametrize("precision", ["f64", "ds", "f32"])
def test_adjoint_takes_the_stages_that_the_forward_took_at_the_domain_edge(lm, precision):
    """A steady zonal flow towards the domain's edge: the longest step whose last stage the forward still finds inside has
    a gradient in the backward, and the next longer one, which the forward freezes, has none. The two agree only if
    their stage positions do, to the last bit."""
    from lagrangian_microbes_gb300.adjoint import AdjointTape
    axis = 0.125 * np.arange(17)
    lats = np.linspace(25.03, 26.96, 48).astype(np.float32)
    dev = torch.device("cuda:0")
    u = torch.full((2, 17, 17), 0.731, device=dev)
    args = (u, torch.zeros_like(u), 200.0 + axis, 25.0 + axis, np.array([0.0, 20000.0]), 0.0)
    tape = AdjointTape(precision=precision)

    def ends(lat, dt):  # is the step taken?
        lon0, lat0 = torch.full((len(lat),), 201.9375, device=dev), torch.from_numpy(lat).to(dev)
        lon, _ = tape.forward(lon0, lat0, *args, dt, 1, 1, True)
        return (lon.double() != lon0.double()).cpu().numpy()

    one = torch.ones(1, device=dev)
    step = np.float32 if precision != "f64" else np.float64  # the kernels' type of dt
    for lat in lats:
        lo, hi = step(5000.0), step(15000.0)
        assert ends(lat[None], float(lo))[0] and not ends(lat[None], float(hi))[0]
        while np.nextafter(lo, hi) < hi:
            mid = step((float(lo) + float(hi)) / 2)
            if ends(lat[None], float(mid))[0]:
                lo = mid
            else:
                hi = mid
        for dt, taken in ((lo, True), (hi, False)):
            assert ends(lat[None], float(dt))[0] == taken
            assert tape.backward(one, 0 * one)[2].any().item() == taken, (lat, dt)
    tape.close()
    tape.ctx.close()


@pytest.mark.parametrize("n", [30, 500])
def test_adjoint_finite_sums_of_a_cell_with_an_infinite_adjoint_are_exact(lm, n):
    """One infinite longitude adjoint makes its cell's sums of dL/dU infinite or undefined; dL/dV at the last stage's
    frame has finite terms only and stays what it is, for shuffled microbes bit by bit."""
    f = _still_field(lm)
    rng = np.random.default_rng(64 + n)
    lon = (200.5 + 0.03125 * rng.integers(0, 4, n)).astype(np.float32)
    lat = (25.5 + 0.03125 * rng.integers(0, 4, n)).astype(np.float32)
    g = (rng.standard_normal((2, n)) * 10.0 ** rng.uniform(-3, 3, n)).astype(np.float32)
    g[0, n // 2] = np.inf
    got = _tape_backward(f, lon, lat, g, 1, 1, "f32", dt=7200.0)  # the stages at frames 0, 1, 1 and 2
    share = (0.0, 0.0, 1200.0)
    want, size = (_still_gradient(f, lon, lat, np.where(np.isfinite(g), g, 0), share, m)[1, 2] for m in (False, True))
    assert (np.abs(got[3][2].astype(np.float64) - want) <= 1.5e-6 * size).all()
    assert not np.isfinite(got[2][2, 4:6, 4:6]).any() and (got[2][2] == 0).sum() >= 17 * 17 - 9
    for _ in range(3):
        p = rng.permutation(n)
        again = _tape_backward(f, lon[p], lat[p], np.ascontiguousarray(g[:, p]), 1, 1, "f32", dt=7200.0)
        for a, b in zip(again[2:], got[2:]):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("n", [40, 400])
def test_adjoint_dense_cells_match_fp64_autograd(lm, orc, small_field, n):
    """n microbes per field cell of a 3 x 3 patch, against the FP64 autograd on the same cell paths
    (float32 terms, so the bound of the scattered cases)."""
    f = small_field
    lon, lat, tlon, tlat = _case(f, 9 * n, 61, box=(200.0, 200.75, 25.0, 25.75))
    t0, dt, n_steps = float(f.times[0]), 3600.0, 10
    sig = _gpu_grads(f, lon, lat, tlon, tlat, t0, dt, n_steps, 4)[4]
    same = sig == _fp64_signature(orc, f, lon, lat, t0, dt, n_steps)
    assert same.mean() >= 0.97
    g = _gpu_grads(f, lon, lat, tlon, tlat, t0, dt, n_steps, 4, weight=same)[3]
    _, g64 = _fp64_grads(f, lon, lat, tlon, tlat, t0, dt, n_steps, weight=same)
    errs = [_rel(a, b) for a, b in zip(g, g64)]
    assert max(errs) < 1e-4, errs


@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_adjoint_non_finite_gradients_stay_in_their_cells(small_field, bad):
    f = small_field
    rng = np.random.default_rng(62)
    lon = np.concatenate([200.05 + 0.15 * rng.random(300), [202.6]]).astype(np.float32)
    lat = np.concatenate([25.05 + 0.15 * rng.random(300), [26.6]]).astype(np.float32)
    g = rng.standard_normal((2, lon.size)).astype(np.float32)
    clean = _tape_backward(f, lon[:-1], lat[:-1], np.ascontiguousarray(g[:, :-1]), 4, 4, "f32")
    g[:, -1] = bad
    got = _tape_backward(f, lon, lat, g, 4, 4, "f32")
    assert not np.isfinite(got[0][-1]) and np.isfinite(got[0][:-1]).all()
    for a, b in zip(got[2:], clean[2:]):
        touched = ~np.isfinite(a)
        assert touched.any() and not b[touched].any()  # the nodes around the one microbe alone
        np.testing.assert_array_equal(a[~touched], b[~touched])
    few = int((~np.isfinite(got[2])).sum())
    g[:, 5] = bad  # and in a cell of several items
    got = _tape_backward(f, lon, lat, g, 4, 4, "f32")
    assert int((~np.isfinite(got[2])).sum()) > few


def test_forward_without_a_gradient_does_not_store_its_states(lm, small_field, monkeypatch):
    """Only a run that autograd records stores the last segment's states; a backward finds the same gradient either way."""
    from lagrangian_microbes_gb300 import adjoint
    f, dev = small_field, torch.device("cuda:0")
    lon, lat, _, _ = _case(f, 700, 6)
    put = lambda a: torch.from_numpy(np.ascontiguousarray(a, np.float32)).to(dev)
    args = [put(a) for a in (lon, lat, f.u, f.v)]
    rest = (f.lon, f.lat, f.times, float(f.times[0]), 3600.0, 5)
    asked, plain = [], adjoint.AdjointTape.forward
    monkeypatch.setattr(adjoint.AdjointTape, "forward",
                        lambda self, *a, **k: asked.append(k.get("keep_states", a[12] if len(a) > 12 else True)) or plain(self, *a, **k))
    tape = adjoint.AdjointTape()
    adjoint.advect_rk4(*args, *rest, tape=tape)
    args[0].requires_grad_()
    with torch.no_grad():
        adjoint.advect_rk4(*args, *rest, tape=tape)
    adjoint.advect_rk4(*args, *rest, tape=tape)
    assert asked == [False, False, True]
    one = torch.ones(700, device=dev)
    got = []
    for keep in (True, False):
        plain(tape, *(t.detach() for t in args), *rest, checkpoint_every=2, keep_states=keep)
        got.append(tape.backward(one, 2 * one))
    for a, b in zip(*got):
        assert torch.equal(a, b)
    tape.close()


def test_adjoint_takes_smaller_batches_where_memory_is_short(lm, small_field):
    """4,000,000 microbes with 1.4 GB left on the device: one set of batch buffers for one step fits (283 bytes a microbe
    with the tape's own), two do not. The gradients are those of a run with the memory it likes."""
    from lagrangian_microbes_gb300.adjoint import AdjointTape
    f, n, dev = small_field, 4_000_000, torch.device("cuda:0")
    gen = torch.Generator(device=dev).manual_seed(5)
    lon, lat = (lo + 2.0 * torch.rand(n, device=dev, generator=gen) for lo in (199.5, 24.5))
    g = [torch.randn(n, device=dev, generator=gen) for _ in range(2)]
    u, v = torch.from_numpy(f.u).to(dev), torch.from_numpy(f.v).to(dev)

    def run():
        tape = AdjointTape(precision="ds")
        out = tape.forward(lon, lat, u, v, f.lon, f.lat, f.times, float(f.times[0]), 3600.0, 4, 4)
        out = [t.cpu() for t in (*out, *tape.backward(*g))]
        tape.close()
        tape.ctx.close()
        return out

    want = run()
    torch.cuda.empty_cache()
    left = torch.cuda.mem_get_info()[0] - 1400 * 10 ** 6
    if left < 0:
        pytest.skip("less than 1.4 GB free")
    hog = torch.empty(left, dtype=torch.uint8, device=dev)
    try:
        got = run()
    finally:
        del hog
        torch.cuda.empty_cache()
    for a, b in zip(got, want):
        assert torch.equal(a, b)


def test_tape_waits_for_the_default_streams_work(lm, small_field):
    """Inputs still being written on the default stream when the call is made (a pause of some milliseconds before
    them), forward and backward: the results of finished inputs."""
    from lagrangian_microbes_gb300.adjoint import AdjointTape
    lon, lat, _, _ = _case(small_field, 4000, 5)
    dev = torch.device("cuda:0")
    ready = [torch.from_numpy(np.ascontiguousarray(a, np.float32)).to(dev) for a in (lon, lat, small_field.u, small_field.v)]
    weights = [torch.linspace(-1, 1, 4000, device=dev), torch.linspace(2, -1, 4000, device=dev)]
    axes = (small_field.lon, small_field.lat, small_field.times)
    t0 = float(small_field.times[0])
    tape = AdjointTape(precision="ds")
    want = tape.forward(*ready, *axes, t0, 3600.0, 6), None
    want = want[0], tape.backward(*weights)
    late = [torch.zeros_like(t) for t in ready + weights]
    late[0].fill_(200.5), late[1].fill_(25.5)
    torch.cuda.synchronize()
    torch.cuda._sleep(20_000_000)
    for a, b in zip(late[:4], ready):
        a.copy_(b)
    got = tape.forward(*late[:4], *axes, t0, 3600.0, 6)
    torch.cuda._sleep(20_000_000)
    for a, b in zip(late[4:], weights):
        a.copy_(b)
    for a, b in zip((*got, *tape.backward(*late[4:])), (*want[0], *want[1])):
        assert torch.equal(a, b)
    tape.close()


@pytest.mark.parametrize("n, dtype, target_dtype", [(1, "float32", "float32"), (255, "float64", "float32"), (257, "float32", "float64"),
                                                    (4099, "float16", "float64"), (152 * 8 * 256 + 1, "float64", "float64")])
def test_squared_distance_kernel_equals_the_tensor_operations(lm, n, dtype, target_dtype):
    """k_loss against the same loss as torch operations. Each side rounds some 20 times on the way to a derivative, and
    1 - q^2 >= 0.02 amplifies by at most 50: 20 x 51 x 2^-53 = 1.1e-13 a side, relative to the terms that are added."""
    import torch
    from lagrangian_microbes_gb300 import adjoint
    gen = torch.Generator().manual_seed(n)
    u = lambda lo, hi: (lo + (hi - lo) * torch.rand(n, generator=gen, dtype=torch.float64))
    lon, lat = (t.to(getattr(torch, dtype)).cuda().requires_grad_() for t in (u(-180, 180), u(-89, 89)))
    if n > 300:  # near and far targets (great circles up to 160 degrees)
        tl, ta = lon.detach().cpu().double() + u(-0.5, 0.5), (lat.detach().cpu().double() + u(-0.5, 0.5)).clamp(-89, 89)
    else:
        tl, ta = lon.detach().cpu().double() + u(-100, 100), u(-40, 40)
    tl, ta = (t.to(getattr(torch, target_dtype)).cuda() for t in (tl, ta))
    assert adjoint._one_kernel((lon, lat, tl, ta))
    want = adjoint._squared_distance_mean(lon, lat, tl, ta)
    w_lon, w_lat = torch.autograd.grad(want, (lon, lat))
    kept = tl.clone(), ta.clone()
    got = adjoint.mean_squared_distance(lon, lat, tl, ta)
    assert got.dtype == torch.float64 and got.shape == () and got.requires_grad
    with torch.no_grad():
        np.testing.assert_allclose(adjoint.mean_squared_distance(lon, lat, tl, ta).item(), want.item(), rtol=5e-13)
        tl.zero_(), ta.zero_()  # the caller's buffers may be filled again before the backward
    g_lon, g_lat = torch.autograd.grad(got, (lon, lat))
    tl.copy_(kept[0]), ta.copy_(kept[1])
    np.testing.assert_allclose(got.item(), want.item(), rtol=5e-13)
    p1, p2 = lat.detach().double() * np.pi / 180, ta.double() * np.pi / 180
    dl = (tl.double() - lon.detach().double()) * np.pi / 360
    a, c = torch.sin((p2 - p1) / 2), torch.sin(dl)
    terms = (a * torch.cos((p2 - p1) / 2)).abs() + (torch.sin(p1) * torch.cos(p2) * c * c).abs()
    net = (a * torch.cos((p2 - p1) / 2) + torch.sin(p1) * torch.cos(p2) * c * c).abs()
    eps = {"float16": 2.0 ** -10, "float32": 2.0 ** -23}.get(dtype, 0.0)  # the result's own rounding
    for g, w, t in ((g_lon, w_lon, torch.ones_like(terms)), (g_lat, w_lat, terms / net.clamp(min=1e-300))):
        assert g.dtype == lon.dtype
        bound = w.double().abs() * (5e-13 * t + eps) + (6e-8 if dtype == "float16" else 1e-44)
        assert bool(((g == w) | ((g.double() - w.double()).abs() <= bound)).all())  # (float16 overflows alike)


def test_squared_distance_beyond_the_plain_call(lm):
    """What the loss kernel does not take goes through the tensor operations, with their results: functorch transforms,
    forward mode, derivatives by the targets, broadcast shapes, the CPU; and what it takes: second derivatives,
    batched gradients, capture, another stream, a microbe on its target (its derivative is undefined there)."""
    import torch
    from lagrangian_microbes_gb300 import adjoint
    f = adjoint.mean_squared_distance
    gen = torch.Generator().manual_seed(3)
    lon, lat, tl, ta = (torch.rand(2, 33, generator=gen, dtype=torch.float64).cuda() + k for k in (10, 20, 10.2, 20.1))
    ref = adjoint._squared_distance_mean
    close = lambda a, b: torch.testing.assert_close(a, b, rtol=1e-11, atol=0, equal_nan=True)
    close(torch.func.vmap(f)(lon, lat, tl, ta), torch.func.vmap(ref)(lon, lat, tl, ta))
    close(torch.func.grad(f)(lon, lat, tl, ta), torch.func.grad(ref)(lon, lat, tl, ta))
    close(torch.func.jvp(f, (lon, lat, tl, ta), (lon, lat, tl, ta))[1], torch.func.jvp(ref, (lon, lat, tl, ta), (lon, lat, tl, ta))[1])
    close(f(lon, lat[0], tl, ta[:, :1]), ref(lon, lat[0], tl, ta[:, :1]))
    close(f(*(t.cpu() for t in (lon, lat, tl, ta))).cuda(), ref(lon, lat, tl, ta))
    assert torch.isnan(f(lon[:, :0], lat[:, :0], tl[:, :0], ta[:, :0]))
    x, y, tx = (t.clone().requires_grad_() for t in (lon, lat, tl))
    for a, b in zip(torch.autograd.grad(f(x, y, tx, ta), (x, y, tx)), torch.autograd.grad(ref(x, y, tx, ta), (x, y, tx))):
        close(a, b)
    second = []
    for g in (f, ref):
        gx, gy = torch.autograd.grad(g(x, y, tl, ta), (x, y), create_graph=True)
        second.append(torch.autograd.grad((gx * gx).sum() + (gx * gy).sum(), (x, y)))
    for a, b in zip(*second):
        torch.testing.assert_close(a, b, rtol=1e-9, atol=1e-3)
    weights = torch.tensor([1.0, -2.0, 0.5], dtype=torch.float64).cuda()
    (rows,) = torch.autograd.grad(f(x.t(), y.t(), tl.t(), ta.t()), x, weights, is_grads_batched=True)
    close(rows, weights[:, None, None] * torch.autograd.grad(ref(x, y, tl, ta), x)[0])
    (g,) = torch.autograd.grad(f(x, y, torch.cat([lon[:1], tl[1:]]), torch.cat([lat[:1], ta[1:]])), x)
    assert torch.isnan(g[0]).all() and torch.isfinite(g[1]).all()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        f(lon, lat, tl, ta)
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = f(lon, lat, tl, ta)
    lon.add_(0.25)
    graph.replay()
    close(out, ref(lon, lat, tl, ta))


def test_squared_distance_compiles_and_traces_as_one_graph(lm):
    """Under torch.compile without graph breaks, and under torch.jit.trace, the loss is its tensor operations."""
    from lagrangian_microbes_gb300 import adjoint
    f = adjoint.mean_squared_distance
    gen = torch.Generator().manual_seed(4)
    lon, lat, tl, ta = (torch.rand(65, generator=gen, dtype=torch.float64).cuda() + k for k in (10, 20, 10.2, 20.1))
    close = lambda a, b: torch.testing.assert_close(a, b, rtol=1e-11, atol=0)
    want = adjoint._squared_distance_mean(lon, lat, tl, ta)
    close(torch.compile(f, fullgraph=True, backend="eager")(lon, lat, tl, ta), want)
    x = lon.clone().requires_grad_()
    (g,) = torch.autograd.grad(torch.compile(f, fullgraph=True, backend="eager")(x, lat, tl, ta), x)
    (w,) = torch.autograd.grad(adjoint._squared_distance_mean(x, lat, tl, ta), x)
    close(g, w)
    traced = torch.jit.trace(f, (lon, lat, tl, ta))
    close(traced(lon + 0.5, lat, tl, ta), adjoint._squared_distance_mean(lon + 0.5, lat, tl, ta))
