"""Stage kernels, run loop and host copies at the sizes and values where they
switch paths: the dealing of interface-band cells, steep fields, spikes and
spacings at the ends of the FP32 range, the FP32 operators' error, the FP64
weights outside their fast range, the default tiles and the autotuner's
candidates, the CFL maxima shared by a run's steps, the Airy generator at its
limits, rejected launches, and pageable copies."""
import numpy as np
import pytest

import reef3d_b200 as r3d
from test_gpu_parity import relmax
from test_oracle_golden import interior, visible_mask

pytestmark = pytest.mark.gpu

FLAGS = dict(f43=0.5, f44=2, f45=2.1, f49=1, n47=0.125)
EPS32 = 2.0 ** -24


def instance(dims, precision=r3d.FP32, nodes=None, **kw):
    return r3d.LevelSet(*dims, *(nodes or ()), precision=precision, **dict(FLAGS, **kw))


def dense(ls):
    return ls.download(r3d.PHI, r3d.LAYOUT_DENSE)


@pytest.mark.parametrize("f49", [1, 0])
@pytest.mark.parametrize("cfg", [0, 1, 6])
@pytest.mark.parametrize("cells", [1, 3, 5, 6, 10, 11, 15, 16, 20, 21, 32, 64])
def test_band_cells_dealt_to_lanes(cells, cfg, f49):
    """A sheet that crosses `cells` cells of every row of 64: a warp of a 64 x 8
    tile with one row a thread (configuration 0) holds `cells` band cells of a
    plane, with two rows (1) twice as many, and of a 32 x 16 tile with two rows
    (6) up to four times as many.  They are dealt out in rounds of ten cells up
    to twenty, of 32 beyond.  The tiled kernels against the one-cell-per-thread
    ones.  Both form the band in FP64, so a cell differs by the rounding of the
    other cells' FP32 right-hand sides: two pseudo-steps of dtau <= h, RHS
    errors of a few ulp of 1."""
    n = 64
    x = (np.arange(n) + 0.5) / n
    rng = np.random.default_rng(cells)
    phi = np.broadcast_to(x[:, None, None] - 0.5, (n, n, n)).copy()
    # the sheet lies on a plane z = const over `cells` columns, elsewhere above
    phi[:, :, cells:] += 4.0 / n
    phi += 1e-3 / n * rng.standard_normal(phi.shape)
    out = []
    for tiled in (1, 0):
        with instance((n, n, n), f49=f49) as ls:
            ls.set_option(r3d.OPT_TILED, tiled)
            ls.set_option(r3d.OPT_TILE_CFG, cfg)
            ls.upload(r3d.PHI, phi, r3d.LAYOUT_DENSE)
            ls.ghost_fill()
            ls.reinit(1)
            ls.sync()
            out.append(dense(ls))
    h = 1.0 / n
    assert np.max(np.abs(out[0] - out[1])) <= 3 * h * 64 * EPS32 + 2 * EPS32


@pytest.mark.parametrize("scale", [1.0, 1e2, 1e4, 1e7])
@pytest.mark.parametrize("tiled", [1, 0])
def test_steep_fields_fp32(scale, tiled):
    """Gradients up to 1e7, jumps included: the FP32 operator against FP64's on
    the same FP32 values, relative to its largest value.  An axis's derivative
    is off by some 8 roundings of the largest difference in its stencil, of
    which the derivative itself, from the smooth side, may be a small part."""
    n = 32
    rng = np.random.default_rng(3)
    res = []
    x = (np.arange(n) + 0.5) / n
    phi = np.sin(5 * x)[None, None, :] * np.cos(4 * x)[None, :, None] + 0.5 * np.sin(6 * x)[:, None, None]
    phi = scale * (phi + 0.3 * np.sign(phi) + 0.01 * rng.standard_normal(phi.shape))
    phi = phi.astype(np.float32).astype(np.float64)
    for prec in (r3d.FP64, r3d.FP32):
        with instance((n, n, n), prec) as ls:
            if prec == r3d.FP32:
                ls.set_option(r3d.OPT_TILED, tiled)
            ls.init_spheres_tg([(0.5, 0.5, 0.5, 0.2)], [(1, 0.5), (2, 0.25)])
            ls.upload(r3d.PHI, phi, r3d.LAYOUT_DENSE)
            ls.ghost_fill()
            ls.set_dt(1e4)  # phi + dt L is dt L
            ls.stage(r3d.STAGE_CONVECTION, 1)
            ls.sync()
            res.append(ls.download(r3d.WORK1, r3d.LAYOUT_DENSE))
    assert np.all(np.isfinite(res[1]))
    assert relmax(res[1], res[0]) <= 64 * EPS32


@pytest.mark.parametrize("spike", [10.0, 1e3, 1e6, 1e9, 1e12, 1e16])
@pytest.mark.parametrize("kind", [r3d.STAGE_CONVECTION, r3d.STAGE_REINIT])
@pytest.mark.parametrize("f49", [1, 0])
def test_spikes_fp32(spike, kind, f49):
    """Isolated values far above the rest, up to the ends of the packed form's
    range: finite, and FP64's to the rounding of the largest value within three
    cells."""
    from scipy.ndimage import maximum_filter
    if kind == r3d.STAGE_REINIT and spike > 1e12:
        pytest.skip("gradients beyond the squares' range")
    n = 40
    rng = np.random.default_rng(7)
    x = (np.arange(n) + 0.5) / n
    phi = (x[:, None, None] - 0.45) + 0.2 * np.sin(5 * x)[None, :, None] * np.cos(4 * x)[None, None, :]
    at = rng.integers(0, n, (40, 3))
    at[:4] = [[0, 0, 0], [n - 1, n - 1, n - 1], [20, 0, n - 1], [n - 1, 7, 0]]
    for k, j, i in at:
        phi[k, j, i] = spike * rng.uniform(-1.0, 1.0)
    phi = phi.astype(np.float32).astype(np.float64)
    out = []
    for prec in (r3d.FP64, r3d.FP32):
        with instance((n, n, n), prec, f49=f49) as ls:
            ls.init_spheres_tg([(0.5, 0.5, 0.5, 0.2)], [(1, 0.5), (2, 0.25)])
            ls.upload(r3d.PHI, phi, r3d.LAYOUT_DENSE)
            ls.ghost_fill()
            ls.set_dt(1.0 / n)
            ls.stage(kind, 1)
            ls.sync()
            out.append(ls.download(r3d.WORK1, r3d.LAYOUT_DENSE))
    assert np.all(np.isfinite(out[1]))
    # a derivative times h is at most 4 differences of values within three cells,
    # three axes of them times a velocity (pseudo-step) of at most h a step
    size = maximum_filter(np.abs(phi), size=7, mode="nearest")
    assert np.all(np.abs(out[1] - out[0]) <= 16 * EPS32 * (size + 1.0))


@pytest.mark.parametrize("dims", [(32, 32, 32), (32, 1, 32)])
@pytest.mark.parametrize("e", [-56, -50, -44, -40, -30, 0, 40, 46, 52, 56, 60, 64])
def test_spacings_fp32(e, dims):
    """Boxes of 2^e a side, flat parts included: the kernels square h, and leave
    the tiles, then the undivided differences, where that leaves the FP32
    range.  Scaling by a power of two changes nothing else: FP64's convection
    to eight roundings of the values."""
    s = 2.0 ** e
    x = (np.arange(32) + 0.5) / 32
    phi = np.sin(5 * x)[None, None, :] * np.cos(4 * x[:dims[1]])[None, :, None] + 0.5 * np.sin(6 * x)[:, None, None]
    phi[:, :, :8] = 0.25
    phi = phi.astype(np.float32).astype(np.float64)
    nodes = [r3d.uniform_nodes(n, s if n > 1 else s / 32) for n in dims]
    out = []
    for prec in (r3d.FP64, r3d.FP32):
        with instance(dims, prec, nodes) as ls:
            for f in (r3d.U, r3d.V, r3d.W):
                ls.upload(f, np.full(ls.reef3d_shape, 0.5))
            ls.upload(r3d.PHI, phi * s, r3d.LAYOUT_DENSE)
            ls.ghost_fill()
            ls.set_dt(s / 64)
            ls.stage(r3d.STAGE_CONVECTION, 1)
            ls.sync()
            out.append(ls.download(r3d.WORK1, r3d.LAYOUT_DENSE) / s)
    assert np.max(np.abs(out[1] - out[0])) <= 8 * EPS32


@pytest.mark.parametrize("dims,stretch,tiled,roundings", [
    ((128, 1, 128), 0.0, 1, 9), ((301, 1, 157), 0.0, 1, 9), ((97, 61, 120), 0.0, 0, 9), ((50, 111, 83), 0.0, 1, 9),
    ((413, 1, 211), 0.3, 1, 13), ((96, 80, 112), 0.3, 1, 13)])
def test_convection_error_fp32(dims, stretch, tiled, roundings):
    """The FP32 convection operator against FP64's on the same (FP32) values, by
    its 2-norm: the roundings on the way of a value's leading part (difference,
    the reconstruction's sums, 1/h, three of the velocity and its product, the
    axes' sum: up to 9; the quotient, its reciprocal's and two of the tables
    more: 13), each 0.42 2^-24 rms for mantissas spread over a binade, added in
    quadrature.  Weights add nothing of that order: they multiply differences of
    reconstructions."""
    rng = np.random.default_rng(dims[0])
    nodes = []
    for n in dims:
        length = 1.0 if n > 1 else 1.0 / dims[0]
        x = r3d.uniform_nodes(n, length)
        nodes.append(x + (stretch * np.sin(2 * np.pi * x / length) * length / (2 * np.pi) if n > 1 else 0.0))
    spheres = [(*map(float, rng.uniform(0.2, 0.8, 3)), float(rng.uniform(0.05, 0.2))) for _ in range(4)]
    modes = [(int(rng.integers(1, 4)), float(rng.normal(0.0, 0.5))) for _ in range(4)]
    with instance(dims, r3d.FP64, nodes) as ls:
        ls.init_spheres_tg(spheres, modes)
        ls.run(10)
        fields = {f: ls.download(f).astype(np.float32).astype(np.float64) for f in (r3d.PHI, r3d.U, r3d.V, r3d.W)}
    out = []
    for prec in (r3d.FP64, r3d.FP32):
        with instance(dims, prec, nodes) as ls:
            if prec == r3d.FP32:
                ls.set_option(r3d.OPT_TILED, tiled)
            for f, a in fields.items():
                ls.upload(f, a)
            ls.ghost_fill()
            ls.set_dt(1e4)  # phi + dt L is dt L
            ls.stage(r3d.STAGE_CONVECTION, 1)
            ls.sync()
            out.append(ls.download(r3d.WORK1, r3d.LAYOUT_DENSE))
    err = np.linalg.norm(out[1] - out[0]) / np.linalg.norm(out[0])
    assert err <= 0.42 * EPS32 * np.sqrt(roundings)


@pytest.mark.parametrize("scale", [1.0, 1e20, 1e34, 1e35, 1e36, 1e70, 1e80])
def test_fp64_weights_range(port_lib, scale):
    """The FP64 operators bit for bit where the squared indicators pass 2^499
    (weights_any) and where they do not, mixed in one field."""
    nx, ny, nz = 20, 11, 14
    rng = np.random.default_rng(5)
    xn, yn, zn = (r3d.uniform_nodes(n) for n in (nx, ny, nz))
    phi = rng.standard_normal((nx + 6, ny + 6, nz + 6))
    phi[: nx // 2] *= scale
    u, v, w = (rng.standard_normal(phi.shape) for _ in range(3))
    o = port_lib(nx, ny, nz, xn, yn, zn, **FLAGS)
    with instance((nx, ny, nz), r3d.FP64, (xn, yn, zn)) as ls:
        for f, a in ((r3d.PHI, phi), (r3d.U, u), (r3d.V, v), (r3d.W, w)):
            ls.upload(f, a)
        ls.convection_L()
        got = ls.download(r3d.L)
        ls.reinidisc_L()
        got_r = ls.download(r3d.L)
    for mine, ref in ((got, o.weno_L(phi, u, v, w)), (got_r, o.reinidisc_L(phi))):
        assert np.array_equal(interior(mine, nx, ny, nz), interior(ref, nx, ny, nz), equal_nan=True)


@pytest.mark.parametrize("dims", [(2, 2, 2), (33, 17, 5), (64, 8, 1), (65, 9, 40), (96, 96, 96)])
def test_default_tiles(dims):
    """The size-dependent default gives the level set of any other choice."""
    out = []
    for pick in (None, (1, 10), (0, 16)):
        with instance(dims) as ls:
            ls.init_spheres_tg([(0.5, 0.4, 0.6, 0.2), (0.3, 0.6, 0.3, 0.1)], [(1, 0.5), (2, -0.3)])
            assert ls.get_option(r3d.OPT_TILED) == 1 and ls.get_option(r3d.OPT_CHUNK) >= 1
            if pick:
                ls.set_option(r3d.OPT_TILE_CFG, pick[0])
                ls.set_option(r3d.OPT_CHUNK, pick[1])
            ls.run(2)
            ls.sync()
            out.append(dense(ls))
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])


@pytest.mark.parametrize("dims", [(47, 45, 43), (161, 133, 119), (255, 130, 131)])
def test_autotune_sweep_size(dims):
    """A sweep launches 24 stages for each of at most 7 z chunks of a
    configuration and for the default, and times the three best of a kind three
    times again (22 launches each), whatever the grid's size; the choice comes
    from the candidates or is the default."""
    chunks = set(r3d.tile_chunks())
    with instance(dims) as ls:
        ls.init_spheres_tg([(0.5, 0.5, 0.5, 0.25)], [(1, 0.5), (2, 0.3)])
        default = ls.get_option(r3d.OPT_CHUNK), ls.get_option(r3d.OPT_CHUNK_REINIT)
        before = ls.launch_count()
        ls.autotune()
        most = 2 * 12 * (7 * len(r3d.tile_configs()) + 1) + 2 * 3 * 3 * 22 + 8
        assert 0 < ls.launch_count() - before <= most
        for option, first in zip((r3d.OPT_CHUNK, r3d.OPT_CHUNK_REINIT), default):
            kc = ls.get_option(option)
            assert kc == first or (kc in chunks and first < 2 * kc and kc <= 4 * first)


@pytest.mark.parametrize("dims", [(33, 17, 5), (64, 40, 24), (96, 96, 96)])
def test_instance_and_batch_defaults(dims):
    """An instance alone and a batch's member start with different tiles and
    chunks: the same level set, volume sums in another order (of at most
    dims cells, each half an ulp)."""
    out = []
    for batched in (False, True):
        with instance(dims) as ls:
            ls.init_spheres_tg([(0.5, 0.4, 0.6, 0.2), (0.3, 0.6, 0.3, 0.1)], [(1, 0.5), (2, -0.3)])
            if batched:
                with r3d.Batch() as b:
                    b.add(ls)
                    b.step(3)
                    b.sync()
                    out.append((dense(ls), ls.last_volume()))
            else:
                ls.run(3)
                ls.sync()
                out.append((dense(ls), ls.last_volume()))
    assert np.array_equal(out[0][0], out[1][0])
    for x, y in zip(out[0][1], out[1][1]):
        assert abs(x - y) <= 2.0 ** -53 * np.prod(dims) * abs(y)


@pytest.mark.parametrize("precision", [r3d.FP32, r3d.FP64])
@pytest.mark.parametrize("dims", [(40, 24, 18), (48, 1, 37)])
@pytest.mark.parametrize("airy", [False, True])
def test_run_shares_cfl_maxima(precision, dims, airy):
    """An adaptive run's time steps are those of single steps with r3d_cfl_dt
    before each, for stored velocities (scaled by the clock), the Airy
    generator (beside an uploaded v), and velocities uploaded between runs."""
    def make():
        ls = instance(dims, precision)
        ls.init_spheres_tg([(0.5, 0.5, 0.5, 0.25)], [(1, 0.5), (2, 0.3)])
        if airy:
            ls.set_time(0.0)
            ls.set_velocity_airy(0.05, 2.0, 0.5)
            ls.upload(r3d.V, np.full(ls.reef3d_shape, 0.01))
        else:
            ls.set_velocity_period(1.0)
            ls.set_time(0.1)
        return ls
    shape = (dims[0] + 6, dims[1] + 6, dims[2] + 6)
    faster = np.random.default_rng(1).standard_normal(shape)
    a, b = make(), make()
    try:
        for field in (None, r3d.W, r3d.U):
            for ls in (a, b):
                if field is not None and not airy:
                    ls.upload(field, 3.0 * faster)
            a.run(3)
            for _ in range(3):
                b.step(b.cfl_dt())
            assert a.time() == b.time()
            assert np.array_equal(dense(a), dense(b))
    finally:
        a.close()
        b.close()


@pytest.mark.parametrize("nz", [11, 12, 24, 61, 128])
@pytest.mark.parametrize("precision", [r3d.FP64, r3d.FP32])
def test_pageable_copies(nz, precision):
    """Copies between pageable host arrays of 4 to 47 MB and the device against
    the same fields through a pinned array, in both layouts."""
    import torch
    nx, ny = 220, 208
    a = np.random.default_rng(nz).standard_normal((nz, ny, nx)).astype(np.float32).astype(np.float64)
    pin = torch.empty(a.shape, dtype=torch.float64, pin_memory=True)
    with instance((nx, ny, nz), precision) as ls:
        ls.upload(r3d.PHI, a, r3d.LAYOUT_DENSE)
        ls.download_ptr(r3d.PHI, pin.data_ptr(), r3d.LAYOUT_DENSE)
        assert np.array_equal(pin.numpy(), a)
        pin *= 2.0
        ls.upload_ptr(r3d.PHI, pin.data_ptr(), r3d.LAYOUT_DENSE)
        assert np.array_equal(dense(ls), 2.0 * a)
        r = np.random.default_rng(1).standard_normal(ls.reef3d_shape).astype(np.float32).astype(np.float64)
        ls.upload(r3d.U, r)
        m = visible_mask(nx, ny, nz)
        got = ls.download(r3d.U)
        assert np.array_equal(got[m], r[m]) and not np.any(got[~m])


def airy_flume(nx, nz, precision):
    """A thin flume of nx x nz cells, its depth half the height, with a sheet
    at the still water and the Airy generator on."""
    nodes = (r3d.uniform_nodes(nx, nx / nz), r3d.uniform_nodes(1, 1.0 / nz), r3d.uniform_nodes(nz))
    ls = instance((nx, 1, nz), precision, nodes)
    z = (np.arange(nz) + 0.5) / nz
    ls.upload(r3d.PHI, np.broadcast_to(0.5 - z[:, None, None], (nz, 1, nx)).copy(), r3d.LAYOUT_DENSE)
    ls.ghost_fill()
    ls.set_time(0.0)
    ls.set_velocity_airy(0.05, 2.0, 0.5)
    return ls


@pytest.mark.parametrize("precision", [r3d.FP32, r3d.FP64])
@pytest.mark.parametrize("edge", [3052, 3053, 3060, 3061, 14508, 14509, 14516])
def test_airy_run_at_the_shared_memory_limits(edge, precision):
    """Adaptive runs of the Airy generator where its tables, 16 (nx + nz + 12)
    bytes, reach the 48 KB that need no opt-in and the 227 KB of a block: one
    step (launched) and three (replayed from a graph) are single steps with
    r3d_cfl_dt before each."""
    nz = 56
    a, b = airy_flume(edge - nz, nz, precision), airy_flume(edge - nz, nz, precision)
    try:
        for steps in (1, 3):
            a.run(steps, adaptive=True)
            for _ in range(steps):
                b.step(b.cfl_dt())
            assert a.time() == b.time() > 0.0
            assert np.array_equal(dense(a), dense(b))
    finally:
        a.close()
        b.close()


def test_airy_refused_beyond_shared_memory():
    """One cell more than the tables' limit is refused when the generator is
    set."""
    with pytest.raises(r3d.R3DError):
        airy_flume(14517 - 56, 56, r3d.FP32).close()


def test_airy_instances_leave_each_other_their_shared_memory():
    """A shorter flume set up later does not lower what a longer one's launches
    may take."""
    long, short = airy_flume(6000, 56, r3d.FP32), airy_flume(3100, 56, r3d.FP32)
    try:
        for ls in (long, short):
            ls.run(1, adaptive=True)
            ls.sync()
    finally:
        long.close()
        short.close()


@pytest.mark.parametrize("call", ["step", "run1", "run3"])
@pytest.mark.parametrize("airy", [False, True])
def test_rejected_launch_leaves_the_level_set(call, airy):
    """A step whose first launch the runtime refuses fails before a stage runs
    and leaves no graph behind that lacks the launch: the next run is a fresh
    instance's."""
    def make():
        ls = instance((40, 24, 18))
        ls.init_spheres_tg([(0.5, 0.5, 0.5, 0.25)], [(1, 0.5), (2, 0.3)])
        if airy:
            ls.set_time(0.0)
            ls.set_velocity_airy(0.05, 2.0, 0.5)
        return ls
    a, b = make(), make()
    try:
        before = dense(a)
        dt = a.cfl_dt()
        a.set_option(r3d.OPT_LAUNCH_TEST, 1)
        with pytest.raises(r3d.R3DError):
            a.step(dt) if call == "step" else a.run(int(call[3:]), adaptive=True)
        a.sync()
        assert a.get_option(r3d.OPT_LAUNCH_TEST) == 0
        assert np.array_equal(dense(a), before) and a.time() == 0.0
        for ls in (a, b):
            ls.run(3, adaptive=True)
            ls.sync()
        assert a.time() == b.time() and np.array_equal(dense(a), dense(b))
    finally:
        a.close()
        b.close()
