"""The mutual sweep (each pair evaluated once, added to both particles) at the
sizes where its tiling, its centre-column rules and its slab ranges change,
against the FP64 oracle: RMS fractional error <= 2e-6, max <= 1e-4 (the bounds
of the other GPU tests), and against itself bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RMS, MAX = 2e-6, 1e-4


def _box(synth, cpd, counts, seed=0):
    """Uniform positions inside cells of the given occupancies."""
    rng = np.random.default_rng(seed)
    cs = np.zeros(cpd ** 3 + 1, np.int64)
    cs[1:] = np.cumsum(np.asarray(counts).ravel())
    h = 1.0 / cpd
    p = ((rng.random((3, int(cs[-1])), dtype=np.float32) - np.float32(0.5)) * np.float32(0.999 * h))
    return synth.Box(cpd=cpd, x=p[0].copy(), y=p[1].copy(), z=p[2].copy(), cell_start=cs)


def _check(oracle, box, soft, eps, a, R=2, step=1, first=0):
    sinks = np.arange(first, first + len(a), step)
    rms, mx, _ = oracle.frac_errors(a[::step, :3], oracle.fp64_sinks(box, soft, eps, sinks, R=R))
    assert rms <= RMS and mx <= MAX, (rms, mx)


# sinks of the pencils around the filled column: below, at and above every tile size
@pytest.mark.parametrize("n", [1, 31, 32, 33, 64, 65, 96, 97, 128, 129, 160, 192, 193, 256, 257, 300])
@pytest.mark.parametrize("soft", [0, 1, 2, 3])
def test_tile_edges(capi, oracle, synth, n, soft):
    cpd = 7
    counts = np.zeros((cpd, cpd, cpd), int)
    counts[3, 3, 3] = n - n // 2       # pencil (3, 3, 3) holds n sinks
    counts[3, 3, 4] = n // 2
    counts[3, 4, 3] = counts[4, 2, 3] = counts[5, 3, 5] = 1 + n % 37
    counts[0, 0, 0] = counts[6, 6, 6] = counts[1, 6, 5] = 33  # neighbours across the faces
    box = _box(synth, cpd, counts, seed=n)
    length = 0.3 / cpd / max(2, n) ** (1 / 3)
    eps = synth.kernel_eps(soft, length)
    shapes = range(capi.lib().nf_kernel_variant_count()) if soft < 2 else [0]
    for v in shapes:
        with capi.Context(softening=soft, eps=eps, kernel_variant=v) as ctx:
            db = ctx.box(box)
            a = db.forces()
            t = ctx.last_timing()
            db.close()
        assert t.pairs == oracle.pair_count(box)
        _check(oracle, box, soft, eps, a)


# occupancies around the one at which a cell meets its column mutually (192)
@pytest.mark.parametrize("own,near,far", [(191, 191, 191), (192, 10, 10), (10, 192, 10),
                                          (10, 10, 193), (400, 192, 191), (1000, 0, 300),
                                          (256, 256, 256)])
@pytest.mark.parametrize("cpd", [5, 7])
def test_dense_columns(capi, oracle, synth, own, near, far, cpd):
    counts = np.zeros((cpd, cpd, cpd), int)
    counts[2, 2, 0], counts[2, 2, 1], counts[2, 2, 2] = own, near, far   # and across z = 0
    counts[2, 2, cpd - 1] = near // 2
    counts[2, 3, 0] = 50
    box = _box(synth, cpd, counts, seed=own + near)
    eps = synth.kernel_eps(1, 0.02 / cpd)
    b2 = float(np.float32((0.2 / cpd) ** 2))
    with capi.Context(softening=1, eps=eps) as ctx:
        db = ctx.box(box)
        a = db.forces()
        db.close()
    with capi.Context(softening=1, eps=eps, b2=b2) as ctx:
        db = ctx.box(box)
        d = db.forces()
        db.close()
    sinks = np.arange(box.n)
    for r in (a, d):
        _check(oracle, box, 1, eps, r)
    # a sum of positive terms in FP32 over at most `box.n` of them: 1e-5
    np.testing.assert_allclose(d[:, 3], oracle.fp64_density(box, b2, sinks), rtol=1e-5,
                               atol=1e-6 * b2)


@pytest.mark.parametrize("R", [1, 2])
def test_slab_ranges(capi, oracle, synth, R):
    """Ranges of every length, at the periodic faces too: columns outside the
    range are met one-sided."""
    box = synth.clustered_box(9000, 7, seed=71, n_clumps=8)
    eps = synth.kernel_eps(0, synth.plummer_eps(21))
    with capi.Context(softening=0, eps=eps, near_field_radius=R) as ctx:
        db = ctx.box(box)
        for lo in range(box.cpd):
            for hi in range(lo + 1, box.cpd + 1):
                p0, p1 = db.slab_particles(lo, hi)
                a = db.forces(lo, hi)
                assert ctx.last_timing().pairs == db.pair_count(lo, hi)
                _check(oracle, box, 0, eps, a, R=R, step=5, first=p0)
        db.close()


def test_softening_below_the_fixed_point_range(capi, oracle, synth):
    """A softening so small that fixed point would not resolve ordinary pairs
    takes the one-sided sweep: the results are as good.  2e-4 and 3e-6 lie on
    either side of the limit of this box for every softening (a pencil meets at
    least 2000 sources: see nf_last_engine in the header)."""
    box = synth.uniform_box(6000, 7, seed=72)
    for soft in (0, 1, 2, 3):
        for length, want in ((2e-4, capi.ENGINE_MUTUAL), (3e-6, capi.ENGINE_ONE_SIDED),
                             (4e-7, capi.ENGINE_ONE_SIDED)):
            eps = synth.kernel_eps(soft, length)
            with capi.Context(softening=soft, eps=eps) as ctx:
                db = ctx.box(box)
                a = db.forces()
                assert ctx.last_engine() == want
                db.close()
            _check(oracle, box, soft, eps, a, step=3)


def test_non_finite_positions_reach_their_neighbours(capi, synth):
    """A NaN position makes the records of all particles that meet it NaN, as
    one-sided sums would, and leaves the others."""
    box = synth.uniform_box(8000, 9, seed=73)
    bad = box.n // 2
    x = box.x.copy()
    x[bad] = np.nan
    cell = np.searchsorted(box.cell_start, np.arange(box.n), side="right") - 1
    c = np.stack(np.unravel_index(cell, (9, 9, 9)))
    d = np.abs(c - c[:, bad:bad + 1])
    meets = (np.minimum(d, 9 - d) <= 2).all(0)
    eps = synth.kernel_eps(1, synth.plummer_eps(20))
    with capi.Context(softening=1, eps=eps) as ctx:
        db = ctx.box(box)
        want = db.forces()
        db.update(x, box.y, box.z)
        a = db.forces()
        db.close()
    assert np.isnan(a[meets, :3]).all()
    np.testing.assert_allclose(a[~meets], want[~meets], rtol=0, atol=1e-6 * np.abs(want).max())


def test_bits_do_not_depend_on_the_order_of_the_work(capi, synth):
    """The same range from a new box and a new context: the same bits, although
    the work list's order and the order of the additions are not fixed."""
    box = synth.clustered_box(60000, 13, seed=74, n_clumps=20)
    eps = synth.kernel_eps(1, synth.plummer_eps(39))
    outs = []
    for _ in range(3):
        with capi.Context(softening=1, eps=eps, kernel_variant=0) as ctx:
            for _ in range(2):
                db = ctx.box(box)
                outs.append((db.forces(), db.forces(2, 9)))
                db.close()
    for o in outs[1:]:
        for x, y in zip(o, outs[0]):
            assert np.array_equal(x.view(np.uint32), y.view(np.uint32))


@pytest.mark.parametrize("soft,R,counts", [
    (0, 2, "one"), (1, 2, "edges"), (1, 2, "dense"), (2, 1, "edges"), (3, 2, "edges"), (0, 1, "dense")])
def test_allocation_free_sweep(capi, oracle, synth, soft, R, counts):
    """nf_forces_noalloc cuts few pencils into pieces: one particle, pencils
    around the tile sizes, a dense cell, whole boxes and slab ranges."""
    import ctypes

    import torch
    cpd = 7
    c = np.zeros((cpd, cpd, cpd), int)
    if counts == "one":
        c[2, 3, 4] = 1
    elif counts == "edges":
        c[:] = np.arange(cpd ** 3).reshape(c.shape) % 41
        c[3, 3, :3] = 129, 64, 0
    else:
        c[3, 3, 3], c[3, 3, 4], c[4, 3, 3] = 700, 200, 33
    box = _box(synth, cpd, c, seed=5)
    eps = synth.kernel_eps(soft, 0.02 / cpd)
    cfg = capi.default_config(softening=soft, eps=eps, near_field_radius=R)
    pos = torch.zeros((box.n, 4), device="cuda")
    for k, v in enumerate((box.x, box.y, box.z)):
        pos[:, k] = torch.from_numpy(v).cuda()
    cs = torch.from_numpy(box.cell_start).cuda()
    for lo, hi in ((0, cpd), (2, 5), (3, 4), (6, 7)):
        p0, p1 = int(box.cell_start[lo * cpd * cpd]), int(box.cell_start[hi * cpd * cpd])
        out = torch.full((max(p1 - p0, 1), 4), float("nan"), device="cuda")
        capi.check(capi.lib().nf_forces_noalloc(
            ctypes.byref(cfg), cpd, pos.data_ptr(), cs.data_ptr(), lo, hi, out.data_ptr(),
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        if p1 == p0:
            continue
        a = out[:p1 - p0].cpu().numpy()
        if counts == "one":
            assert np.all(a == 0)
        else:
            _check(oracle, box, soft, eps, a, R=R, first=p0)
