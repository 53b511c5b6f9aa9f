"""Both engines by name: which one a call takes, and the one-sided engine's
results where the mutual one does not apply (plain accumulation, softenings
below its fixed-point range), for every entry point, against the FP64 oracle.
RMS fractional error <= 2e-6, max <= 1e-4, as in the other GPU tests."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RMS, MAX = 2e-6, 1e-4
SMALL = 2e-5  # softening length, cells: below the fixed-point range of these boxes


def _check(oracle, box, soft, eps, a, R=2, sinks=None):
    sinks = np.arange(box.n) if sinks is None else sinks
    rms, mx, _ = oracle.frac_errors(a[sinks, :3], oracle.fp64_sinks(box, soft, eps, sinks, R=R))
    assert rms <= RMS and mx <= MAX, (rms, mx)


def test_engine_of_a_sweep(capi, synth):
    """Ordinary softenings take the mutual engine; plain accumulation and tiny
    softenings the one-sided one; nothing has run at first."""
    box = synth.uniform_box(4000, 7, seed=1)
    for soft in range(4):
        for acc, cells, want in ((capi.ACC_COMPENSATED, 0.02, capi.ENGINE_MUTUAL),
                                 (capi.ACC_PLAIN, 0.02, capi.ENGINE_ONE_SIDED),
                                 (capi.ACC_COMPENSATED, SMALL, capi.ENGINE_ONE_SIDED)):
            eps = synth.kernel_eps(soft, cells / 7)
            with capi.Context(softening=soft, eps=eps, accumulation=acc) as ctx:
                with pytest.raises(capi.NfError) as e:
                    ctx.last_engine()
                assert e.value.status == capi.NF_ENOTREADY
                db = ctx.box(box)
                for _ in range(3):  # launched, captured, replayed
                    db.forces()
                    assert ctx.last_engine() == want
                db.forces(2, 3)
                assert ctx.last_engine() == want
                out = np.empty((box.n, 4), np.float32)
                db.step(box.x, box.y, box.z, out)
                assert ctx.last_engine() == want
                db.close()


@pytest.mark.parametrize("soft", [0, 1])
def test_shapes_of_the_one_sided_engine(capi, oracle, synth, soft):
    """Every shape runs where it is asked for, and gives the same results to
    rounding; left to itself the tuner times those of the engine that runs."""
    box = synth.clustered_box(30000, 11, seed=3, n_clumps=25)
    eps = synth.kernel_eps(soft, synth.plummer_eps(31))
    L = capi.lib()
    n = L.nf_kernel_variant_count()
    names = {L.nf_engine_variant_name(e, v) for e in (0, 1) for v in range(n)}
    assert len(names) == 2 * n
    outs, padded = [], []
    for v in range(n):
        with capi.Context(softening=soft, eps=eps, kernel_variant=v, accumulation=capi.ACC_PLAIN) as ctx:
            db = ctx.box(box)
            outs.append(db.forces())
            t = ctx.last_timing()
            assert ctx.last_engine() == capi.ENGINE_ONE_SIDED and t.variant == v
            padded.append(t.padded_pairs)
            db.close()
    assert len(set(padded)) >= 3  # tiles of 64, 128 and 256 sinks pad differently
    for o in outs[1:]:
        np.testing.assert_allclose(o, outs[0], rtol=0, atol=2e-6 * np.abs(outs[0]).max())
    _check(oracle, box, soft, eps, outs[2], sinks=np.arange(0, box.n, 7))
    with capi.Context(softening=soft, eps=eps, accumulation=capi.ACC_PLAIN) as ctx:
        db = ctx.box(box)
        db.forces()
        v, ms = db.tuning()
        assert ctx.last_timing().variant == v and all(m > 0 for m in ms) and ms[v] == min(ms)
        db.close()


def test_tuning_is_by_engine(capi, synth):
    """A box that changes engine is tuned for each; a later box takes over the
    choice of the engine it runs on, and no other."""
    box = synth.clustered_box(30000, 11, seed=4, n_clumps=25)
    eps, tiny = (synth.kernel_eps(0, c / 11) for c in (0.02, SMALL))
    with capi.Context(softening=0, eps=eps) as ctx:
        a = ctx.box(box)
        a.set_eps(tiny)
        a.forces()
        assert ctx.last_engine() == capi.ENGINE_ONE_SIDED
        one = a.tuning()
        a.set_eps(0.0)
        a.forces()
        assert ctx.last_engine() == capi.ENGINE_MUTUAL
        both = a.tuning()
        assert all(m > 0 for m in both[1]) and both[1] != one[1]
        a.close()
        b = ctx.box(box)
        b.forces()
        assert b.tuning() == both
        b.set_eps(tiny)
        b.forces()
        assert b.tuning() == one
        b.close()


@pytest.mark.parametrize("kw", [dict(softening=2), dict(softening=3), dict(softening=1, b2=1e-4)])
def test_one_shape_is_not_tuned(capi, synth, kw):
    """Kernels with one shape run it, whatever is asked for, and time nothing."""
    box = synth.uniform_box(6000, 7, seed=5)
    eps = synth.kernel_eps(kw["softening"], 0.02 / 7)
    outs = []
    for acc in (capi.ACC_COMPENSATED, capi.ACC_PLAIN):
        for v in (-1, 0, 2, 4):
            with capi.Context(eps=eps, accumulation=acc, kernel_variant=v, **kw) as ctx:
                db = ctx.box(box)
                outs.append(db.forces())
                assert ctx.last_timing().variant == 0
                assert not any(db.tuning()[1])
                db.close()
    for o in outs:
        np.testing.assert_allclose(o, outs[0], rtol=0, atol=2e-6 * np.abs(outs[0]).max())


def _engine_of(capi, drv):
    e = ctypes.c_int(-1)
    capi.check(capi.lib().nf_last_engine(capi.lib().nf_driver_context(drv.h), ctypes.byref(e)))
    return e.value


@pytest.mark.parametrize("pinned", [0, 1])
@pytest.mark.parametrize("nodes", [[None], [(11, 5), (3, 8)]])
@pytest.mark.parametrize("soft,plain", [(0, 1), (1, 1), (2, 1), (3, 1), (0, 0), (1, 0), (2, 0), (3, 0)])
def test_drop_in_on_the_one_sided_engine(capi, oracle, synth, soft, plain, nodes, pinned):
    """SICs that the mutual engine's lists do not serve: plain accumulation, and
    compensated with a tiny softening; whole domain and a 2D split whose nodes
    lie across z = 0, buffers pinned and not."""
    box = synth.clustered_box(20000, 13, seed=6, n_clumps=15)
    length = synth.plummer_eps(27) if plain else SMALL / 13
    acc = capi.ACC_PLAIN if plain else capi.ACC_COMPENSATED
    a = np.zeros((box.n, 4), np.float32)
    for node in nodes:
        drv = capi.Driver(box, softening=soft, softening_length=length, direct_bpd=2, node_z=node,
                          accumulation=acc, use_pinned=pinned)
        try:
            got = drv.run_all()
            assert _engine_of(capi, drv) == capi.ENGINE_ONE_SIDED
            m = drv.slabs.mask if node else np.ones(box.n, bool)
        finally:
            drv.close()
        a[m] = got[m]
    _check(oracle, box, soft, synth.kernel_eps(soft, length), a, sinks=np.arange(0, box.n, 9))


@pytest.mark.parametrize("soft", [0, 1, 2, 3])
@pytest.mark.parametrize("dens", [False, True])
def test_allocation_free_call_on_the_one_sided_engine(capi, oracle, synth, soft, dens):
    """nf_forces_noalloc with plain accumulation, and with a tiny softening:
    whole boxes and slab ranges, with and without the density channel."""
    import torch
    box = synth.clustered_box(15000, 9, seed=7, n_clumps=10)
    b2 = float(np.float32((0.2 / box.cpd) ** 2)) if dens else 0.0
    pos = torch.zeros((box.n, 4), device="cuda")
    for k, v in enumerate((box.x, box.y, box.z)):
        pos[:, k] = torch.from_numpy(v).cuda()
    cs = torch.from_numpy(box.cell_start).cuda()
    c2 = box.cpd ** 2
    for acc, cells in ((capi.ACC_PLAIN, 0.02), (capi.ACC_COMPENSATED, SMALL)):
        eps = synth.kernel_eps(soft, cells / box.cpd)
        cfg = capi.default_config(softening=soft, eps=eps, b2=b2, accumulation=acc)
        for lo, hi in ((0, box.cpd), (4, 6)):
            p0, p1 = int(box.cell_start[lo * c2]), int(box.cell_start[hi * c2])
            out = torch.full((p1 - p0, 4), float("nan"), device="cuda")
            capi.check(capi.lib().nf_forces_noalloc(
                ctypes.byref(cfg), box.cpd, pos.data_ptr(), cs.data_ptr(), lo, hi, out.data_ptr(),
                ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
            a = out.cpu().numpy()
            sinks = np.arange(p0, p1, 5)
            rms, mx, _ = oracle.frac_errors(a[::5, :3], oracle.fp64_sinks(box, soft, eps, sinks))
            assert rms <= RMS and mx <= MAX, (rms, mx)
            if dens:  # positive terms, FP32 sums
                np.testing.assert_allclose(a[::5, 3], oracle.fp64_density(box, b2, sinks), rtol=1e-5,
                                           atol=1e-6 * b2)
            else:
                assert np.all(a[:, 3] == 0)


@pytest.mark.parametrize("soft", [0, 1, 2, 3])
@pytest.mark.parametrize("cells", [0.02, 0.09, 0.3])
def test_density_of_every_softening(capi, oracle, synth, soft, cells):
    """The density channel beside every softening, from lengths far below the
    density radius (0.2 cells) to above it, on both engines."""
    box = synth.clustered_box(15000, 9, seed=8, n_clumps=10)
    b2 = float(np.float32((0.2 / box.cpd) ** 2))
    eps = synth.kernel_eps(soft, cells / box.cpd)
    sinks = np.arange(0, box.n, 4)
    want = oracle.fp64_density(box, b2, sinks)
    for acc, engine in ((capi.ACC_COMPENSATED, capi.ENGINE_MUTUAL), (capi.ACC_PLAIN, capi.ENGINE_ONE_SIDED)):
        with capi.Context(softening=soft, eps=eps, b2=b2, accumulation=acc) as ctx:
            db = ctx.box(box)
            a = db.forces()
            assert ctx.last_engine() == engine
            db.close()
        np.testing.assert_allclose(a[sinks, 3], want, rtol=1e-5, atol=1e-6 * b2)
        _check(oracle, box, soft, eps, a, sinks=sinks)


def test_serving_on_the_one_sided_engine(capi, synth):
    """Served slabs of plain and of tiny-softening boxes: the bits of the same
    slabs swept alone."""
    box = synth.clustered_box(15000, 9, seed=9, n_clumps=10)
    for acc, cells in ((capi.ACC_PLAIN, 0.02), (capi.ACC_COMPENSATED, SMALL)):
        with capi.Context(softening=0, eps=synth.kernel_eps(0, cells / 9), accumulation=acc,
                          kernel_variant=0) as ctx:
            db = ctx.box(box)
            alone = [db.forces(s, s + 1) for s in range(9)]
            srv = capi.Server(ctx)
            outs = [np.full_like(a, np.nan) for a in alone]
            tickets = [srv.submit(db, s, outs[s]) for s in (4, 0, 8, 1, 2, 7, 3, 5, 6)]
            for t in tickets:
                srv.wait(t)
            assert ctx.last_engine() == capi.ENGINE_ONE_SIDED
            srv.close()
            db.close()
        for a, b in zip(alone, outs):
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32))


@pytest.mark.parametrize("soft,b2,engine", [(3, 5e-9, 0), (3, 2e-9, 1), (2, 1e-12, 0), (1, 1e-13, 1),
                                            (0, 1e-12, 0), (0, 1e-13, 1)])
def test_tiny_density_radii(capi, oracle, synth, soft, b2, engine):
    """The mutual engine takes the density from r^2 only where what r^2 carries
    on top (1e-16 with the cubic Plummer softening) is below the rounding of b2,
    and only while the scale of its sums is a float.  Pairs at half the
    radius."""
    cpd = 11
    rng = np.random.default_rng(11)
    n = np.zeros((cpd,) * 3, int)
    n[::4, ::4, ::4] = 2
    cs = np.zeros(cpd ** 3 + 1, np.int64)
    cs[1:] = np.cumsum(n.ravel())
    m = int(cs[-1])
    d = rng.normal(size=(3, m // 2))
    d *= 0.5 * np.sqrt(b2) / np.linalg.norm(d, axis=0)
    p = np.stack([d / 2, -d / 2], 2).reshape(3, m).astype(np.float32)  # about the cell centre: exact enough
    box = synth.Box(cpd=cpd, x=p[0].copy(), y=p[1].copy(), z=p[2].copy(), cell_start=cs)
    with capi.Context(softening=soft, eps=synth.kernel_eps(soft, 0.02 / cpd), b2=b2) as ctx:
        db = ctx.box(box)
        a = db.forces()
        assert ctx.last_engine() == engine
        db.close()
    want = oracle.fp64_density(box, b2, np.arange(m))
    np.testing.assert_allclose(a[:, 3], want, rtol=1e-6)
