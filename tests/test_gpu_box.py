"""Parity of the batched B200 path (nf_box_forces, through the C ABI) with
the oracle.

Tolerances (stated once, used below):
  * against the reference's own CPU direct (golden vectors / oracle
    restatement): for every sink and component |a_k - a_ref,k| <= 1e-4 |a_ref|,
    and RMS over sinks of |a - a_ref| / |a_ref| <= 5e-6.  The reference itself
    carries ~1e-6 RMS FP32 error (shifted frames, long FP32 running sums), so
    bit equality with it is neither expected nor desirable.
  * against the FP64 oracle: RMS fractional force error <= 2e-6 (the
    acceptance bar), and max <= 1e-4.
  * the FOF density channel w: relative 1e-5 against FP64.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GOLDEN_TOL_COMP = 1e-4
GOLDEN_TOL_RMS = 5e-6
FP64_RMS = 2e-6
FP64_MAX = 1e-4


def _golden(path):
    f = np.load(path)
    from abacus_public_b200 import synth
    box = synth.Box(cpd=int(f["cpd"]), x=f["x"], y=f["y"], z=f["z"], cell_start=f["cell_start"])
    return box, int(f["softening"]), float(f["eps"]), list(f["slabs"]), f["rows"], f["acc"]


def _check_vs_ref(a, ref):
    norm = np.linalg.norm(ref.astype(np.float64), axis=1)
    ok = norm > 0
    diff = np.abs(a[:, :3].astype(np.float64) - ref)
    assert np.all(diff[ok] <= GOLDEN_TOL_COMP * norm[ok, None]), \
        float((diff[ok] / norm[ok, None]).max())
    rel = np.linalg.norm(diff, axis=1)[ok] / norm[ok]
    assert np.sqrt(np.mean(rel ** 2)) <= GOLDEN_TOL_RMS


def _forces_rows(ctx, box, slabs):
    """GPU accelerations of the given slabs, indexed by global particle row."""
    db = ctx.box(box)
    try:
        out = np.zeros((box.n, db.record_width()), np.float32)
        for s in slabs:
            p0, p1 = db.slab_particles(s, s + 1)
            out[p0:p1] = db.forces(s, s + 1)
        return out
    finally:
        db.close()


@pytest.mark.parametrize("name", ["uniform_cpd7", "clustered_cpd9", "sparse_cpd5"])
@pytest.mark.parametrize("soft", [0, 1, 2, 3])
def test_golden_parity(capi, oracle, name, soft):
    import pathlib
    path = pathlib.Path(__file__).parent / "golden" / f"{name}_{oracle.SOFTENING_NAMES[soft]}.npz"
    box, soft_, eps, slabs, rows, acc = _golden(path)
    with capi.Context(softening=soft_, eps=eps) as ctx:
        a = _forces_rows(ctx, box, slabs)[rows]
    _check_vs_ref(a, acc)
    a64 = oracle.fp64_sinks(box, soft_, eps, rows)
    rms, mx, _ = oracle.frac_errors(a[:, :3], a64)
    assert rms <= FP64_RMS and mx <= FP64_MAX, (rms, mx)
    assert np.all(a[:, 3] == 0)  # density channel off


def test_uniform_64_plummer_full_box(capi, oracle, synth):
    """64^3 uniform, cpd 17, Plummer eps = spacing/40: every slab against the
    reference CPU restatement, and a sink sample against FP64."""
    box = synth.config_uniform_64()
    eps = synth.kernel_eps(0, synth.plummer_eps(64))
    with capi.Context(softening=0, eps=eps) as ctx:
        db = ctx.box(box)
        a = db.forces(0, box.cpd)
        t = ctx.last_timing()
        pairs = db.pair_count()
        db.close()
    assert t.pairs == pairs == oracle.pair_count(box)
    ref = np.zeros((box.n, 3), np.float32)
    for s in range(box.cpd):
        oracle.ref32_slab(box, 0, eps, s, acc=ref)
    _check_vs_ref(a, ref)
    # the thinnest margin of the parity bound in the suite: print it (-s)
    norm = np.linalg.norm(ref.astype(np.float64), axis=1)
    worst = float((np.abs(a[:, :3].astype(np.float64) - ref).max(axis=1) / norm).max())
    print(f"\n[uniform 64^3 Plummer] worst per-component deviation from the reference "
          f"CPU direct: {worst:.3e} of |a_ref| (bound {GOLDEN_TOL_COMP:g})")
    sinks = np.sort(np.random.default_rng(0).choice(box.n, 3000, replace=False))
    rms, mx, _ = oracle.frac_errors(a[sinks, :3], oracle.fp64_sinks(box, 0, eps, sinks))
    assert rms <= FP64_RMS and mx <= FP64_MAX, (rms, mx)


@pytest.mark.parametrize("acc_mode", [0, 1])
def test_clustered_single_spline(capi, oracle, synth, acc_mode):
    """Clustered 96^3 box, cpd 25 (occupancy 0 .. thousands): the heavy-tile
    split path, the spline near branch, both accumulation modes."""
    box = synth.clustered_box(96 ** 3, 25, seed=7, n_clumps=300)
    assert box.counts.max() > 1000
    eps = synth.kernel_eps(1, synth.plummer_eps(96))
    with capi.Context(softening=1, eps=eps, accumulation=acc_mode) as ctx:
        db = ctx.box(box)
        a = db.forces()
        db.close()
    rng = np.random.default_rng(1)
    sinks = np.sort(rng.choice(box.n, 2000, replace=False))
    a64 = oracle.fp64_sinks(box, 1, eps, sinks)
    rms, mx, _ = oracle.frac_errors(a[sinks, :3], a64)
    assert rms <= FP64_RMS and mx <= FP64_MAX, (rms, mx)
    cells = np.unique(np.searchsorted(box.cell_start, sinks, side="right") - 1)
    ref = oracle.ref32_cells(box, 1, eps, cells)
    _check_vs_ref(a[sinks], ref[sinks])


def test_deterministic_and_range_consistent(capi, synth):
    box = synth.clustered_box(40000, 13, seed=8, n_clumps=40)
    eps = synth.kernel_eps(1, synth.plummer_eps(34))
    with capi.Context(softening=1, eps=eps) as ctx:
        db = ctx.box(box)
        a1 = db.forces()
        a2 = db.forces()
        assert np.array_equal(a1.view(np.uint32), a2.view(np.uint32))
        p0, p1 = db.slab_particles(4, 9)
        b = db.forces(4, 9)
        db.close()
    np.testing.assert_allclose(b, a1[p0:p1], rtol=0, atol=1e-6 * np.abs(a1).max())


def test_density_channel(capi, oracle, synth):
    box = synth.clustered_box(30000, 11, seed=9, n_clumps=20)
    eps = synth.kernel_eps(0, synth.plummer_eps(31))
    b2 = float(np.float32((0.2 / 31) ** 2))
    with capi.Context(softening=0, eps=eps, b2=b2) as ctx:
        db = ctx.box(box)
        a = db.forces()
        db.close()
    sinks = np.arange(0, box.n, 7)
    w64 = oracle.fp64_density(box, b2, sinks)
    np.testing.assert_allclose(a[sinks, 3], w64, rtol=1e-5, atol=1e-6 * b2)
    assert (w64 > 0).mean() > 0.5
    rms, mx, _ = oracle.frac_errors(a[sinks, :3], oracle.fp64_sinks(box, 0, eps, sinks))
    assert rms <= FP64_RMS


def test_radius_one_and_float3(capi, oracle, synth):
    box = synth.uniform_box(20000, 9, seed=10)
    eps = synth.kernel_eps(0, synth.plummer_eps(27))
    with capi.Context(softening=0, eps=eps, near_field_radius=1, out_kind=capi.OUT_FLOAT3) as ctx:
        db = ctx.box(box)
        a = db.forces()
        db.close()
    assert a.shape == (box.n, 3)
    sinks = np.arange(0, box.n, 5)
    a64 = oracle.fp64_sinks(box, 0, eps, sinks, R=1)
    rms, mx, _ = oracle.frac_errors(a[sinks], a64)
    assert rms <= FP64_RMS, rms


@pytest.mark.parametrize("soft", [0, 1])
def test_kernel_shapes_agree(capi, synth, soft):
    """Every kernel shape the autotuner can pick, and forced tile sizes, give
    the same accelerations to rounding; the autotuner records its timings."""
    box = synth.clustered_box(30000, 11, seed=11, n_clumps=25)
    eps = synth.kernel_eps(soft, synth.plummer_eps(31))
    outs = []
    nv = capi.lib().nf_kernel_variant_count()
    assert nv >= 4
    for v in range(nv):
        with capi.Context(softening=soft, eps=eps, kernel_variant=v) as ctx:
            db = ctx.box(box)
            outs.append(db.forces())
            assert ctx.last_timing().variant == v
            db.close()
    for S in (1, 2):
        with capi.Context(softening=soft, eps=eps, sinks_per_lane=S) as ctx:
            db = ctx.box(box)
            outs.append(db.forces())
            db.close()
    with capi.Context(softening=soft, eps=eps) as ctx:
        db = ctx.box(box)
        outs.append(db.forces())
        v, ms = db.tuning()
        assert 0 <= v < nv and ctx.last_timing().variant == v
        assert all(m > 0 for m in ms) and ms[v] == min(ms)
        db.close()
    for o in outs[1:]:
        np.testing.assert_allclose(o, outs[0], rtol=0, atol=2e-6 * np.abs(outs[0]).max())


def test_edge_cases(capi, oracle, synth):
    # all particles in a single cell; most cells empty; minimum cpd for R=2
    rng = np.random.default_rng(12)
    n = 3000
    cpd = 5
    h = 1.0 / cpd
    x = (rng.random(n, dtype=np.float32) - 0.5) * np.float32(0.999 * h)
    y = (rng.random(n, dtype=np.float32) - 0.5) * np.float32(0.999 * h)
    z = (rng.random(n, dtype=np.float32) - 0.5) * np.float32(0.999 * h)
    cs = np.zeros(cpd ** 3 + 1, np.int64)
    cs[63:] = n
    box = synth.Box(cpd=cpd, x=x, y=y, z=z, cell_start=cs)
    eps = synth.kernel_eps(1, 0.002)
    with capi.Context(softening=1, eps=eps) as ctx:
        db = ctx.box(box)
        a = db.forces()
        db.close()
        # empty box
        e = synth.Box(cpd=cpd, x=x[:0], y=y[:0], z=z[:0], cell_start=np.zeros(cpd ** 3 + 1, np.int64))
        db = ctx.box(e)
        assert db.forces().shape == (0, 4)
        db.close()
    sinks = np.arange(0, n, 3)
    rms, mx, _ = oracle.frac_errors(a[sinks, :3], oracle.fp64_sinks(box, 1, eps, sinks))
    assert rms <= FP64_RMS and mx <= FP64_MAX, (rms, mx)


def test_errors_are_status_codes(capi, synth):
    with pytest.raises(capi.NfError) as ei:
        capi.Context(softening=7, eps=1.0)
    assert ei.value.status == capi.NF_EINVAL
    with pytest.raises(capi.NfError):
        capi.Context(eps=float("inf"))
    box = synth.uniform_box(1000, 5, seed=1)
    with capi.Context(softening=0, eps=1e-6) as ctx:
        db = ctx.box(box)
        with pytest.raises(capi.NfError) as ei:
            db.forces(3, 2)
        assert ei.value.status == capi.NF_EINVAL
        with pytest.raises(capi.NfError):
            db.forces(0, 6)
        db.close()


def test_box_rejects_cpd_beyond_32_bit_pencil_ids(capi):
    """Work items name a pencil by its centre cell's 32-bit linear id, so a box
    must have cpd^3 < 2^31: cpd = 1291 is refused before any cell is read."""
    import ctypes
    dummy = np.zeros(4, np.int64)
    with capi.Context(softening=0, eps=1e-6) as ctx:
        h = ctypes.c_void_p()
        rc = capi.lib().nf_box_create(ctx.h, 1291, 0, dummy.ctypes.data_as(ctypes.c_void_p),
                                      None, None, None, ctypes.byref(h))
        assert rc == capi.NF_EINVAL and not h.value
        assert "1290" in capi.last_error()


def test_memory_of_destroyed_boxes(capi, synth):
    """A context without boxes holds no device memory of its own; destroyed
    boxes leave at most 2 GiB with it, which nf_trim and nf_shutdown give back,
    and which the next box takes over."""
    import torch
    mib = 1 << 20

    def free():
        return torch.cuda.mem_get_info()[0]

    box = synth.uniform_box(1_500_000, 29, seed=31)
    with capi.Context(softening=0, eps=1e-6) as ctx:  # kernels loaded before anything is counted
        db = ctx.box(box)
        db.forces()
        db.close()
    capi.lib().nf_trim()
    base = free()
    ctx = capi.Context(softening=0, eps=1e-6, kernel_variant=0)
    assert base - free() < 4 * mib
    db = ctx.box(box)
    want = db.forces()
    held = base - free()
    assert held > 64 * mib
    db.close()
    assert 0 < base - free() <= held <= 2 << 30
    db = ctx.box(box)  # out of what was kept, but for the gaps between its blocks
    assert np.array_equal(db.forces(), want)
    assert base - free() <= 1.5 * held
    db.close()
    capi.lib().nf_trim()
    assert base - free() < 4 * mib
    db = ctx.box(box)
    assert np.array_equal(db.forces(), want)
    db.close()
    ctx.close()
    assert base - free() < 4 * mib


def test_step_scratch_is_a_chunks(capi, synth):
    """The pipelined step after a sweep of the whole box: positions staged
    (12 bytes a particle), a record buffer per chunk (16), work lists, and a
    second set of sums for the largest chunk only (25 bytes a particle would be
    the whole box again; a chunk of 3 of 17 slabs holds a sixth)."""
    box = synth.uniform_box(64 ** 3, 17, seed=32)
    with capi.Context(softening=0, eps=1e-6, kernel_variant=0) as ctx:
        db = ctx.box(box)
        db.forces()
        before = db.device_bytes()
        out = np.empty((box.n, 4), np.float32)
        db.step(box.x, box.y, box.z, out)
        assert db.device_bytes() - before < (12 + 16 + 15) * box.n
        want = db.forces()
        db.close()
    np.testing.assert_allclose(out, want, rtol=0, atol=2e-6 * np.abs(want).max())


def test_trim_beside_a_running_context(capi, synth):
    """nf_trim from one thread while another sweeps, captures its graphs and
    makes boxes: no call fails and no result changes."""
    import threading
    box = synth.uniform_box(20000, 11, seed=33)
    stop = threading.Event()

    def trim():
        while not stop.is_set():
            capi.lib().nf_trim()

    t = threading.Thread(target=trim)
    with capi.Context(softening=0, eps=1e-6, kernel_variant=0) as ctx:
        db = ctx.box(box)
        want = db.forces()
        db.close()
        t.start()
        try:
            for _ in range(100):
                db = ctx.box(box)
                for _ in range(3):  # launched, captured, replayed
                    assert np.array_equal(db.forces(), want)
                db.close()
        finally:
            stop.set()
            t.join()


@pytest.mark.parametrize("n,cpd,rounds", [(20000, 11, 60), (2_500_000, 51, 8)])
def test_contexts_side_by_side(capi, synth, n, cpd, rounds):
    """Two threads, each with a context of its own, make boxes, sweep them
    (launched, captured as a graph, replayed), change their softening, step them
    and drop them, while a third trims: no call fails and no result changes.
    (The larger box's blocks come from cudaMalloc, the smaller one's from the
    pool.)"""
    import threading
    box = synth.uniform_box(n, cpd, seed=34)
    errors, stop = [], threading.Event()
    with capi.Context(softening=0, eps=1e-6, kernel_variant=0) as ctx:
        db = ctx.box(box)
        want = db.forces()
        stepped = np.empty_like(want)
        db.step(box.x, box.y, box.z, stepped)
        db.close()

    def work():
        try:
            with capi.Context(softening=0, eps=1e-6, kernel_variant=0) as ctx:
                out = np.empty_like(want)
                for _ in range(rounds):
                    db = ctx.box(box)
                    for _ in range(3):
                        assert np.array_equal(db.forces(), want)
                    db.step(box.x, box.y, box.z, out)
                    assert np.array_equal(out, stepped)
                    db.set_eps(2e-6)
                    db.set_eps(0.0)
                    assert np.array_equal(db.forces(), want)
                    db.close()
        except Exception as e:  # noqa: BLE001 -- reported by the main thread
            errors.append(e)

    def trim():
        while not stop.is_set():
            capi.lib().nf_trim()

    threads = [threading.Thread(target=work) for _ in range(2)]
    trimmer = threading.Thread(target=trim)
    for t in threads + [trimmer]:
        t.start()
    for t in threads:
        t.join()
    stop.set()
    trimmer.join()
    assert not errors, errors


def test_calls_beside_a_graph_capture(capi, synth):
    """While one thread captures a CUDA graph (thread-local mode), another makes
    a box, sweeps, steps, changes the softening, serves and destroys it: neither
    fails.  (A wait for the whole device in any of these calls is an error during
    a capture, and breaks it.)"""
    import threading

    import torch
    box = synth.uniform_box(20000, 11, seed=35)
    errors = []

    def work(ctx):
        try:
            db = ctx.box(box)
            want = db.forces()
            for _ in range(3):
                assert np.array_equal(db.forces(), want)
            out = np.empty_like(want)
            db.step(box.x, box.y, box.z, out)
            db.forces(2, 4)
            db.set_eps(2e-6)
            db.forces()
            with capi.Server(ctx) as srv:
                p0, p1 = db.slab_particles(3, 4)
                part = np.empty((p1 - p0, 4), np.float32)
                srv.wait(srv.submit(db, 3, part))
            capi.lib().nf_trim()
            db.close()
        except Exception as e:  # noqa: BLE001 -- reported by the main thread
            errors.append(e)

    x = torch.zeros(1000, device="cuda")
    with capi.Context(softening=0, eps=1e-6, kernel_variant=0) as ctx:
        work(ctx)  # everything loaded
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, capture_error_mode="thread_local"):
            x.add_(1)
            t = threading.Thread(target=work, args=(ctx,))
            t.start()
            t.join()
            x.add_(1)
        g.replay()
        torch.cuda.synchronize()
        assert x[0].item() == 2.0
    assert not errors, errors
