"""Both engines by name: which one a call takes, and the one-sided engine's
results where the mutual one does not apply (plain accumulation, softenings
below its fixed-point range), for every entry point, against the FP64 oracle.
RMS fractional error <= 2e-6, max <= 1e-4, as in the other GPU tests."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RMS, MAX = 2e-6, 1e-4
SMALL = 1e-6  # softening length, cells: below the fixed-point range of these boxes


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
