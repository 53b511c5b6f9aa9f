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
