"""FP32 precision of single pairs: boxes of isolated pairs, each in one cell, so
that a record is one kernel evaluation and its roundings.  Expected errors come
from the same operations emulated in numpy, each rounded to FP32."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

F, D = np.float32, np.float64
CPD, EVERY = 55, 5  # a pair in every fifth cell each way: none meets another


def _fma(a, b, c):
    """Rounded once: the product of two floats is exact in double, and a sum in
    double is within 2^-53 of exact."""
    return (np.asarray(a, D) * np.asarray(b, D) + np.asarray(c, D)).astype(F)


def _pairs(synth, seed, lo, hi):
    """Pairs with separations uniform in [lo, hi) (box units, below 0.4 cells)."""
    rng = np.random.default_rng(seed)
    n = CPD // EVERY
    cell = np.arange(CPD ** 3).reshape((CPD,) * 3)[::EVERY, ::EVERY, ::EVERY][:n, :n, :n].ravel()
    v = rng.normal(size=(3, len(cell)))
    v *= rng.uniform(lo, hi, len(cell)) / np.linalg.norm(v, axis=0)
    a = rng.uniform(-0.05, 0.05, v.shape) / CPD
    p = np.stack([a + v / 2, a - v / 2], 2).reshape(3, -1).astype(F)  # sinks 2k, 2k + 1
    cs = np.zeros(CPD ** 3 + 1, np.int64)
    cs[cell + 1] = 2
    return synth.Box(cpd=CPD, x=p[0].copy(), y=p[1].copy(), z=p[2].copy(), cell_start=np.cumsum(cs))


def _records(capi, synth, soft, eps, acc, lo, hi, seeds=12):
    """Records and separations (sink - other) of all pairs of some boxes."""
    rec, sep = [], []
    with capi.Context(softening=soft, eps=eps, accumulation=acc, kernel_variant=0) as ctx:
        for seed in range(seeds):
            box = _pairs(synth, seed, lo, hi)
            db = ctx.box(box)
            rec.append(db.forces()[:, :3])
            db.close()
            p = np.stack([box.x, box.y, box.z], 1)
            sep.append(p - p.reshape(-1, 2, 3)[:, ::-1].reshape(-1, 3))  # rounds as the kernel's
    return np.concatenate(rec), np.concatenate(sep)


def _exact_separation_error(a, f64, sep, d64):
    want = f64[:, None] * d64
    e = np.linalg.norm(a - want, axis=1) / np.linalg.norm(want, axis=1)
    return float(np.sqrt(np.mean(e ** 2))), e


def _r2(sep, add):
    x, y, z = sep.T
    return _fma(z, z, _fma(y, y, _fma(x, x, np.full(len(sep), F(add)))))


def _newton_full(r2):
    y = (1 / np.sqrt(r2.astype(D))).astype(F)
    y2 = y * y
    y3 = y2 * y
    return _fma(y3 * _fma(r2, y2, F(-1)), F(-1.5), y3)


@pytest.mark.parametrize("soft", [0, 1])
def test_one_sided_step(capi, synth, soft):
    """The one-sided engine's pairs are as exact as the full Newton step: within
    5 % of its emulation over 31 944 records (sampling error of an RMS: 1/sqrt(2 N)
    = 0.4 %; the hardware estimate adds below 1 %).  The four-instruction step
    is 13 % above."""
    length = 0.002 / CPD
    eps = float(F(synth.kernel_eps(soft, length)))
    a, sep = _records(capi, synth, soft, eps, capi.ACC_PLAIN, 0.05 / CPD, 0.38 / CPD)
    add = eps if soft == 0 else 1e-25
    unit = eps ** -1.5 if soft == 1 else 1.0
    r64 = (sep.astype(D) ** 2).sum(1) + (eps if soft == 0 else 0.0)
    rms, _ = _exact_separation_error(a, unit * r64 ** -1.5, sep, sep.astype(D))
    emu = (_newton_full(_r2(sep, add))[:, None] * sep).astype(F)
    if soft == 1:
        emu = emu * F(unit)
    want, _ = _exact_separation_error(emu, unit * r64 ** -1.5, sep, sep.astype(D))
    assert rms <= 1.05 * want, (rms, want)


def _newton_short(r2):
    """The four-instruction step times NEWTON_UNIT, and that unit."""
    k = F(5) / F(3)
    y = (1 / np.sqrt(r2.astype(D))).astype(F)
    y2 = y * y
    return (y2 * y) * _fma(r2, y2, -k), 1.0 - D(k)


@pytest.mark.parametrize("soft", [0, 1])
def test_mutual_records_round_once(capi, synth, soft):
    """Records of the fixed-point sums: the pair's own roundings and one more.
    Within 2 % of their emulation (estimate and sampling error below 1 %); the
    sum and the scale each rounded to a float first are 4 % above."""
    length = 0.002 / CPD
    eps = float(F(synth.kernel_eps(soft, length)))
    a, sep = _records(capi, synth, soft, eps, capi.ACC_COMPENSATED, 0.05 / CPD, 0.38 / CPD)
    add = eps if soft == 0 else 1e-25
    unit = eps ** -1.5 if soft == 1 else 1.0
    r64 = (sep.astype(D) ** 2).sum(1) + (eps if soft == 0 else 0.0)
    rms, _ = _exact_separation_error(a, unit * r64 ** -1.5, sep, sep.astype(D))
    g, newton_unit = _newton_short(_r2(sep, add))
    emu = ((g[:, None] * sep).astype(F).astype(D) * (unit / newton_unit)).astype(F)
    want, _ = _exact_separation_error(emu, unit * r64 ** -1.5, sep, sep.astype(D))
    assert rms <= 1.02 * want, (rms, want)


def _cubic_spline64(u, e):
    far = (u * e) ** -3
    mid = far * (-1 / 15 + u ** 3 * (8 / 3 - 3 * u + 1.2 * u ** 2 - u ** 3 / 6))
    near = e ** -3 * (4 / 3 - 1.2 * u ** 2 + 0.5 * u ** 3)
    return np.where(u >= 2, far, np.where(u >= 1, mid, near))


@pytest.mark.parametrize("acc", [0, 1])
def test_cubic_spline_over_its_reach(capi, synth, acc):
    """RMS error below 1.6e-7 wherever the pair lies: the force factor's in an
    FP32 emulation is at most 9.3e-8 (u just above 1), the product's and the
    record's roundings add 3e-8 each.  Evaluated by powers of u, the middle
    branch loses 2e-6 at u = 2."""
    e = 0.17 / CPD
    eps = float(F(synth.kernel_eps(2, e)))
    a, sep = _records(capi, synth, 2, eps, acc, 0.02 * e, 2.3 * e)
    d64 = sep.astype(D)
    u = np.sqrt((d64 ** 2).sum(1)) * eps
    _, err = _exact_separation_error(a, _cubic_spline64(u, 1.0 / eps), sep, d64)
    edges = [0.02, 0.5, 1, 1.25, 1.5, 1.75, 2, 2.3]
    for lo, hi in zip(edges, edges[1:]):
        q = err[(u >= lo) & (u < hi)]
        assert len(q) > 1000
        rms = np.sqrt(np.mean(q ** 2))
        assert rms <= 1.6e-7, (lo, hi, rms)


@pytest.mark.parametrize("acc", [0, 1])
def test_cubic_plummer_reciprocal(capi, synth, acc):
    """The reciprocal is as good as a division: within 3 % of the emulation with
    one (estimate and sampling error below 1 %); a Newton step whose factor is
    rounded near 1 is 5 % above or more."""
    e = 0.1 / CPD
    eps = float(F(synth.kernel_eps(3, e)))
    a, sep = _records(capi, synth, 3, eps, acc, 0.2 * e, 3.5 * e)
    d64 = sep.astype(D)
    g64 = 1 / (((d64 ** 2).sum(1) + D(F(1e-16))) ** 1.5 + eps)
    rms, _ = _exact_separation_error(a, g64, sep, d64)
    r2 = _r2(sep, 1e-16)
    rinv = (1 / np.sqrt(r2.astype(D))).astype(F)
    g = F(1) / _fma(r2 * r2, rinv, F(eps))
    want, _ = _exact_separation_error((g[:, None] * sep).astype(F), g64, sep, d64)
    assert rms <= 1.03 * want, (rms, want)


@pytest.mark.parametrize("soft", [0, 3])
def test_density_terms_carry_no_common_error(capi, synth, soft):
    """Density sums of softenings that put a constant into r^2: its rounding is
    not in every term.  The mean signed error of 31 944 records is below 6e-9 of
    b2 (roundings of 6e-8 at most average to 4e-10); b2 + eps^2 rounded to a
    float is off by more than 2e-8 for the lengths taken here."""
    b2 = float(F((0.2 / CPD) ** 2))
    if soft == 0:
        for k in range(1000):
            eps = float(F(b2 / 32 * (1 + k * 1e-5)))
            if abs(b2 + eps - float(F(b2 + eps))) > 2.2e-8 * b2:
                break
    else:
        eps = float(F(synth.kernel_eps(3, 0.03 / CPD)))
    w, want = [], []
    with capi.Context(softening=soft, eps=eps, b2=b2) as ctx:
        for seed in range(12):
            box = _pairs(synth, seed, 0.02 / CPD, 0.25 / CPD)
            db = ctx.box(box)
            w.append(db.forces()[:, 3])
            db.close()
            p = np.stack([box.x, box.y, box.z], 1)
            sep = (p - p.reshape(-1, 2, 3)[:, ::-1].reshape(-1, 3)).astype(D)
            want.append(b2 + np.maximum(b2 - (sep ** 2).sum(1), 0))
    err = (np.concatenate(w) - np.concatenate(want)) / b2
    assert np.abs(err).max() < 3e-7
    assert abs(err.mean()) < 6e-9, err.mean()
