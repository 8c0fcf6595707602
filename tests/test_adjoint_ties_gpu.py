"""The low-pass filter's medians choose between pressures that may differ by one rounding.  The
preprocessing forms the filter's input term by term with fixed roundings, restated here in exact
arithmetic, and the adjoint sends each cotangent to the step that those very values choose."""
from fractions import Fraction

import numpy as np
import pytest

from acum3_periodic_gb300 import synth

from test_dropin_gpu import call_dropin

pytestmark = pytest.mark.gpu

T = 24


def _periodic(cp, pscale):
    """mathfunc.cu:165-206 on one element's Cp (floats), every operation rounded to double."""
    r = lambda v: float(v)  # noqa: E731  (a Fraction rounds correctly)
    F = Fraction
    p = [r(F(float(c)) * F(pscale)) for c in cp]
    k2, k1 = p[-1], p[0] - (p[1] - p[0])
    ds, dk = (p[0] - k1) - (p[-1] - p[-2]), k1 - k2
    bb = -2.0 * ds / T - 3.0 * dk / T / T
    aa = -bb / T - ds / T / T - dk / T / T / T
    out = []
    for t in range(T):
        u = float(t + 1)
        cub = r(F(ds) * F(u) + F(r(F(bb * u) * F(u) + F(aa * u * u * u)))) + k1
        out.append(p[t] - (cub - k2))
    return np.array(out)


def _choice(x):
    """The 3-point periodic median as the matrix of its choices (mathfunc.cu:208-341)."""
    S = np.zeros((T, T))
    for t in range(T):
        l, m, r = x[t - 1], x[t], x[(t + 1) % T]
        hi, lo = max(l, m, r), min(l, m, r)
        S[t, (t - 1) % T if lo < l < hi else t if lo < m < hi else (t + 1) % T] = 1.0
    return S


def _deck(lowpass):
    """Ends that match to a rounding (2 Cp[0] - Cp[1] = Cp[T-1] and equal end slopes, before the
    scaling), so that make_periodic moves equal neighbours by a rounding or two."""
    spec = synth.RotorSpec(blades=2, n_span=2, n_chord_side=6, ntime=T, dpsi_deg=360.0 / T, tip_mach=0.6, lowpass=lowpass)
    d = synth.rotor_deck(spec, synth.observers("circle", 3, 10.0), 1)
    rng = np.random.default_rng(4)
    for s in d.surfaces:
        for e in range(s.shape[1]):
            c, step = np.float32(1.0 + rng.random()), np.float32(2.0 ** -22)
            cp = c + step * np.repeat(rng.integers(-4, 5, T // 3), 3).astype(np.float32)
            cp[[0, 1, T - 2, T - 1]] = c + step * np.array([0, 1, -2, -1], np.float32)
            s[:, e, 3] = cp
    return d


def _pscale(d):
    from acum3_periodic_gb300 import native
    i = native.inputs_of(d)
    return 0.5 * i.rhoRef * (i.Mref * i.Mref) * (i.a0 * i.a0)


def test_filter_input_has_fixed_roundings():
    from acum3_periodic_gb300 import native
    d = _deck(0)
    ctx = native.Context(0)
    ctx.set_deck(d, bb=False)
    P = ctx.fields()[:, :, 16]
    cps = np.concatenate([s[:, :, 3].T for s in d.surfaces])
    for e in range(d.E):
        np.testing.assert_array_equal(P[e], _periodic(cps[e], _pscale(d)))


def test_cotangents_go_to_the_steps_that_the_medians_chose():
    torch = pytest.importorskip("torch")
    from acum3_periodic_gb300 import native
    L = native.lib()
    d = _deck(1)
    ctx = native.Context(0)
    ctx.set_deck(d, bb=False)
    f, w = ctx.fields(), np.random.default_rng(5).standard_normal((T, d.nObs))
    gcp = ctx.adjoint(native.PLAIN_FP64, w)[1]
    g = np.exp(-0.5 * (np.arange(13) - 6.0) ** 2 / 4.0)
    G = sum(v * np.roll(np.eye(T), k - 6, 1) for k, v in enumerate(g / g.sum()))
    i = np.arange(1, T + 1)
    E = np.eye(T)
    k1, k2, ds = 2 * E[0] - E[1], E[-1], (E[1] - E[0]) - (E[-1] - E[-2])
    bb = -2 * ds / T - 3 * (k1 - k2) / T ** 2
    aa = -bb / T - ds / T ** 2 - (k1 - k2) / T ** 3
    M = E - (np.outer(i ** 3, aa) + np.outer(i ** 2, bb) + np.outer(i, ds) + k1 - k2)
    cps = np.concatenate([s[:, :, 3].T for s in d.surfaces])
    dt = d.derived()["dTau"]
    for e in (23, 37):  # where a rounding tells neighbours apart
        p0 = _periodic(cps[e], _pscale(d))
        S1 = _choice(p0)
        p1 = G @ (S1 @ p0)
        assert np.abs(np.diff(p1)).min() > 1e-11 * np.abs(p1).max()  # the second medians have no ties
        # the pressure of a filtered unit pulse at each step: what the filter's transpose starts from
        b = np.zeros(T)
        for t in range(T):
            h = f.copy()
            h[:, :, 16:18] = 0.0
            h[e, t, 16] = 1.0
            h[e, (t - 1) % T, 17], h[e, (t + 1) % T, 17] = 0.5 / dt, -0.5 / dt
            rc, _, pL, _ = call_dropin(L.acum_find_pressure_time_history_f64, d, h, np.float64, torch)
            assert rc == 0
            b[t] = (w * pL).sum()
        want = _pscale(d) * (M.T @ S1.T @ G.T @ _choice(p1).T @ G.T @ b)
        np.testing.assert_allclose(gcp[e], want, rtol=0, atol=1e-8 * np.abs(want).max())
