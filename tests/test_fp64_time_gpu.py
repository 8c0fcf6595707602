"""The observer time of the FP64 form against extended precision: rounding errors that differ from
element to element cancel in the bins, what every element shares shifts the whole signal in time."""
import numpy as np
import pytest

from acum3_periodic_gb300 import synth

pytestmark = pytest.mark.gpu

L = np.longdouble


def _signal(f, obs, c):
    """core.cu:93-231 on preprocessed fields [element][step][18], in extended precision:
    [steps][observers], and the largest travel time in bins."""
    f = f.astype(L)
    x, ds, n, nd, V, Vd, P, Pd = (f[..., k] for k in (slice(0, 3), 3, slice(4, 7), slice(7, 10), slice(10, 13),
                                                      slice(13, 16), 16, 17))
    a0, rho, oM, dPsi, dTau = (L(c[k]) for k in ("a0", "rhoRef", "oM", "dPsi", "dTau"))
    v = np.asarray(c["vInf"]).astype(L)
    dot = lambda a, b: (a * b).sum(-1)  # noqa: E731
    T = f.shape[1]
    out, far = np.zeros((T, len(obs)), L), 0.0
    for i, o in enumerate(obs.astype(L)):
        d = o - x
        beta, al = dot(d, v), a0 * a0 - dot(v, v)
        tr = (np.sqrt(al * dot(d, d) + beta * beta) - beta) / al
        R = a0 * tr
        rh = (d - v * tr[..., None]) / R[..., None]
        M, load = V / a0, P[..., None] * n
        Mr, Lr = dot(M, rh), dot(load, rh)
        G = 1 / (1 - Mr)
        K = dot(Vd / a0, rh) + a0 / R * (Mr - dot(M, M))
        Ldr = dot(Pd[..., None] * n + P[..., None] * nd, rh)
        p = ds / (4 * L(np.pi) * a0) / R * G * G * (rho * a0 * dot(V, n) * G * K + Ldr + a0 / R * (Lr - dot(load, M)) +
                                                    Lr * G * K)
        u = (np.arange(T, dtype=L) * dTau + tr) * oM / dPsi
        far = max(far, float((tr * oM / dPsi).max()))
        u, p = np.concatenate([u, u[:, :1] + T], 1), np.concatenate([p, p[:, :1]], 1)
        a, b = u[:, :-1], u[:, 1:]
        na, nb = np.floor(a), np.floor(b)
        for q in (1, 2, 3):
            use = na + q <= nb
            w = ((na + q - a) / (b - a))[use]
            np.add.at(out[:, i], np.mod((na + q)[use], T).astype(int), p[:, :-1][use] + w * (p[:, 1:] - p[:, :-1])[use])
    return out, far


@pytest.mark.parametrize("ntime,radii", [(360, 10.0), (720, 30.0), (1440, 10.0)])
def test_no_shared_shift_in_hover(ntime, radii):
    from acum3_periodic_gb300 import native
    spec = synth.RotorSpec(blades=2, n_span=3, n_chord_side=4, ntime=ntime, dpsi_deg=360.0 / ntime, minf=0.0, tip_mach=0.6)
    d = synth.rotor_deck(spec, synth.observers("sphere", 5, radii), 1)
    ctx = native.Context(0)
    ctx.set_deck(d, bb=False)
    pA = ctx.tonal(native.PLAIN_FP64)[2]
    ref, far = _signal(ctx.fields(), np.asarray(d.observers(), np.float64), d.derived())
    err, slope = pA - ref, (np.roll(ref, -1, 0) - np.roll(ref, 1, 0)) / 2
    shift = -(err * slope).sum(0) / (slope * slope).sum(0)  # in bins
    # shared: the constants a0^2 and its reciprocal, each rounded once, enter the travel time as
    # their half and their whole; not shared: the bin time's own rounding, over the elements
    tol = 1.5 * 2.0 ** -53 * far + 3 * np.spacing(far) / np.sqrt(12.0 * d.E)
    assert np.abs(shift).max() < tol, (shift, tol)
