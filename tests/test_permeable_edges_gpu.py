"""The permeable-surface preprocessing at the edges of its kernel: periods around a filter
run of 17 steps and around the series a block filters at one time (256 runs), arrays and
surfaces that start at odd elements, more surfaces than travel with the launch, steps whose
reciprocal is and is not near a double, and series that are zero, tiny or huge.  FP64 storage
equals the oracle; float storage equals the oracle's results rounded once."""
import numpy as np
import pytest

from acum3_periodic_gb300 import synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _check(ne, X, N, U, PR, args):
    from acum3_periodic_gb300 import native
    V0 = np.zeros_like(N)
    for nm, a, b in zip("XNVUP", native.preprocess_per(ne, X, N, V0, U, PR, *args),
                        O.preprocess_per(X, N, U, PR, *args)):
        np.testing.assert_array_equal(a, b, err_msg=nm)
    f = lambda a: np.asarray(a, np.float32).astype(np.float64)  # noqa: E731
    fargs = tuple(float(np.float32(x)) for x in args[:5]) + args[5:]
    with np.errstate(over="ignore"):
        for nm, a, b in zip("XNVUP", native.preprocess_per(ne, X, N, V0, U, PR, *args, dtype=np.float32),
                            O.preprocess_per(f(X), f(N), f(U), f(PR), *fargs)):
            np.testing.assert_array_equal(a, b.astype(np.float32), err_msg=nm)


@pytest.mark.parametrize("ntime", [6, 7, 13, 16, 17, 18, 34, 35, 160, 161, 255, 256, 257, 512, 513, 529, 530, 867, 871, 1088, 1445, 1446, 2176, 2193])
@pytest.mark.parametrize("periodic,lowpass", [(1, 1), (0, 1), (0, 0)])
def test_periods(ntime, periodic, lowpass):
    X, N, U, PR = synth.permeable_rows(60 + ntime, [2, 1], ntime)
    rng = np.random.default_rng(ntime)
    PR[:, :, 0] += 0.05 * rng.standard_normal(PR.shape[:2])
    U[:, :, 1] += 0.01 * rng.standard_normal(U.shape[:2])
    _check([2, 1], X, N, U, PR, (1.0 / (ntime * 11.0), 340.0, 1.2, 0.08, 1.5, periodic, lowpass))


@pytest.mark.parametrize("step", [2.0 ** -9, 1e-3, 3e-3, 1.0 / 3.0, 7e-4, 2.0 ** -120, 3e31])
def test_steps_and_special_series(step):
    """Constant, zero and negative-zero series, values at both ends of the double range, and
    steps inside and outside the range of the short quotient."""
    T = 40
    X, N, U, PR = synth.permeable_rows(61, [9], T)
    rng = np.random.default_rng(3)
    U[0, :, :3] = 0.0
    U[1, :, :3] = -0.0
    U[2, :, :3] = 1e-300 * rng.standard_normal((T, 3))
    U[3, :, :3] = 1e290 * rng.standard_normal((T, 3))
    U[4, :, :3] = 5e-324 * rng.integers(-9, 9, (T, 3))
    U[5, :, :3] = 1e-40 * rng.standard_normal((T, 3))
    PR[6, :, 2] = 1.25
    X[7, :, :3] = 0.0
    X[8, :, 2] = 1e-45 * rng.standard_normal(T)
    for lowpass in (0, 1):
        from acum3_periodic_gb300 import native
        args = (step, 341.0, 1.1875, 0.11, 1.0, 1, lowpass)
        with np.errstate(over="ignore", invalid="ignore", under="ignore"):
            got, want = native.preprocess_per([9], X, N, np.zeros_like(N), U, PR, *args), O.preprocess_per(X, N, U, PR, *args)
        for nm, a, b in zip("XNVUP", got, want):
            ok = np.isfinite(b) & ((np.abs(b) > 1e-280) | (b == 0))  # the quotient of a normal range
            np.testing.assert_array_equal(a[ok], b[ok], err_msg=nm)
            assert ok.mean() > 0.5


def test_many_surfaces_and_odd_starts():
    """150 surfaces (some empty), each array in a buffer that starts at an odd element and
    leaves odd gaps between surfaces: every element is found through its surface's pointers,
    and nothing between the surfaces is written."""
    import ctypes as C
    torch = pytest.importorskip("torch")
    from acum3_periodic_gb300 import native
    rng = np.random.default_rng(5)
    for nsurf in (3, 48, 49, 150):
        ne = [int(k) for k in rng.integers(0, 3, nsurf)]
        ne[-1] = 2
        T, etot = 21, sum(ne)
        X, N, U, PR = synth.permeable_rows(62, ne, T)
        args = (0.004, 340.0, 1.2, 0.08, 1.0, 0, 1)
        want = O.preprocess_per(X, N, U, PR, *args)
        for dt, tdt in ((np.float64, torch.float64), (np.float32, torch.float32)):
            if dt == np.float32:
                f = lambda a: np.asarray(a, np.float32).astype(np.float64)  # noqa: E731
                args = tuple(float(np.float32(x)) for x in args[:5]) + args[5:]
                want = O.preprocess_per(f(X), f(N), f(U), f(PR), *args)
            dev, ptrs, where = [], [], []
            for a, w in zip((X, N, np.zeros_like(N), U, PR), (4, 6, 6, 6, 4)):
                gaps = rng.integers(0, 4, nsurf)
                start, at, rows = [], 1, []
                e = 0
                for k in range(nsurf):
                    at += int(gaps[k])
                    start.append(at)
                    rows.append((at, e, ne[k]))
                    at += ne[k] * T * w
                    e += ne[k]
                buf = np.full(at + 5, 7.0, dt)
                for s0, e0, n in rows:
                    buf[s0:s0 + n * T * w] = np.asarray(a[e0:e0 + n], dt).reshape(-1)
                dev.append(torch.tensor(buf, device="cuda:0"))
                ptrs.append(np.array(start, np.int32))
                where.append(rows)
            E = np.array(ne, np.int32)
            vp = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
            torch.cuda.synchronize()
            rc = native.lib().acum_preprocess_per_device(*[C.c_void_p(t.data_ptr()) for t in dev],
                                                         int(dt == np.float64), nsurf, *[vp(q) for q in ptrs], vp(E), T,
                                                         *args, C.c_void_p(0))
            assert rc == 0 and etot > 0
            torch.cuda.synchronize()
            for nm, t, b, rows, w in zip("XNVUP", dev, want, where, (4, 6, 6, 6, 4)):
                got, seen = t.cpu().numpy(), np.zeros(t.numel(), bool)
                for s0, e0, n in rows:
                    np.testing.assert_array_equal(got[s0:s0 + n * T * w], b[e0:e0 + n].astype(dt).reshape(-1), err_msg=nm)
                    seen[s0:s0 + n * T * w] = True
                assert (got[~seen] == 7.0).all(), nm


@pytest.mark.parametrize("ntime", [2944, 2945, 3000, 4080, 4096])
@pytest.mark.parametrize("periodic,lowpass", [(1, 1), (0, 1), (0, 0)])
def test_long_periods(ntime, periodic, lowpass):
    """Both sides of the period from which a block filters one series at a time, in short runs."""
    test_periods(ntime, periodic, lowpass)
