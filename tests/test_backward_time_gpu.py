"""Time that runs backwards (a negative azimuth step, or a negative rotor speed where the caller
gives it) in the mixed form: no ring bounds it, so the whole-row kernel serves it and reports the
order of the samples, as the FP64 form does; the choice of the kernel takes no time of its own."""
import ctypes as C
import time

import numpy as np
import pytest

from acum3_periodic_gb300 import synth
from oracle import oracle as O

from test_dropin_gpu import call_dropin

pytestmark = pytest.mark.gpu


def _deck(ntime, minf):
    return synth.config_deck(1, replicate=720, scale=dict(n_span=3, n_chord_side=3, ntime=ntime, nobs=5, bb_nsect=3,
                                                          bb_small=True, n_bb=1, minf=minf))


@pytest.mark.parametrize("ntime,minf", [(72, 0.0), (72, 0.1), (2100, 0.1)])
def test_backward_azimuth_in_the_mixed_form(ntime, minf):
    from acum3_periodic_gb300 import native
    d = _deck(ntime, minf)
    d.dPsi = -d.dPsi
    out = []
    for ring in (0, 1):
        ctx = native.Context(0)
        ctx.set_deck(d, bb=False)
        ctx.L.acum_set_ring(ctx.h, ring)
        t = time.perf_counter()
        out.append(ctx.tonal(native.MIXED))
        assert time.perf_counter() - t < 2.0
        assert ctx.error_word() == 2
        ctx.close()
    for a, b in zip(*out):
        # the FP64 sums of several blocks add in any order
        np.testing.assert_allclose(a, b, rtol=0, atol=1e-6 * np.abs(b).max())


@pytest.mark.parametrize("name", ["", "_noalloc"])
def test_backward_rotor_in_the_drop_ins(name):
    torch = pytest.importorskip("torch")
    from acum3_periodic_gb300 import native
    fn = getattr(native.lib(), "acum_find_pressure_time_history" + name)
    d = _deck(72, 0.1)
    f = O.preprocess(d)

    def backward(*a):
        a = list(a)
        a[22] = C.c_float(-a[22].value)  # oM
        t = time.perf_counter()
        rc = fn(*a)
        assert time.perf_counter() - t < 2.0
        return rc

    assert call_dropin(fn, d, f, np.float32, torch)[0] == 0
    assert call_dropin(backward, d, f, np.float32, torch)[0] == 0
