"""What the reference-shaped calls do after, and beside, calls that fail."""
import ctypes as C

import numpy as np
import pytest

from acum3_periodic_gb300 import synth
from oracle import oracle as O

from test_dropin_gpu import call_dropin

pytestmark = pytest.mark.gpu


def _deck(k=0, **scale):
    return synth.config_deck(0, replicate=700 + k, scale=dict(dict(n_span=2, n_chord_side=2, ntime=40, nobs=3), **scale))


@pytest.mark.parametrize("name,dtype", [("noalloc", np.float32), ("", np.float32), ("f64", np.float64)])
def test_after_a_failed_allocation(name, dtype):
    """An allocation that failed on the same thread (the reason to turn to the allocation-free
    entry point) is that call's error, not the next one's."""
    torch = pytest.importorskip("torch")
    from acum3_periodic_gb300 import native
    L = native.lib()
    fn = getattr(L, "_".join(["acum_find_pressure_time_history"] + [name] * bool(name)))
    d = _deck()
    f = O.preprocess(d)
    rc, *ref = call_dropin(fn, d, f, dtype, torch)
    assert rc == 0

    def failed_first(*a):
        p = C.c_void_p()
        assert L.acum_host_alloc(C.byref(p), 1 << 60) != 0
        return fn(*a)

    rc, *got = call_dropin(failed_first, d, f, dtype, torch)
    assert rc == 0
    for a, b in zip(got, ref):
        # the FP64 sums of several blocks add in any order
        np.testing.assert_allclose(a, b, rtol=0, atol=1e-6 * np.abs(b).max())


@pytest.mark.parametrize("name,dtype", [("", np.float32), ("_f64", np.float64)])
def test_beside_refused_calls(name, dtype):
    """A call whose period no kernel holds is refused with nothing of it left running on the
    workspaces: calls on another stream give what they give alone."""
    torch = pytest.importorskip("torch")
    import threading
    from acum3_periodic_gb300 import native
    fn = getattr(native.lib(), "acum_find_pressure_time_history" + name)
    good, long = _deck(1, n_span=6, n_chord_side=5, ntime=90, nobs=20), _deck(2, n_span=1, nobs=2, ntime=40000)
    f = O.preprocess(good)
    x = np.zeros((long.E, long.nTime, 18))
    x[:, :, 0] = 1.0

    def on(stream, repeat):
        def call(*a):
            torch.cuda.synchronize()
            rcs = [fn(*a[:-1], C.c_void_p(stream.cuda_stream)) for _ in range(repeat)]
            return rcs[0] if len(set(rcs)) == 1 else None
        return call

    rc, *ref = call_dropin(on(torch.cuda.Stream(), 1), good, f, dtype, torch)
    assert rc == 0
    refused = []
    t = threading.Thread(target=lambda: refused.append(
        call_dropin(on(torch.cuda.Stream(), 200), long, x, dtype, torch)[0]))
    t.start()
    s = torch.cuda.Stream()
    got = [call_dropin(on(s, 1), good, f, dtype, torch) for _ in range(40)]
    t.join()
    assert refused == [-3]
    for rc, *out in got:
        assert rc == 0
        for a, b in zip(out, ref):
            np.testing.assert_allclose(a, b, rtol=0, atol=1e-6 * np.abs(b).max())
