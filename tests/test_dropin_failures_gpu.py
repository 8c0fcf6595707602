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


AFTER_RESET = """
import ctypes as C, glob, os, sys
sys.path[:0] = [%r, %r]
import numpy as np
from acum3_periodic_gb300 import native
from test_dropin_workspaces_gpu import _bb_call, _bb_deck
rt = C.CDLL(sorted(glob.glob(os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "lib64", "libcudart.so*")))[0])
d = _bb_deck(1, 70, 7, 3)
rng = np.random.default_rng(0)
rows = [rng.standard_normal((3, 40, w)) for w in (4, 6, 6, 6, 4)]
def per():
    return native.preprocess_per([3], *[r.copy() for r in rows], 1e-4, 340.0, 1.2, 0.5, 1.0)
first = _bb_call(d), per()
for _ in range(2):
    assert rt.cudaDeviceReset() == 0
    again = _bb_call(d), per()
    for a, b in zip(first, again):
        for x, y in zip(a, b):
            np.testing.assert_array_equal(x, y)
"""


def test_after_a_device_reset():
    """What the calls keep belongs to a CUDA context; after a reset they start anew."""
    import os
    import subprocess
    import sys
    from conftest import ROOT
    r = subprocess.run([sys.executable, "-c", AFTER_RESET % (ROOT, os.path.join(ROOT, "tests"))],
                       stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=300)
    assert r.returncode == 0, r.stdout


def test_workspaces_are_given_back():
    """An allocation of the library that fails frees what idle calls keep; they allocate it again."""
    torch = pytest.importorskip("torch")
    from acum3_periodic_gb300 import native
    from test_dropin_workspaces_gpu import _bb_call
    d = synth.config_deck(1, replicate=730, scale=dict(n_span=1, n_chord_side=2, ntime=720, nobs=9, bb_nsect=50,
                                                       bb_small=True, n_bb=4))
    first = _bb_call(d)
    ctx = native.Context(0)
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    # 3.2 million elements x 4096 steps: more rows than the device holds, refused before any is read
    ins = native.inputs_of(d)
    ins.nTime = 4096
    ne = np.array([3200000], np.int32)
    obs = np.ones(3, np.float32)
    rc = ctx.L.acum_set_deck(ctx.h, C.byref(ins), 1, obs.ctypes.data_as(C.POINTER(C.c_float)), 1,
                             ne.ctypes.data_as(C.POINTER(C.c_int)), obs.ctypes.data_as(C.POINTER(C.c_float)), 0)
    assert rc == -4  # ACUM_ERR_NOMEM
    # 200 sections x 720 steps: 42 bands x 8 amplitudes alone are 193 MB
    assert torch.cuda.mem_get_info()[0] - free0 > 190 << 20
    ctx.close()
    for a, b in zip(_bb_call(d), first):
        np.testing.assert_array_equal(a, b)
