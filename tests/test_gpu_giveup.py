"""Bounded waits of the column-distributed pivoted QR: a cluster that misses a message gives up,
the call reports it, and the device stays usable.

The library is built once more from a copy of its sources in which CTA 1 of a cluster never posts
its candidate column, with waits of about two milliseconds: every wait on it runs out."""
import ctypes
import os
import shutil

import numpy as np
import pytest

from alf_gb300 import _lib, build, model as mdl, rng, sweep
from alf_gb300.sweep import Chains

pytestmark = pytest.mark.gpu

POST = "if (lane < (int)CL && lane != (int)rank) qrc_push16("


@pytest.fixture(scope="module")
def silent():
    """A context in which the package's calls go to that library."""
    from device import HERE, load
    root = os.path.join(HERE, "_build", "silent")
    shutil.rmtree(root, ignore_errors=True)
    shutil.copytree(build.CSRC, os.path.join(root, "alf_gb300", "csrc"))
    shutil.copytree(os.path.dirname(_lib.HEADER), os.path.join(root, "include"))
    qr = os.path.join(root, "alf_gb300", "csrc", "qr_cols.cuh")
    with open(qr) as f:
        txt = f.read()
    assert txt.count(POST) == 1
    with open(qr, "w") as f:
        f.write(txt.replace(POST, POST.replace("(lane <", "(rank != 1 && lane <")))
    load("silent", os.path.join(root, "alf_gb300", "csrc", "alfgpu.cu"),
         ("-DQRC_WAIT_CYCLES=(1ll<<22)", "-Xptxas", "-O1"))
    path = os.path.join(HERE, "_build", "silent.so")

    class Use:
        def __enter__(self):
            self.kept = (_lib._lib, build.LIB)
            _lib._lib, build.LIB = None, path

        def __exit__(self, *a):
            _lib._lib, build.LIB = self.kept
    return Use()


def _start(L):
    m = mdl.hubbard("square", L, L, U=4.0, beta=0.4, dtau=0.1, nwrap=2)
    g = Chains(m)
    g.set_fields(0, rng.initial_fields(3, 0, m.n_op, m.ltrot))
    g.init_state()
    G = g.green(0)
    g.close()
    return G


# 4, 8 and 16 CTAs; the step's winner is the silent CTA's column (pushed to peers that have given up) or not
@pytest.mark.parametrize("L", [6, 7, 10, 12])
def test_init_state_reports_a_missing_candidate(silent, L):
    G = _start(L)
    with silent:
        for _ in range(2):
            with pytest.raises(_lib.AlfGpuError) as e:
                _start(L)
            assert e.value.code == 104
    assert np.array_equal(_start(L), G)


# the one-shot calls on host buffers: the error, and the outputs untouched
@pytest.mark.parametrize("N", [40, 100, 144])
def test_one_shot_calls_report_it(silent, N):
    r = np.random.default_rng(N)
    U = np.linalg.qr(r.standard_normal((N, N)) + 1j * r.standard_normal((N, N)))[0]
    V = np.eye(N, dtype=complex)
    D = np.exp(np.linspace(3.0, -3.0, N)).astype(complex)
    want = sweep.cgr(1, U, D, V, U, D, V), sweep.decompose("r", U, D, V)
    with silent:
        with pytest.raises(_lib.AlfGpuError) as e:
            sweep.cgr(1, U, D, V, U, D, V)
        assert e.value.code == 104
        with pytest.raises(_lib.AlfGpuError) as e:
            sweep.decompose("r", U, D, V)
        assert e.value.code == 104
        u, d, v = U.T.copy(), D.copy(), V.T.copy()
        kept = u.copy(), d.copy(), v.copy()
        p = lambda a: ctypes.c_void_p(a.ctypes.data)
        assert _lib.lib().alfgpu_decompose(N, ctypes.c_char(b"r"), p(u), p(d), p(v)) == 104
        assert all(np.array_equal(a, b) for a, b in zip((u, d, v), kept))
    (G, ph), dec = sweep.cgr(1, U, D, V, U, D, V), sweep.decompose("r", U, D, V)
    assert np.array_equal(G, want[0][0]) and ph == want[0][1]
    assert all(np.array_equal(a, b) for a, b in zip(dec, want[1]))
