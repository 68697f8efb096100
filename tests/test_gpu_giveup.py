"""Bounded waits of the column-distributed pivoted QR and of the tensor-core product: a cluster (a CTA)
that misses a message gives up, the call reports it, and the device stays usable.

The library is built once more from a copy of its sources in which CTA 1 of a cluster never posts
its candidate column, and products with 77 rows never signal their end, with waits of about two
milliseconds: every wait on these runs out."""
import ctypes
import os
import shutil

import numpy as np
import pytest

from alf_gb300 import _lib, build, model as mdl, rng, sweep
from alf_gb300.sweep import Chains

pytestmark = pytest.mark.gpu

PATCHES = {"qr_cols.cuh": ("if (lane < (int)CL && lane != (int)rank) qrc_push16(",
                           "if (rank != 1 && lane < (int)CL && lane != (int)rank) qrc_push16("),
           "ozaki.cuh": ("if (oz_elect()) oz_commit(done);", "if (p.M != 77 && oz_elect()) oz_commit(done);")}


@pytest.fixture(scope="module")
def silent():
    """A context in which the package's calls go to that library."""
    from device import HERE, load
    root = os.path.join(HERE, "_build", "silent")
    shutil.rmtree(root, ignore_errors=True)
    shutil.copytree(build.CSRC, os.path.join(root, "alf_gb300", "csrc"))
    shutil.copytree(os.path.dirname(_lib.HEADER), os.path.join(root, "include"))
    for name, (old, new) in PATCHES.items():
        path = os.path.join(root, "alf_gb300", "csrc", name)
        with open(path) as f:
            txt = f.read()
        assert txt.count(old) == 1
        with open(path, "w") as f:
            f.write(txt.replace(old, new))
    load("silent", os.path.join(root, "alf_gb300", "csrc", "alfgpu.cu"),
         ("-DQRC_WAIT_CYCLES=(1ll<<22)", "-DOZ_WAIT_CYCLES=(1ll<<22)", "-Xptxas", "-O1"))
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


# one and several tiles, one and several K chunks; a product with another row count ends as ever
@pytest.mark.parametrize("n,k", [(5, 9), (300, 200), (64, 448)])
def test_products_report_a_missing_end(silent, n, k):
    r = np.random.default_rng(n + k)

    def product(m):
        A, B = np.asfortranarray(r.standard_normal((m, k))), np.asfortranarray(r.standard_normal((k, n)))
        C = np.full((m, n), 7.0, order="F")
        p = lambda a: ctypes.c_void_p(a.ctypes.data)
        rc = _lib.lib().alfgpu_oz_dgemm(m, n, k, p(A), m, p(B), k, p(C), m, 0)
        return rc, C, A @ B

    with silent:
        rc, C, _ = product(77)
        assert rc == 104 and np.all(C == 7.0)
        rc, C, want = product(78)
        assert rc == 0 and np.max(np.abs(C - want)) < 1e-12 * k
    rc, C, want = product(77)
    assert rc == 0 and np.max(np.abs(C - want)) < 1e-12 * k
