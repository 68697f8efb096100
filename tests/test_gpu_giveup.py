"""Bounded waits of the column-distributed pivoted QR: a cluster that misses a message gives up,
the call reports it, and the device stays usable.

The library is built once more from a copy of its sources in which CTA 1 of a cluster never posts
its candidate column, with waits of about two milliseconds: every wait on it runs out."""
import os
import shutil

import numpy as np
import pytest

from alf_gb300 import _lib, build, model as mdl, rng
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
