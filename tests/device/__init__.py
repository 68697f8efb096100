"""Test-only device code: small CUDA sources over the library's headers, compiled on first use."""
import ctypes
import os
import subprocess

from alf_gb300 import build

HERE = os.path.dirname(os.path.abspath(__file__))


def load(name, source=None, flags=()):
    """The shared library of `source` (default: <name>.cu here), rebuilt when a header is newer."""
    src = source or os.path.join(HERE, name + ".cu")
    out = os.path.join(HERE, "_build", name + ".so")
    os.makedirs(os.path.dirname(out), exist_ok=True)
    if not os.path.exists(out) or any(os.path.getmtime(s) > os.path.getmtime(out) for s in [src, *build.sources()]):
        subprocess.check_call([build.nvcc(), *build.ARCH, "-O3", "-std=c++17", "--extended-lambda", *flags, "-Xcompiler",
                               "-fPIC,-ffp-contract=off", "-shared", "-o", out + ".tmp", src])
        os.replace(out + ".tmp", out)
    return ctypes.CDLL(out)
