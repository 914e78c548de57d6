"""Builds the CUDA test harnesses of this folder: shipped translation units
with C entries around single kernels."""
import ctypes
import os
import subprocess

from aeroflex_gb300 import build as afx_build

HERE = os.path.dirname(os.path.abspath(__file__))


def load(name, out_dir, unit):
    """Compile <name>.cu with the flags that the shipped unit is compiled with."""
    units, _ = afx_build._units()
    flags = [f for f, src in units if src == unit][0]
    so = os.path.join(str(out_dir), name + ".so")
    cmd = [f for f in flags if f != "-c"] + ["-shared", os.path.join(HERE, name + ".cu"), "-o", so]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    return ctypes.CDLL(so)
