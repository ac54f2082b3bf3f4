"""Runs Python programs whose libmpsq sees the stand-in of the CUDA runtime (tests/fake_cudart.c)."""
import os
import subprocess
import sys
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent
HEAD = r"""
import ctypes as C
import sys
import numpy as np
sys.path.insert(0, %r)
fake = C.CDLL(%r)
fake.fake_held.restype = fake.fake_most.restype = fake.fake_launches.restype = C.c_int64
fake.fake_default_threshold.restype = C.c_uint64
fake.fake_set_capacity.argtypes = [C.c_int64]
from mp_tools_gb300 import _lib
from mp_tools_gb300.sqom import QGrid, SqomJob, TimeAxis
_lib.load(build_if_missing=False)
"""


def run(tmp_path, program: str) -> str:
    """The program's output; it finds `fake`, np, _lib, QGrid, SqomJob and TimeAxis."""
    so = Path(tmp_path) / "libfake_cudart.so"
    subprocess.run(["gcc", "-O1", "-Wall", "-Werror", "-fPIC", "-shared", "-o", str(so),
                    str(ROOT / "tests" / "fake_cudart.c")], check=True)
    r = subprocess.run([sys.executable, "-c", HEAD % (str(ROOT), str(so)) + program], capture_output=True,
                       text=True, timeout=300, env=dict(os.environ, LD_PRELOAD=str(so)))
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout
