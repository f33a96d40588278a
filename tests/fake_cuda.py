"""The library's host side on the CPU: a snippet of Python run in a process of its own with fake_cudart.c in place of
the CUDA runtime (no device, no kernel runs)."""
from __future__ import annotations

import json
import os
import subprocess
import sys
import textwrap

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PRELUDE = """
import ctypes, json, sys
import numpy as np
import adaptivemesh_gb300 as am
import cases
fake = ctypes.CDLL(None)
for f in ("fake_launches", "fake_graphs", "fake_attribute_queries"): getattr(fake, f).restype = ctypes.c_long
for f in ("fake_allocated", "fake_uploaded", "fake_copy_bytes"): getattr(fake, f).restype = ctypes.c_ulonglong
fake.fake_copy_dst.restype = ctypes.c_void_p
fake.fake_kernel.restype = ctypes.c_char_p
fake.fake_reset.argtypes = fake.fake_kernel.argtypes = [ctypes.c_long]
"""


def run(tmp_path, body: str):
    """The JSON value that the snippet prints last."""
    lib = os.path.join(str(tmp_path), "libfake_cudart.so")
    subprocess.run([os.environ.get("CC", "gcc"), "-shared", "-fPIC", "-O1", "-w", "-o", lib,
                    os.path.join(ROOT, "tests", "fake_cudart.c")], check=True)
    env = dict(os.environ, LD_PRELOAD=lib, PYTHONPATH=os.pathsep.join((ROOT, os.path.join(ROOT, "tests", "golden"))))
    r = subprocess.run([sys.executable, "-c", PRELUDE + textwrap.dedent(body)], env=env, cwd=ROOT, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr[-4000:]
    return json.loads(r.stdout.splitlines()[-1])
