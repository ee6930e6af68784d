"""Runs a piece of Python in a process whose CUDA runtime is tests/fake_cudart.c:
device memory on the host, kernels that do nothing, every call noted."""
import json
import os
import subprocess
import sys
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]
PRELUDE = f"""
import ctypes, json, sys
sys.path[:0] = [{str(ROOT)!r}, {str(ROOT / 'tests')!r}]
import numpy as np
from lymph3d_apsc_gb300 import MatrixFree, _lib, ensemble as E, mesh as M
from lymph3d_apsc_gb300._lib import LymphError
fake = ctypes.CDLL(None)
fake.fake_log.restype = ctypes.c_char_p
def calls():
    return fake.fake_log().decode()
def out(x):
    print("OUT " + json.dumps(x))
"""


def run(code, tmp_path, **env):
    """What `code` passed to out(), in order."""
    so = tmp_path / "fake_cudart.so"
    if not so.exists():
        subprocess.run(["gcc", "-O1", "-shared", "-fPIC", "-o", str(so), str(ROOT / "tests" / "fake_cudart.c")], check=True)
    e = dict(os.environ, LD_PRELOAD=str(so), LYMPH_TUNE_CACHE=str(tmp_path / "tune.txt"), **env)
    r = subprocess.run([sys.executable, "-c", PRELUDE + code], env=e, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-3000:]
    return [json.loads(line[4:]) for line in r.stdout.splitlines() if line.startswith("OUT ")]
