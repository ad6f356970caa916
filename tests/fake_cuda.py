"""Runs Python code against the built library over a CUDA runtime without a
device (fake_cudart.c), in a process of its own."""
import os
import shutil
import subprocess
import sys

import pytest

from conftest import PKG, ROOT

PRELUDE = """
import ctypes, os, sys
sys.path.insert(0, os.environ["FQ_PKG"])
import numpy as np
import forqaoa as fq
fake = ctypes.CDLL(os.environ["FQ_FAKE"])
def log():
    buf = ctypes.create_string_buffer(1 << 20)
    fake.fake_log.restype = ctypes.c_size_t
    n = fake.fake_log(buf, ctypes.c_size_t(len(buf)))
    return buf.raw[:n].decode().splitlines()
def graph(n, seed=1):
    return np.triu(np.random.default_rng([n, seed]).integers(1, 11, (n, n)).astype(float), 1)
"""


def run(code, tmp_path, timeout=60):
    """Runs `code` after PRELUDE; returns what it printed."""
    cc = shutil.which("gcc") or shutil.which("cc")
    if cc is None:
        pytest.skip("no C compiler")
    fake = os.path.join(tmp_path, "fake_cudart.so")
    src = os.path.join(ROOT, "tests", "fake_cudart.c")
    subprocess.run([cc, "-O1", "-shared", "-fPIC", "-w", "-o", fake, src, "-lpthread"], check=True)
    env = dict(os.environ, LD_PRELOAD=fake, FQ_FAKE=fake, FQ_PKG=PKG)
    p = subprocess.run([sys.executable, "-c", PRELUDE + code], env=env, timeout=timeout,
                       capture_output=True, text=True)
    assert p.returncode == 0, p.stderr[-3000:]
    return p.stdout
