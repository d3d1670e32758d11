"""Runs Python code against the library with the CUDA runtime of
fake_cudart.c in front of the real one, and returns its log: the host side of
plans and calls without a GPU."""
import os
import subprocess
import sys

from conftest import ROOT

HEAD = """
import ctypes as C, sys
sys.path.insert(0, {root!r})
import numpy as np
import mpk_gb300 as M
fake = C.CDLL(None)
fake.fake_limit.argtypes = [C.c_size_t]
fake.fake_live.restype = fake.fake_peak.restype = C.c_size_t
fake.fake_upload.argtypes, fake.fake_upload.restype = [C.c_size_t, C.c_int], C.c_void_p
def upload(count, dtype, back=0):
    p = fake.fake_upload(count * np.dtype(dtype).itemsize, back)
    return np.ctypeslib.as_array((C.c_byte * (count * np.dtype(dtype).itemsize)).from_address(p)).view(dtype)
def mark(s): fake.fake_mark(s.encode())
def live(): return int(fake.fake_live())
def peak(): return int(fake.fake_peak())
def raises(code, f):
    try: f()
    except M.MpkError as e:
        assert e.code == code, e
        return
    raise AssertionError("no error")
"""


def run(tmp, code):
    """The log's lines, split into words; what the code prints is in out.txt."""
    so = os.path.join(tmp, "libfake_cudart.so")
    if not os.path.exists(so):
        cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
        subprocess.run(["gcc", "-O1", "-w", "-shared", "-fPIC", "-I", os.path.join(cuda, "include"), "-o", so,
                        os.path.join(ROOT, "tests", "fake_cudart.c")], check=True)
    log = os.path.join(tmp, "log.txt")
    if os.path.exists(log):
        os.remove(log)
    r = subprocess.run([sys.executable, "-c", HEAD.format(root=ROOT) + code], stdout=subprocess.PIPE,
                       stderr=subprocess.STDOUT, text=True, timeout=300,
                       env={**os.environ, "LD_PRELOAD": so, "FAKE_CUDART_LOG": log})
    assert r.returncode == 0, r.stdout
    with open(os.path.join(tmp, "out.txt"), "w") as f:
        f.write(r.stdout)
    return [line.split() for line in open(log)]


def launches(log):
    """(kernel, blocks, threads, dynamic shared memory, stream) of every launch."""
    return [(w[1], int(w[2]), int(w[3]), int(w[4]), w[5]) for w in log if w[0] == "launch"]
