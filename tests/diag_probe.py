"""The diagonal wavefront's layout of a matrix (diag_probe.cc), without a GPU."""
import json
import os
import subprocess
import tempfile

import numpy as np

import mpk_gb300 as M
from conftest import ROOT

FMA, FMA_VAL, SEP, SEP_VAL, DF, DF_VAL, F32, BF16 = range(8)  # the forms
ALL, PAIR, DEEP = range(3)                                    # the modes
_exe = None


def layout(a, form, nlevel, nsm=152, smem=232448 - 1024):
    global _exe
    if _exe is None:
        _exe = os.path.join(tempfile.mkdtemp(), "diag_probe")
        cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
        subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(cuda, "include"), "-o", _exe,
                        os.path.join(ROOT, "tests", "diag_probe.cc"), M.LIB_PATH,
                        "-Wl,-rpath," + os.path.dirname(M.LIB_PATH)], check=True)
    with tempfile.NamedTemporaryFile(suffix=".csr") as f:
        for x in ([a.n], a.ptr, a.col):
            np.asarray(x, dtype=np.int32).tofile(f)
        f.flush()
        r = subprocess.run([_exe, f.name, str(form), str(nlevel), str(nsm), str(smem)], stdout=subprocess.PIPE, check=True)
    return json.loads(r.stdout)
