"""Solves on a stand-in for the CUDA runtime (tests/cpp/fake_cudart.cpp): what the host code launches, and what it
answers when a call of the runtime is refused, without a GPU. run() makes the solves in a process of its own."""
import json
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "tests", "cpp", "fake_cudart.cpp")


def kernels(tmp_path):
    """The kernels that the library holds."""
    return json.loads(_child(tmp_path, "kernels"))


def run(tmp_path, *cases):
    """A case: material, shells, bands, k, and optionally plane_waves (the first so many of the basis), nl, soc, mixed,
    vectors, tuning, autotune, refuse. Returns for each its error
    (None: it was solved), its launches (kernel, grid, threads, shared memory) and the shared-memory limits set."""
    out = []
    for error, log in json.loads(_child(tmp_path, json.dumps(cases))):
        lines = [x.split() for x in log.splitlines()]
        out.append((error, [(x[1], *map(int, x[2:])) for x in lines if x[0] == "launch"],
                    [(x[1], int(x[2])) for x in lines if x[0] == "smem"]))
    return out


def _child(tmp_path, what):
    from ultimateepm_gb300 import build

    lib = os.path.join(str(tmp_path), "libfake_cudart.so")
    if not os.path.exists(lib):
        inc = os.path.join(build._cuda_home(), "include")
        subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I" + inc, SRC, "-o", lib], check=True)
    r = subprocess.run([sys.executable, os.path.abspath(__file__), what], env=dict(os.environ, LD_PRELOAD=lib, PYTHONPATH=ROOT),
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    return r.stdout


def _solve(c, fake):
    import ctypes as C

    import numpy as np

    from ultimateepm_gb300 import _native as N
    from ultimateepm_gb300 import api

    ms = api.Materials()
    ms.load_material_parameters(os.path.join(ROOT, "params", "materials.yaml"))
    ctx = api._Context(ms.materials[c["material"]], api.generate_basis_vectors(c["shells"])[:c.get("plane_waves")], c.get("nl", False), c.get("soc", False),
                       N.UEPM_PREC_MIXED if c.get("mixed") else N.UEPM_PREC_FP64)
    N.check(N.load().uepm_ctx_set_tuning(ctx.h, C.byref(N.UepmTuning(**c.get("tuning", {})))))
    fake.fake_clear()
    if "autotune" in c:
        N.check(N.load().uepm_ctx_autotune(ctx.h, c["bands"], N.UEPM_WANT_VALUES, c["autotune"], None))
    fake.fake_refuse(c.get("refuse", "").encode())
    error = None
    try:
        ctx.solve(np.full((c["k"], 3), 0.1), c["bands"], vectors=c.get("vectors", False))
    except (RuntimeError, ValueError, IndexError) as e:
        error = str(e)
    log = fake.fake_log().decode()
    fake.fake_refuse(b"")
    ctx.close()
    return error, log


if __name__ == "__main__":
    import ctypes

    fk = ctypes.CDLL(None)
    fk.fake_log.restype = ctypes.c_char_p
    fk.fake_kernels.restype = ctypes.c_char_p
    if sys.argv[1] == "kernels":
        from ultimateepm_gb300 import _native

        _native.load()
        print(json.dumps(fk.fake_kernels().decode().split()))
    else:
        print(json.dumps([_solve(c, fk) for c in json.loads(sys.argv[1])]))
