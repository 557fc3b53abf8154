"""The library's host code on a stub of the CUDA runtime (tests/host), for what a
GPU is not needed for: built once per session, used from child processes so that a
crash is one test's failure."""
import concurrent.futures
import os
import subprocess
import sys
import textwrap

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "piko-public_b200", "csrc")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")


def build(out):
    """Every host source unoptimised (an operation whose result goes unused stays in),
    device code only as far as the launches need its registration."""
    host = os.path.join(ROOT, "tests", "host")
    jobs = []
    for src in ["runtime.cu", "raster_kernels.cu", "server.cu", "tuner.cu", "noalloc.cu", "assets.cpp"]:
        jobs.append(os.path.join(CSRC, src))
    jobs += [os.path.join(host, "decode.cu"), os.path.join(host, "cuda_stub.cpp")]   # (decode.cu holds reyes_kernels.cu)

    def compile_one(src):
        obj = os.path.join(out, os.path.basename(src) + ".o")
        subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=compute_100a", "-O0", "-Xcicc", "-O0", "-std=c++17",
                        "--fmad=false", "-Xcompiler", "-fPIC", "-I", os.path.join(ROOT, "include"), "-c", "-o", obj, src],
                       check=True)
        return obj

    with concurrent.futures.ThreadPoolExecutor(os.cpu_count()) as pool:
        objs = list(pool.map(compile_one, jobs))
    lib = os.path.join(out, "libpiko_host.so")
    subprocess.run(["g++", "-shared", "-Wl,-Bsymbolic", "-o", lib] + objs + ["-lpthread"], check=True)
    return lib


PRELUDE = """
import ctypes, sys
import numpy as np
sys.path.insert(0, {root!r})
import piko_loader
pk = piko_loader.load()
lib = pk.load_library({lib!r})
lib.stub_stream.restype = lib.stub_end_capture.restype = ctypes.c_void_p
for f in ["stub_destroy_stream", "stub_begin_capture", "stub_end_capture"]:
    getattr(lib, f).argtypes = [ctypes.c_void_p]
lib.stub_replay.argtypes = [ctypes.c_void_p, ctypes.c_void_p]

def log():
    b = ctypes.create_string_buffer(1 << 20)
    lib.stub_log(b, len(b))
    return b.value.decode().splitlines()

def tri_scene(W=96, H=64, n=40, seed=1):
    return pk.scenes.plain_scene(n=n, W=W, H=H, seed=seed)

def camera(x):
    vp = np.eye(4, dtype=np.float32).reshape(16).copy()
    vp[12] = x
    return pk.const_state(view_proj=vp)

ctx = pk.Context()
"""


def run(lib, code):
    """Runs code after PRELUDE in a child process; returns what it printed."""
    script = PRELUDE.format(root=ROOT, lib=lib) + textwrap.dedent(code)
    p = subprocess.run([sys.executable, "-c", script], capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, f"exit status {p.returncode}\n{p.stdout}{p.stderr}"
    return p.stdout
