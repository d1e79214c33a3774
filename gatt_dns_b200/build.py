"""Build recipe of the CUDA library (nvcc, sm_100a) -- ``python -m gatt_dns_b200.build``."""
from __future__ import annotations

import glob
import os
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OUT = os.path.join(HERE, "libgatt_dns_b200.so")

NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-lineinfo", "-std=c++17",
              "-Xcompiler", "-fPIC"]


def sources():
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def headers():
    return sorted(glob.glob(os.path.join(CSRC, "*.cuh"))) + [os.path.join(HERE, "..", "include", "gatt_dns.h")]


def needs_build():
    if not os.path.exists(OUT):
        return True
    t = os.path.getmtime(OUT)
    return any(os.path.getmtime(p) > t for p in sources() + headers() if os.path.exists(p))


def build(force=False, verbose=False):
    """Compile the sources side by side and link them into the library."""
    if not force and not needs_build():
        return OUT
    nvcc = os.environ.get("NVCC", "nvcc")
    flags = (["-Xptxas=-v"] if verbose else []) + NVCC_FLAGS
    objs = [os.path.join(HERE, "build", os.path.basename(p) + ".o") for p in sources()]
    os.makedirs(os.path.join(HERE, "build"), exist_ok=True)
    # a source is compiled again when it or any header changed
    newest = max(os.path.getmtime(p) for p in headers() if os.path.exists(p))
    stale = [(src, obj) for src, obj in zip(sources(), objs)
             if force or not os.path.exists(obj) or max(newest, os.path.getmtime(src)) > os.path.getmtime(obj)]
    with ThreadPoolExecutor(max_workers=os.cpu_count() or 1) as pool:
        list(pool.map(lambda so: subprocess.run([nvcc] + flags + ["-c", "-o", so[1], so[0]], check=True), stale))
    subprocess.run([nvcc] + NVCC_FLAGS + ["-shared", "-o", OUT] + objs, check=True)
    return OUT


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
