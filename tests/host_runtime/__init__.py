"""The library linked with a CUDA runtime that runs nothing (runtime.cpp): what a call launches, seen on the CPU."""
import concurrent.futures
import ctypes as C
import importlib.util
import os
import shutil
import subprocess

from zignn_b200 import _lib

HERE = os.path.dirname(os.path.abspath(__file__))
REPO = os.path.dirname(os.path.dirname(HERE))


class Launch:
    def __init__(self, name, shape):
        self.name, self.grid, self.threads, self.smem, self.dependent = name, tuple(shape[:3]), shape[3], shape[4], bool(shape[5])


def build(folder):
    """Path of the library, made from the product's own objects (compiled first where they are missing or old)."""
    spec = importlib.util.spec_from_file_location("zq_build", os.path.join(REPO, "zig-nn_b200", "build.py"))
    product = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(product)
    os.makedirs(product.OBJ, exist_ok=True)
    with concurrent.futures.ThreadPoolExecutor(os.cpu_count()) as pool:
        objects = [o for o, _ in pool.map(lambda s: product._compile(s, False), product.sources())]
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(shutil.which("nvcc") or product._nvcc()))), "include")
    out = os.path.join(str(folder), "libzq_launches.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-I", include, "-o", out, os.path.join(HERE, "runtime.cpp"),
                    *objects, "-Wl,-Bsymbolic", "-Wl,--no-undefined", "-lpthread"], check=True)
    return out


class Library:
    def __init__(self, path):
        self.lib = C.CDLL(path, mode=os.RTLD_LOCAL)
        for name, (res, args) in _lib.SIGNATURES.items():
            fn = getattr(self.lib, name)
            fn.restype, fn.argtypes = res, args
        self.lib.seen_name.restype = C.c_char_p

    def launches(self, call):
        """What `call` launches, and its status."""
        self.lib.seen_clear()
        status = call()
        shape, out = (C.c_uint * 6)(), []
        for i in range(self.lib.seen_count()):
            self.lib.seen_shape(i, shape)
            out.append(Launch(self.lib.seen_name(i).decode(), shape))
        return out, status
