"""The CUDA kernels of quarz_b200/csrc compiled for the host, for tests of what a GPU must not be given to find out:
accesses out of range and missing barriers. `library()` compiles the C ABI, the sweeps, the beam and the adjoint kernels with g++
against host_cuda/cuda_runtime.h (which runs a block's threads as fibers) and returns the ctypes library: the entry
points of include/qz_b200.h on host memory (numpy arrays where a GPU caller passes device pointers), and
`schedule()`, which warps run first. Runs and adjoints go step by step: no pipelined or batched ones.
"""
import ctypes as C
import hashlib
import os
import re
import shutil
import subprocess
import tempfile

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "quarz_b200", "csrc")
EMU = os.path.join(ROOT, "tests", "host_cuda")
UNITS = ["qz_abi.cu", "qz_beam.cu", "qz_sweep.cu", "qz_sweep_m1.cu", "qz_adjoint.cu"]
HEADERS = ["qz_device.cuh", "qz_internal.h", "qz_beam_body.cuh", "qz_sweep_body.cuh", "qz_sweep_m1_body.cuh"]
# (PTX of the kernels, what the host does instead)
PTX = [
    (r'asm volatile\("bar\.sync %0, %1;" ::"r"\(id\), "r"\(threads\) : "memory"\);', "emu::meet(emu::barrier(id), threads);"),
    (r'asm volatile\("prefetch\.global\.L2 \[%0\];" ::"l"\(nx \+ o\)\);', "(void)nx;"),
    (r'asm\("mov\.u32 %0, %%cluster_ctarank;" : "=r"\(t\.rank\)\);', "t.rank = blockIdx.x;"),
    (r'asm\("mov\.u32 %0, %%cluster_nctarank;" : "=r"\(t\.size\)\);', "t.size = emu::cluster_size();"),
    (r'asm volatile\("barrier\.cluster\.arrive[^;]*;" ::: "memory"\);', ""),
    (r'asm volatile\("barrier\.cluster\.wait[^;]*;" ::: "memory"\);',
     "emu::meet(emu::cluster_barrier(), size * emu::block_threads());"),
    (r'asm volatile\("mapa\.shared::cluster.*?\);\n', "r = a;\n"),
    (r'asm volatile\("ld\.shared::cluster.*?\);\n',
     "v = *(const int*)((const char*)emu::dyn_smem_of(0) + ((const char*)p - (const char*)emu::dyn_smem()));\n"),
    (r"__cvta_generic_to_shared\(p\)", "0"),
    # (the pipelined reverse pass is not run: a launch of it is an error)
    (r'asm volatile\("ld\.acquire.*?\);\n', "v = *p;\n"),
    (r'asm volatile\("st\.release.*?\);\n', "*p = v;\n"),
    (r'asm volatile\("mov\.u64 %0, %%globaltimer;".*?\);\n', "t = 0;\n"),
    (r"\b__noinline__\b", ""),
]


def _host_source(text: str) -> str:
    for ptx, host in PTX:
        text = re.sub(ptx, host, text)
    code = re.sub(r"//[^\n]*", "", text)
    assert not re.search(r"\basm\b", code), "inline PTX without a host counterpart (PTX above)"
    text = text.replace("extern __shared__ double smem_raw[];", "double* smem_raw = emu::dyn_smem();")
    text = re.sub(r"([\w:]+(?:<[\w, ]*>)?)<<<([^;]*?)>>>\(([^;]*?)\);", r"emu::launch4([&] { \1(\3); }, \2);", text)
    return text


def _build(out: str) -> None:
    tmp = out + ".build"
    shutil.rmtree(tmp, ignore_errors=True)
    os.makedirs(tmp)
    for name in UNITS + HEADERS:
        with open(os.path.join(CSRC, name)) as f, open(os.path.join(tmp, name.replace(".cu", ".cpp") if name in UNITS
                                                                    else name), "w") as g:
            g.write(_host_source(f.read()))
    flags = ["g++", "-std=c++17", "-O1", "-w", "-fPIC", "-I", EMU, "-I", tmp, "-I", os.path.join(ROOT, "include")]
    srcs = [os.path.join(tmp, n.replace(".cu", ".cpp")) for n in UNITS] + [os.path.join(EMU, "emu.cpp")]
    objs = [os.path.join(tmp, os.path.basename(s)[:-4] + ".o") for s in srcs]
    jobs = [subprocess.Popen(flags + ["-c", s, "-o", o], stderr=subprocess.PIPE, text=True) for s, o in zip(srcs, objs)]
    for j in jobs:
        err = j.communicate()[1]
        assert j.returncode == 0, err[-4000:]
    # the launches of the units left out: an error of the call
    nm = subprocess.run(["nm", "-u"] + objs, capture_output=True, text=True, check=True).stdout
    have = subprocess.run(["nm", "--defined-only"] + objs, capture_output=True, text=True, check=True).stdout
    have = {line.split()[-1] for line in have.splitlines() if len(line.split()) == 3}
    with open(os.path.join(tmp, "rest.s"), "w") as f:
        f.write('.section .note.GNU-stack,"",@progbits\n.text\n')
        for sym in sorted({s for s in re.findall(r"U (_ZN3qzb\w+)", nm)} - have):
            f.write(f".globl {sym}\n{sym}:\n mov $1, %eax\n ret\n")
    subprocess.run(["g++", "-shared", "-o", out + ".part", *objs, os.path.join(tmp, "rest.s")], check=True)
    os.replace(out + ".part", out)
    shutil.rmtree(tmp, ignore_errors=True)


_lib = None


def library():
    global _lib
    if _lib is None:
        h = hashlib.sha256()
        for path in [os.path.join(CSRC, n) for n in UNITS + HEADERS] + [__file__] + \
                [os.path.join(EMU, n) for n in ("cuda_runtime.h", "emu.cpp")] + [os.path.join(ROOT, "include", "qz_b200.h")]:
            with open(path, "rb") as f:
                h.update(f.read())
        out = os.path.join(tempfile.gettempdir(), f"libqz_host_{h.hexdigest()[:16]}.so")
        if not os.path.exists(out):
            _build(out)
        from quarz_b200 import _lib as L

        _lib = C.CDLL(out)
        for name, args in L.SIGNATURES.items():
            getattr(_lib, name).argtypes = args
        _lib.qz_last_error.restype = C.c_char_p
    return _lib


def schedule(first=(), keep=True):
    """The warps to resume first, in this order (with keep: each as far as it can go before a later one)."""
    a = np.asarray(list(first), dtype=np.int32)
    library().emu_schedule(a.ctypes.data_as(C.POINTER(C.c_int)), len(a), int(keep))


def check(rc):
    if rc:
        raise RuntimeError(library().qz_last_error().decode())


def ptr(a):
    """The address of a numpy array, where a GPU caller passes a device pointer."""
    return a.ctypes.data_as(C.c_void_p)


def available():
    import platform

    return shutil.which("g++") is not None and platform.machine() == "x86_64"
