"""Build libminuet_b200.so (nvcc, sm_100a) and the native host path _host.so (g++ against
the installed torch) in-tree.

Run as ``python -m minuet_b200.build`` (or through ``__graft_entry__.build()``).
The shared objects land next to this file so that they travel with the source
tree; nothing is written outside the package directory.
"""
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OUT = os.path.join(HERE, "libminuet_b200.so")
HOST_SRC = os.path.join(CSRC, "host.cpp")
HOST_OUT = os.path.join(HERE, "_host.so")
HEADER = os.path.join(HERE, "..", "include", "minuet_b200.h")
SOURCES = ["mn_api.cu", "mn_map_keys.cu", "mn_map_sort.cu", "mn_map_query.cu", "mn_gms.cu",
           "mn_gemm_tc.cu", "mn_conv_implicit.cu", "mn_conv_pairs.cu", "mn_conv_simt.cu",
           "mn_conv_wgrad.cu", "mn_voxel.cu"]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-lineinfo",
              "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC", "-Xcompiler", "-Wall"]


def _older(out: str, deps) -> bool:
    if not os.path.exists(out):
        return True
    t = os.path.getmtime(out)
    return any(os.path.getmtime(d) > t for d in deps)


def _host_command():
    import sysconfig

    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    lib = os.path.join(root, "lib")
    return ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
            "-DTORCH_EXTENSION_NAME=_host",
            f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
            "-I" + os.path.join(root, "include"),
            "-I" + os.path.join(root, "include", "torch", "csrc", "api", "include"),
            "-I" + os.path.join(cuda, "include"), "-I" + sysconfig.get_paths()["include"],
            HOST_SRC, "-o", HOST_OUT, "-L" + lib, "-lc10", "-lc10_cuda", "-ltorch_cpu",
            "-ltorch_cuda", "-ltorch", "-ltorch_python", "-L" + os.path.join(cuda, "lib64"),
            "-lcudart", "-ldl", "-Wl,-rpath," + lib]


def build(force: bool = False, verbose: bool = False) -> str:
    kernels = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh"))]
    do_lib = force or _older(OUT, kernels + [HEADER])
    do_host = force or _older(HOST_OUT, [HOST_SRC, HEADER])
    procs = []
    objs = []
    if do_host:
        procs.append(("host.cpp", subprocess.Popen(_host_command(), stdout=subprocess.PIPE,
                                                   stderr=subprocess.STDOUT)))
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    if do_lib:
        obj_dir = os.path.join(HERE, "_obj")
        os.makedirs(obj_dir, exist_ok=True)
        for src in SOURCES:
            obj = os.path.join(obj_dir, src.replace(".cu", ".o"))
            objs.append(obj)
            cmd = [nvcc, *NVCC_FLAGS, "-c", os.path.join(CSRC, src), "-o", obj]
            if verbose:
                cmd.insert(1, "-Xptxas")
                cmd.insert(2, "-v")
            procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE,
                                                stderr=subprocess.STDOUT)))
    failed = False
    for src, p in procs:
        out, _ = p.communicate()
        text = out.decode()
        if p.returncode != 0 or verbose:
            sys.stderr.write(f"--- {src}\n{text}\n")
        failed |= p.returncode != 0
    if failed:
        raise RuntimeError("the compiler failed; see the log above")
    if do_lib:
        subprocess.check_call([nvcc, "-shared", "-o", OUT, *objs, "-lcudart", "-lcuda"])
    return OUT


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
