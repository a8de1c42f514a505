"""Build libfa_b200.so for sm_100a with bare nvcc (no torch headers needed), and fa_b200_torch.so, the native autograd
operator on top of it (torch_op.cpp: host code, torch's headers).

Usage: python build.py [--force] [--verbose]
The library lands in ../flash_attention_v100/lib/ so it travels with the package.
"""
import os
import re
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
OUT_DIR = os.path.join(os.path.dirname(HERE), "flash_attention_v100", "lib")
OUT = os.path.join(OUT_DIR, "libfa_b200.so")
OP_OUT = os.path.join(OUT_DIR, "fa_b200_torch.so")
OP_SOURCE = "torch_op.cpp"
SOURCES = ["host_api.cu", "simt_kernels.cu", "fwd_sm100.cu", "fwd_tf32_sm100.cu", "bwd_sm100.cu", "bwd_f32_sm100.cu", "combine.cu", "compact.cu",
           "fwd_pair_sm100.cu", "bwd_pair_sm100.cu"]
HEADERS = ["fa_common.cuh", "philox.cuh", "sm100_ptx.cuh", "tma_host.cuh", "tile_config.cuh",
           os.path.join("..", "..", "include", "fa_b200.h")]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "--use_fast_math", "-Xptxas", "-v",
]


def _newest(paths):
    return max((os.path.getmtime(p) for p in paths if os.path.exists(p)), default=0.0)


def _installed_torch():
    """Folder and version of the torch that Python would import, without importing it."""
    import importlib.util
    folder = os.path.dirname(importlib.util.find_spec("torch").origin)
    with open(os.path.join(folder, "version.py")) as f:
        return folder, re.search(r"^__version__\s*=\s*['\"]([^'\"]+)", f.read(), re.M).group(1)


def _op_command():
    import sysconfig
    torch_dir, version = _installed_torch()
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    return ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", f'-DFA_TORCH_VERSION="{version}"',
            f"-I{torch_dir}/include", f"-I{torch_dir}/include/torch/csrc/api/include",
            f"-I{cuda}/include", f"-I{sysconfig.get_paths()['include']}", os.path.join(HERE, OP_SOURCE), "-o", OP_OUT,
            f"-L{torch_dir}/lib", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda", "-ltorch_python",
            f"-L{OUT_DIR}", "-lfa_b200", "-Wl,-rpath,$ORIGIN"]


def build_op(force=False):
    """The native operator; after the library, which it is linked against.  Built again when its sources are newer or the
    command is another one (another torch, another Python): it is laid out for the torch it was built with."""
    deps = [os.path.join(HERE, OP_SOURCE), os.path.join(HERE, "..", "..", "include", "fa_b200.h"), os.path.abspath(__file__)]
    cmd = _op_command()
    built_by = OP_OUT + ".cmd"
    same = False
    if os.path.exists(built_by):
        with open(built_by) as f:
            same = f.read() == " ".join(cmd)
    if not force and same and os.path.exists(OP_OUT) and os.path.getmtime(OP_OUT) >= _newest(deps):
        return OP_OUT
    r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if r.returncode != 0:
        sys.stderr.write(" ".join(cmd) + "\n" + r.stdout)
        raise RuntimeError("building the native operator failed")
    with open(built_by, "w") as f:
        f.write(" ".join(cmd))
    return OP_OUT


def build(force=False, verbose=False):
    lib = build_library(force, verbose)
    build_op(force)
    return lib


def build_library(force=False, verbose=False):
    os.makedirs(OUT_DIR, exist_ok=True)
    srcs = [os.path.join(HERE, s) for s in SOURCES]
    deps = srcs + [os.path.join(HERE, h) for h in HEADERS] + [os.path.abspath(__file__)]
    if not force and os.path.exists(OUT) and os.path.getmtime(OUT) >= _newest(deps):
        return OUT
    nvcc = os.environ.get("NVCC", "nvcc")
    objs = []
    procs = []
    for s in srcs:
        o = os.path.join(OUT_DIR, os.path.basename(s).replace(".cu", ".o"))
        objs.append(o)
        flags = list(NVCC_FLAGS)
        if os.path.basename(s) == "simt_kernels.cu":
            flags.remove("--use_fast_math")  # exact expf/logf/division in the fp32 family
        cmd = [nvcc] + flags + ["-c", s, "-o", o]
        procs.append((cmd, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    log = []
    for cmd, pr in procs:
        out, _ = pr.communicate()
        log.append(" ".join(cmd) + "\n" + out)
        if pr.returncode != 0:
            sys.stderr.write("\n".join(log))
            raise RuntimeError("nvcc failed: " + " ".join(cmd))
    link = [nvcc, "-shared", "-o", OUT] + objs + ["-gencode", "arch=compute_100a,code=sm_100a"]
    r = subprocess.run(link, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    log.append(" ".join(link) + "\n" + r.stdout)
    if r.returncode != 0:
        sys.stderr.write("\n".join(log))
        raise RuntimeError("link failed")
    with open(os.path.join(OUT_DIR, "build.log"), "w") as f:
        f.write("\n".join(log))
    if verbose:
        print("\n".join(log))
    return OUT


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
