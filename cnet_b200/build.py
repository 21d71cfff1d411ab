"""Builds libcnet_b200.so in-tree: the sm_100a kernels + C ABI (csrc/) and the C++ host
facade (host/), and ops_native.so, the operators' calls from Python (host/ops_native.cpp), for which torch and its headers
have to be there; the library needs neither.
``python -m cnet_b200.build`` or ``build(force=True)``."""
import importlib.util
import os
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
LIB = os.path.join(HERE, "libcnet_b200.so")
OPS = os.path.join(HERE, "ops_native.so")
OPS_KEY = os.path.join(HERE, "build", "ops_native.key")
CSRC = ["context.cu", "elementwise.cu", "rowreduce.cu", "embed.cu", "cgemm_simt.cu", "cgemm_tc.cu", "linear.cu", "fft.cu", "fft_pipe.cu", "fft_mixed.cu", "cgemv_skinny.cu", "dp_allreduce.cu"]
HOST = ["cnet.cpp", "capi.cpp", "dp_nccl.cpp", "model_saver.cpp", "data_reader.cpp"]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O3", "-lineinfo",
              "-Xcompiler", "-fPIC", "-Xcompiler", "-Wall"]


def _sources():
    src = [os.path.join(HERE, "csrc", f) for f in CSRC] + [os.path.join(HERE, "host", f) for f in HOST]
    deps = src + [os.path.join(HERE, "csrc", "common.cuh"), os.path.join(HERE, "csrc", "cgemm_fma.cuh"), os.path.join(HERE, "csrc", "fft_regs.cuh"), os.path.join(HERE, "csrc", "fft_mixed.cuh"), os.path.join(HERE, "host", "cnet.h"), os.path.join(HERE, "host", "dp_nccl.h"), os.path.join(HERE, "host", "data_reader.h"),
                  os.path.join(HERE, "..", "include", "cnet_b200.h"),
                  os.path.join(HERE, "..", "include", "cnet_b200_host.h")]
    return src, deps


def up_to_date():
    if not os.path.exists(LIB):
        return False
    t = os.path.getmtime(LIB)
    return all(os.path.getmtime(d) <= t for d in _sources()[1] if os.path.exists(d))


def ops_command(src, out):
    """The compiler's call that makes a CPython module of host/ops_native.cpp, against this interpreter's and torch's headers."""
    import torch
    root = os.path.dirname(torch.__file__)
    return ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-Wall", "-D_GLIBCXX_USE_CXX11_ABI=%d" % torch._C._GLIBCXX_USE_CXX11_ABI,
            "-isystem", os.path.join(root, "include"), "-isystem", os.path.join(root, "include", "torch", "csrc", "api", "include"),
            "-I", sysconfig.get_paths()["include"], "-isystem", "/usr/local/cuda/include", src, "-o", out,
            "-L", os.path.join(root, "lib"), "-ltorch_python", "-ltorch_cpu", "-ltorch", "-lc10", "-lc10_cuda",
            "-L", HERE, "-l:libcnet_b200.so", "-Wl,-rpath,$ORIGIN"]


def ops_key():
    """What a build of the module depends on beside its sources: the interpreter and the torch whose headers it saw."""
    import torch
    return "%s, torch %s, C++11 ABI %d" % (sysconfig.get_config_var("EXT_SUFFIX"), torch.__version__, torch._C._GLIBCXX_USE_CXX11_ABI)


def _build_ops(env):
    """The module; the library beside it is found by $ORIGIN.  It appears whole: another process may be loading the one before."""
    key = ops_key()
    part = "%s.%d.tmp" % (OPS, os.getpid())
    cmd = ops_command(os.path.join(HERE, "host", "ops_native.cpp"), part) + ['-DCNET_BUILT_FOR="%s"' % key]
    r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, env=env)
    if r.returncode != 0:
        if os.path.exists(part):
            os.remove(part)
        raise RuntimeError("ops_native failed:\n" + r.stdout.decode())
    os.replace(part, OPS)
    os.makedirs(os.path.dirname(OPS_KEY), exist_ok=True)
    with open(OPS_KEY, "w") as f:
        f.write(key)


def _ops_up_to_date():
    deps = [os.path.join(HERE, "host", "ops_native.cpp"), os.path.join(HERE, "..", "include", "cnet_b200.h"), __file__]
    if not os.path.exists(OPS) or not os.path.exists(OPS_KEY) or open(OPS_KEY).read() != ops_key():
        return False
    return all(os.path.getmtime(d) <= os.path.getmtime(OPS) for d in deps)


def build(force=False, verbose=False):
    lib = _build_lib(force, verbose)
    if importlib.util.find_spec("torch") is None:
        print("torch is not installed: without ops_native.so, which cnet_b200.ops needs", file=sys.stderr)
        return lib
    if force or not _ops_up_to_date():
        _build_ops({k: v for k, v in os.environ.items() if k not in ("CXX", "CC")})
    return lib


def _build_lib(force, verbose):
    if not force and up_to_date():
        return LIB
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    obj_dir = os.path.join(HERE, "build")
    os.makedirs(obj_dir, exist_ok=True)
    src, _ = _sources()
    objs, procs = [], []
    env = dict(os.environ)
    env.pop("CXX", None)
    env.pop("CC", None)
    for s in src:
        o = os.path.join(obj_dir, os.path.basename(s) + ".o")
        objs.append(o)
        cmd = [nvcc] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-c", s, "-o", o]
        if s.endswith(".cpp"):
            cmd = [nvcc, "-std=c++17", "-O2", "-Xcompiler", "-fPIC", "-Xcompiler", "-Wall", "-c", s, "-o", o]
        procs.append((s, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, env=env)))
    for s, p in procs:
        out = p.communicate()[0].decode()
        if p.returncode != 0:
            raise RuntimeError("nvcc failed on %s:\n%s" % (s, out))
        if verbose and out.strip():
            print(out)
    cmd = [nvcc, "-shared", "-o", LIB] + objs + ["-lcudart", "-ldl"]
    r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, env=env)
    if r.returncode != 0:
        raise RuntimeError("link failed:\n" + r.stdout.decode())
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
