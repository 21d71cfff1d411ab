"""ops_native.so without a GPU."""
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))

USE = """
import sys
sys.path[:0] = %r
import torch
from cnet_b200 import lib
lib.load()
import ops_throw_probe
for _ in range(3):
    try:
        ops_throw_probe.throwing()
    except (RuntimeError, MemoryError) as e:
        print("raised", e)
print("alive", sum(range(1000)))
"""


def test_a_c_exception_becomes_pythons(tmp_path):
    """The interpreter lock is given up during a call; a C++ exception that leaves the call must not leave Python without it."""
    from cnet_b200 import build
    out = str(tmp_path / "ops_throw_probe.so")
    subprocess.run(build.ops_command(os.path.join(HERE, "cpp", "ops_throw_probe.cpp"), out) + ["-Wl,-rpath," + build.HERE], check=True,
                   env={k: v for k, v in os.environ.items() if k not in ("CXX", "CC")})
    r = subprocess.run([sys.executable, "-c", USE % [str(tmp_path), os.path.dirname(HERE)]], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, (r.returncode, r.stderr[-2000:])
    assert r.stdout.count("raised") == 3 and "alive 499500" in r.stdout, r.stdout
