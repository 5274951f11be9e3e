"""Compiles a test's own .cu file with the library's flags."""
import os
import subprocess

from sodabayes_gb300 import build as B

TESTS = os.path.dirname(os.path.abspath(__file__))


def shared_object(source, out_dir, objects=()):
    out = os.path.join(str(out_dir), source.replace(".cu", ".so"))
    cmd = [B.nvcc()] + B.ARCH + ["-O3", "-std=c++17", "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr",
                                 "-I" + os.path.join(B.ROOT, "include"), "-shared", "-o", out,
                                 os.path.join(TESTS, source)]
    cmd += [os.path.join(B.BUILD, o) for o in objects] + ["-lcudart_static", "-lrt", "-ldl", "-lpthread"]
    proc = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    assert proc.returncode == 0, proc.stdout
    return out
