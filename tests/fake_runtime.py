"""Runs a function of a test module in a child process over the stand-in CUDA runtime (fake_cudart.c): what the host side of the
library asks of the runtime, and how it answers failures, without a GPU."""
import ctypes as C
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
ON_LAUNCH = C.CFUNCTYPE(None, C.c_char_p, C.POINTER(C.c_uint), C.POINTER(C.c_void_p))


def run(tmp_path, module, function, *args):
    """module.function(fake, *args) in a child; fails with the child's output."""
    so = os.path.join(tmp_path, "libfake_cudart.so")
    if not os.path.exists(so):
        subprocess.check_call(["gcc", "-O1", "-shared", "-fPIC", "-o", so, os.path.join(HERE, "fake_cudart.c")])
    code = (f"import sys; sys.path[:0] = [{ROOT!r}, {HERE!r}]; import fake_runtime, {module} as m; "
            f"m.{function}(fake_runtime.Fake({so!r}), *{args!r})")
    env = dict(os.environ, LD_PRELOAD=so)
    env.pop("BUDDY_B200_DECODE", None)
    r = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


class Fake:
    def __init__(self, so):
        self.so = C.CDLL(so)
        self._keep = None

    def value(self, name, kind=C.c_size_t):
        return kind.in_dll(self.so, name)

    def on_launch(self, fn):
        """fn(kernel's mangled name, grid, args): args[i] is the address of parameter i."""
        self._keep = ON_LAUNCH(lambda name, grid, args: fn(name.decode(), (grid[0], grid[1], grid[2]), args))
        C.c_void_p.in_dll(self.so, "fake_on_launch").value = C.cast(self._keep, C.c_void_p).value
