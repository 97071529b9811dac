"""Child processes with the runtime's stand-ins of fake_cudart.c preloaded; `fake`
in the child's program calls them."""
import atexit
import os
import shutil
import subprocess
import sys
import tempfile

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_lib = None

PROLOGUE = """
import ctypes
class fake:
    _l = ctypes.CDLL(None)
    _l.fake_small.restype = ctypes.c_void_p
    arm = staticmethod(lambda text, skip=0: fake._l.fake_arm(text.encode(), skip))
    refused = staticmethod(lambda: fake._l.fake_refused())
    count = staticmethod(lambda text: fake._l.fake_count(text.encode()))
    graphs = staticmethod(lambda: fake._l.fake_graphs())
    reset = staticmethod(lambda: fake._l.fake_reset())
    late = staticmethod(lambda on: fake._l.fake_late(int(on)))
    small = staticmethod(lambda: fake._l.fake_small())
"""


def _build():
    global _lib
    if _lib is None:
        out = tempfile.mkdtemp(prefix="fake_cudart")
        atexit.register(shutil.rmtree, out, True)
        lib = os.path.join(out, "libfake_cudart.so")
        cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
        subprocess.run(["gcc", "-O1", "-shared", "-fPIC", "-I" + os.path.join(cuda, "include"), "-o", lib,
                        os.path.join(ROOT, "tests", "fake_cudart.c"), "-ldl"], check=True)
        _lib = lib
    return _lib


def run_child(program: str) -> None:
    """Run `program` (Python) in a child process with the stand-ins."""
    env = dict(os.environ, LD_PRELOAD=_build())
    r = subprocess.run([sys.executable, "-c", PROLOGUE + program], cwd=ROOT, env=env, capture_output=True, text=True,
                       timeout=120)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
