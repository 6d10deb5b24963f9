"""A process that may not start threads: the exact distribution's host passes (eight
threads from 20,000 outcomes on) run on the caller's, instead of ending the process."""
import os
import resource
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# the outcome with a negative occupation is refused before any GPU is needed; a default
# stack of 2^50 bytes cannot be mapped, so that every new thread is denied
CHILD = """
import ctypes
L = ctypes.CDLL("{lib}")
m, n = 4, 24000
U, S, O = (ctypes.c_double * (2 * m * m))(), (ctypes.c_int32 * m)(1, 1, 0, 0), (ctypes.c_int32 * (n * m))()
P, ms = (ctypes.c_double * n)(), ctypes.c_float()
O[3] = -1
print(*[L.boss_lossy_probabilities(U, m, S, O, n, P, ctypes.byref(ms)) for _ in range(2)])
"""


def test_no_threads_to_be_had():
    lib = os.path.join(ROOT, "theboss_gb300", "libboss_gb300.so")

    def limit():
        resource.setrlimit(resource.RLIMIT_STACK, (2 ** 50, resource.getrlimit(resource.RLIMIT_STACK)[1]))

    r = subprocess.run([sys.executable, "-S", "-c", CHILD.format(lib=lib)], preexec_fn=limit, capture_output=True,
                       text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.split() == ["4", "4"], (r.returncode, r.stdout, r.stderr)
