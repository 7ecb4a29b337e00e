"""A PCG kernel whose launch is refused is reported, not passed over: with no device visible every launch
is, so the solver's launcher is called on a host image of its arguments (no system, no iterations:
nothing it points to is read) and asked for its error."""
import os
import subprocess
import sys

import build_lib

PROGRAM = """
import ctypes, sys
lib = ctypes.CDLL(sys.argv[1])
zeros = [ctypes.create_string_buffer(1 << 16) for _ in range(2)]  # Dev, Proj
epoch = ctypes.c_int(0)
f = lib["_ZN4astg15launch_pcg_fp64ERKNS_3DevERNS_4ProjEdiRiiP11CUstream_stPNS_5KProfE"]
f.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_double, ctypes.c_int, ctypes.c_void_p, ctypes.c_int,
              ctypes.c_void_p, ctypes.c_void_p]
f(*(ctypes.addressof(z) for z in zeros), 1e-6, 0, ctypes.addressof(epoch), 8, None, None)
take = lib["_ZN4astg17take_launch_errorEv"]
print(take(), take())
"""


def test_a_refused_launch_is_noted_and_taken_once():
    env = dict(os.environ, CUDA_VISIBLE_DEVICES="")
    r = subprocess.run([sys.executable, "-c", PROGRAM, build_lib.build()], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    first, second = map(int, r.stdout.split())
    assert first != 0 and second == 0
