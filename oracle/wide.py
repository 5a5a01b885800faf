"""The port (raptor_port.c) in long double: the same source with every
floating-point type, literal and libm call widened (64 significand bits on
x86-64, 113 on AArch64), to tell which of two double-precision results is the
closer one.

TEST INFRASTRUCTURE ONLY."""
from __future__ import annotations

import ctypes
import os
import re
import subprocess

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
LIB_PATH = os.path.join(HERE, "_port", "libraptor_port_wide.so")
_LITERAL = re.compile(r"(?<![\w.])(?:\d+\.\d*(?:[eE][-+]?\d+)?|\.\d+(?:[eE][-+]?\d+)?|\d+[eE][-+]?\d+)(?![\w.])")


def _widen(text):
    """Floating literals of the code (not of its comments) with the long double suffix."""
    parts = re.split(r"(/\*.*?\*/|\"[^\"]*\")", text, flags=re.S)
    return "".join(p if k % 2 else _LITERAL.sub(lambda m: m.group(0) + "L", p) for k, p in enumerate(parts))


def build():
    out = os.path.dirname(LIB_PATH)
    os.makedirs(out, exist_ok=True)
    src = os.path.join(out, "raptor_port_wide.c")
    head = open(os.path.join(HERE, "raptor_port.h")).read()
    body = open(os.path.join(HERE, "raptor_port.c")).read().replace('#include "raptor_port.h"', head)
    with open(src, "w") as f:
        f.write("#include <tgmath.h>\n#include <stdlib.h>\n#include <string.h>\n#undef I\n#define double long double\n")
        f.write(_widen(body).replace("#include <math.h>", ""))
    subprocess.run(["gcc", "-O2", "-std=c11", "-fopenmp", "-fPIC", "-w", "-shared", "-o", LIB_PATH, src, "-lm"],
                   check=True)


def render(geom, prims, width, height, freqs, pixels=None, cam_size=40.0, inclination=60.0, stepsize=0.05,
           mbh=8.9505e39, m_unit=1e19, r_high=3.0, r_low=3.0, integrator=4, camera=0):
    """(pixels, frequencies) intensities as numpy.longdouble."""
    if not os.path.exists(LIB_PATH) or any(os.path.getmtime(LIB_PATH) < os.path.getmtime(os.path.join(HERE, n))
                                           for n in ("raptor_port.c", "raptor_port.h", "wide.py")):
        build()
    lib = ctypes.CDLL(LIB_PATH, mode=ctypes.RTLD_LOCAL)
    L, I, P = ctypes.c_longdouble, ctypes.c_int, ctypes.c_void_p

    class Scene(ctypes.Structure):
        _fields_ = [("n1", I), ("n2", I)] + [(k, L) for k in ("startx1", "startx2", "dx1", "dx2", "a", "hslope", "R0")] + \
                   [("prims", P), ("width", I), ("height", I)] + \
                   [(k, L) for k in ("cam_size_x", "cam_size_y", "inclination", "stepsize", "mbh", "m_unit", "r_high",
                                     "r_low")] + [("integrator", I), ("camera", I), ("emission", I)]

    wide = np.ascontiguousarray(prims, dtype=np.longdouble)
    s = Scene(geom.n1, geom.n2, geom.startx1, geom.startx2, geom.dx1, geom.dx2, geom.a, geom.hslope, geom.R0,
              wide.ctypes.data, width, height, cam_size, cam_size, inclination, stepsize, mbh, m_unit, r_high, r_low,
              integrator, camera, 0)
    nu = np.atleast_1d(np.asarray(freqs, dtype=np.longdouble))
    pix = np.ascontiguousarray(np.arange(width * height) if pixels is None else pixels, dtype=np.int32)
    out = np.zeros((len(pix), len(nu)), dtype=np.longdouble)
    lib.port_render.argtypes = [P, P, I, P, I, P, P, I]
    rc = lib.port_render(ctypes.byref(s), pix.ctypes.data, len(pix), nu.ctypes.data, len(nu), out.ctypes.data, None, 0)
    if rc != 0:
        raise RuntimeError(f"port_render failed ({rc})")
    return out
