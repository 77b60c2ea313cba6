"""wide_exact.npz: one step of a wide robot (test_gpu_rowspace.py, scene "wide", 512 envs) in 64 bits.

The oracle's sources are compiled with double for float in a temporary folder, template and inputs stay the 32-bit values.
Run: python tests/golden/make_wide_exact.py"""
import ctypes
import glob
import os
import re
import subprocess
import sys
import tempfile

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(os.path.dirname(HERE))
sys.path[:0] = [os.path.join(ROOT, "nuka-physics_b200"), os.path.dirname(HERE)]
E, LINKS = 512, 31


def wide_source(text, step):
    text = re.sub(r"\bfloat\b(?!\.h)", "double", text)
    text = re.sub(r"\b(sqrt|fabs|fmin|fmax|fma|hypot|sin|cos|atan2|nextafter)f\b", r"\1", text).replace("FLT_EPSILON", "DBL_EPSILON")
    text = re.sub(r"(memcpy\([^;]*?, )(12|16|24|28)\)", r"\1 2 * \2)", text)               # copies of a few floats
    if step:                                                                               # the template holds floats
        text = text.replace("(double *)blob_arr(blob, bytes, name, (uint64_t)(cnt), &ok)", "widen(blob_arr(blob, bytes, name, (uint64_t)(cnt), &ok), cnt)")
        text = text.replace("const double *cf = (const double *)", "const float *cf = (const float *)")
        text = text.replace("static uint32_t joint_dofs", "static double *widen(const float *p, size_t n) { double *d = calloc(n + 1, 8);"
                            " for (size_t i = 0; p && i < n; ++i) d[i] = p[i]; return d; }\nstatic uint32_t joint_dofs", 1)
        text = text.replace("B + 3, 4)", "B + 3, 8)").replace("4 * B + 4, 4)", "4 * B + 4, 8)").replace("*esz = 4;", "*esz = 8;")
    return text


def main():
    from test_gpu_rowspace import scene
    with tempfile.TemporaryDirectory() as folder:
        for path in glob.glob(os.path.join(ROOT, "oracle", "orc*.[ch]")):
            name = os.path.basename(path)
            with open(path) as f, open(os.path.join(folder, name), "w") as g:
                g.write(wide_source(f.read(), name == "orc_step.c"))
        library = os.path.join(folder, "wide.so")
        subprocess.run(["gcc", "-O2", "-march=x86-64-v3", "-fPIC", "-fopenmp", "-w", "-std=gnu11", "-shared", "-o", library,
                        *glob.glob(os.path.join(folder, "*.c")), "-lm"], check=True)
        orc = ctypes.CDLL(library)
        orc.orc_world_create.restype = ctypes.c_void_p
        blob, state = (lambda tb, s: (tb.blob(), s))(*scene("wide", E))
        world = ctypes.c_void_p(orc.orc_world_create(bytes(blob), ctypes.c_size_t(len(blob)), E))

        def move(call, field, array):
            assert call(world, field.encode(), ctypes.c_void_p(array.ctypes.data), ctypes.c_size_t(array.nbytes)) == 0, field

        for field, value in state.items():
            move(orc.orc_set, field, np.ascontiguousarray(value, np.float64))
        orc.orc_world_refresh(world)
        orc.orc_world_step(world, 1, 0)
        velocity = np.zeros((E, LINKS))
        move(orc.orc_get, "qdot", velocity)
    np.savez_compressed(os.path.join(HERE, "wide_exact.npz"), qdot=velocity)


if __name__ == "__main__":
    main()
