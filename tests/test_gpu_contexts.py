"""What a process keeps beside a solver context must hold for every device, context and thread:
kernels' shared-memory limits, which the runtime keeps a device context (one a device)."""
import subprocess

import pytest

import statics_cuda as sc

from helpers import run_script

pytestmark = pytest.mark.gpu

TWICE = """
    import ctypes, sys
    import numpy as np
    import statics_cuda as sc
    from helpers import lattice_dict, oracle_lattice, piece, z_loads

    name, precision = sys.argv[1], int(sys.argv[2])

    def call():
        solver = sc.Solver(0)
        opt = sc.options(max_iter=5000, tol=1e-8, precision=precision, tile=1 if name == "pencil" else 0)
        if name == "lattice":  # solved at level 0: a dense top of 46 parts, 276 rows
            st = np.ones((3, 2, 3), np.uint8)
            st[:, :, 0] = 2
            loads, ex = z_loads(oracle_lattice(st, np.ones(st.shape, np.float32)))
            out = solver.motions(lattice_dict(ex), None, None, loads, None, opt)
        else:
            shape = (20, 48, 48) if name == "many bricks" else (17, 24, 21)
            out, _ = solver.solve_grid(*piece(0, 3, shape=shape), opt)
        solver.close()
        return out

    first = call()
    assert ctypes.CDLL("libcudart.so.12").cudaDeviceReset() == 0
    assert np.array_equal(call(), first)
"""


@pytest.mark.parametrize("precision", [sc.FP64, sc.MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("name", ["lattice", "few bricks", "many bricks", "pencil"])
def test_a_new_device_context_solves_as_the_first(name, precision):
    """A kernel's limit of dynamic shared memory belongs to the device's context. A second device
    starts without what the first was given; so does the same device once its context is
    ended, which one device is enough to check: the same call in a fresh solver, the same
    bits."""
    run_script(TWICE, name, str(precision))


SHIM = r"""
#include <dlfcn.h>
#include <stdio.h>
static struct { const void* f; int most; } seen[4096];
static int n;
int cudaFuncSetAttribute(const void* f, int attr, int value) {
    static int (*next)(const void*, int, int);
    if (!next)  /* the runtime's own: it is loaded already, in the library's scope */
        next = (int (*)(const void*, int, int))dlsym(dlopen("libcudart.so.12", RTLD_NOW | RTLD_NOLOAD),
                                                     "cudaFuncSetAttribute");
    if (!next) return 999;
    if (attr == 8) {  /* cudaFuncAttributeMaxDynamicSharedMemorySize */
        int i = 0;
        while (i < n && seen[i].f != f) i++;
        if (i == n && n < 4096) seen[n++].f = f;
        if (i < n) {
            if (value < seen[i].most) {
                fprintf(stderr, "limit lowered from %d to %d\n", seen[i].most, value);
                return 1;  /* cudaErrorInvalidValue */
            }
            seen[i].most = value;
        }
    }
    return next(f, attr, value);
}
"""

BOTH = """
    import statics_cuda as sc
    from helpers import piece

    opt = sc.options(max_iter=5000, tol=1e-8)
    for shape in ((31, 29, 37), (9, 8, 7), (24, 24, 24), (12, 20, 9)):
        solver = sc.Solver(0)
        _, info = solver.solve_grid(*piece(0, 3, shape=shape), opt)
        assert info["status"] == sc.OK
        solver.close()
"""


def test_no_limit_is_ever_lowered(tmp_path):
    """A kernel's limit is the device's, so every thread's: lowered to what one launch needs, it
    fails another thread's launch that needs more and was about to run. Here the call that
    sets it is stood in for, and refuses to lower one: large and small pieces in turn solve."""
    (tmp_path / "shim.c").write_text(SHIM)
    shim = str(tmp_path / "shim.so")
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-o", shim, str(tmp_path / "shim.c"), "-ldl"], check=True)
    run_script(BOTH, env={"LD_PRELOAD": shim})
