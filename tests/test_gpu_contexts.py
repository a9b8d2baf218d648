"""What a process keeps beside a solver context must hold for every device, context and thread:
kernels' shared-memory limits, which the runtime keeps a device context (one a device)."""
import os
import subprocess
import sys
import textwrap

import numpy as np
import pytest

import statics_cuda as sc

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def run_script(script, *args, env=None):
    """`script` in a process of its own (its end ends its device context too)."""
    paths = [ROOT, os.path.join(ROOT, "parallax-world_b200"), os.path.join(ROOT, "tests")]
    done = subprocess.run([sys.executable, "-c", textwrap.dedent(script), *args], capture_output=True, text=True,
                          timeout=600, env=dict(os.environ, PYTHONPATH=os.pathsep.join(paths), **(env or {})))
    assert done.returncode == 0, done.stderr[-2000:]


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
