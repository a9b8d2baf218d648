"""The conjugate gradients' iterations: an exact preconditioner, pieces of a batch that stop apart,
iterations driven from the host. Against the oracle's motions."""
import numpy as np
import pytest

import statics_cuda as sc

from helpers import oracle_lattice, piece, rel, run_script, z_loads

pytestmark = pytest.mark.gpu

# as in test_gpu_parity.py
DISP_TOL = 1e-6

TOWERS = [((1, 1),), ((2, 2),), ((3, 3), (3, 3), (1, 2), (1, 1), (1, 1)),
          ((3, 3), (3, 3), (1, 1), (1, 1), (1, 1), (1, 1)), ((3, 3), (3, 3), (3, 3), (2, 2), (2, 2), (1, 1)),
          ((3, 3), (3, 3), (3, 3), (3, 3), (1, 1))]


@pytest.mark.parametrize("layers,rows", list(zip(TOWERS, (30, 96, 510, 516, 816, 822))),
                         ids=["a panel's part", "whole panels", "a column a thread", "two", "most in shared memory",
                              "past it"])
def test_dense_top_is_the_inverse(solver, layers, rows):
    """A piece solved at level 0 by its dense top alone, the rows chosen at the edges of the
    factor's panels, of its threads' columns and of the kernels that keep it in shared
    memory. The preconditioner is K's inverse but for its rounding, at most n kappa eps of
    it, under 1e-8 (n 822, kappa about 1e5), so one iteration reaches 1e-8 where every
    entry is right (a wrong one takes a second iteration at least, as the oracle's one
    shows)."""
    st = np.zeros((3, 3, 1 + len(layers)), np.uint8)
    st[:, :, 0] = 2
    for z, (w, d) in enumerate(layers):
        st[:w, :d, 1 + z] = 1
    _, parts = sc.grid_count(st)
    assert 6 * parts == rows
    k = np.random.default_rng(parts).uniform(0.5, 2.0, st.shape).astype(np.float32)
    lat = oracle_lattice(st, k)
    loads, _ = z_loads(lat)
    u_ref, ir = lat.motions(loads, tol=1e-8, few=parts, hierarchy=True)
    u, info = solver.solve_grid(st, k, sc.options(max_iter=50, tol=1e-8, few=parts))
    assert info["status"] == sc.OK and info["parts"] == ir["counts"] == [parts]
    assert info["iterations"] == ir["iterations"] == 1
    assert rel(u, u_ref) < 1e-8


def _drifting():
    """A piece whose true residual misses 1e-8 when its recursive one meets it, and ones that
    meet both, in one batch (see test_residual_replacement_and_fp64_floor)."""
    return [sc.generate_piece(16, 24, 64, 10256, sc.K_UNIFORM), piece(24, 3), piece(16, 0)]


@pytest.mark.parametrize("precision", [sc.FP64, sc.MIXED], ids=["fp64", "mixed"])
def test_one_piece_goes_on_while_others_rest(solver, precision):
    """In one batch, a piece whose residual is replaced goes on after the others have stopped:
    theirs are not advanced again (each piece's own true residual, and the oracle's motions)."""
    pieces = _drifting()
    outs, infos = solver.solve_grid_batch(pieces, sc.options(max_iter=20000, tol=1e-8, precision=precision))
    assert [i["refinements"] > 0 for i in infos] == [True, False, False]
    assert infos[0]["iterations"] > max(i["iterations"] for i in infos[1:])
    for (st, k), u, info in zip(pieces, outs, infos):
        assert info["status"] == sc.OK and info["residual"] <= 1e-8 * (1 + 1e-9)
        lat = oracle_lattice(st, k)
        loads, _ = z_loads(lat)
        u_ref, _ = lat.motions(loads, tol=1e-12, max_iter=20000)
        assert rel(u, u_ref) < DISP_TOL


@pytest.mark.parametrize("precision", [sc.FP64, sc.MIXED], ids=["fp64", "mixed"])
def test_host_driven_iterations_give_the_same_bits(solver, precision, tmp_path):
    """The iterations launched from the host (SC_NO_GRAPHS=1, read once a process) and looped on
    the device: the same batch, with one piece's residual replaced, and the same single piece,
    bit for bit."""
    opt = sc.options(max_iter=20000, tol=1e-8, precision=precision)
    outs, infos = solver.solve_grid_batch(_drifting(), opt)
    u, info = solver.solve_grid(*piece(20, 5), opt)
    out = str(tmp_path / "host.npz")
    run_script("""
        import sys
        import numpy as np
        import statics_cuda as sc
        from helpers import piece
        from test_gpu_iterations import _drifting

        opt = sc.options(max_iter=20000, tol=1e-8, precision=int(sys.argv[1]))
        solver = sc.Solver(0)
        outs, infos = solver.solve_grid_batch(_drifting(), opt)
        u, info = solver.solve_grid(*piece(20, 5), opt)
        np.savez(sys.argv[2], *outs, u, np.array([i["iterations"] for i in infos + [info]]))
        """, str(precision), out, env={"SC_NO_GRAPHS": "1"})
    with np.load(out) as host:
        for j, want in enumerate(outs + [u, np.array([i["iterations"] for i in infos + [info]])]):
            assert np.array_equal(host[f"arr_{j}"], want)
