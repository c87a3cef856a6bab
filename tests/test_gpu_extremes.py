"""Mixed-precision runs whose state leaves the range of FP32 or holds a NaN or an infinity: which values become non-finite and
which wave speeds still count. The plain formulas in FP32 decide both (a face with a NaN state has the flux and the speed
their comparisons leave, an energy flux that overflows is the difference of two infinities), in the row kernel of the
batches, the marching kernels and the tiled ones alike.

The expected values were taken with every face solved by the plain formulas: the non-finite cells and values after one step
are exact; the time after five steps (the sum of the speeds that counted) holds to 1e-3, four times the 2e-4 by which two
orders of the FP32 sums were seen to differ here, and a speed that no longer counts moves it by 1e-2 .. 1e-1."""
import numpy as np
import pytest

from fenice_b200 import Batch, Run

pytestmark = pytest.mark.gpu

CELLS = {"nan_energy": [1, 0.2, 0.1, np.nan, 0.1], "nan_density": [np.nan, 0.1, 0.1, 2.5, 0.1], "nan_momentum": [1, np.nan, 0.1, 2.5, 0.1],
         "nan_transverse": [1, 0.1, np.nan, 2.5, 0.1], "inf_energy": [1, 0.1, 0.1, -np.inf, 0.1],
         "inf_density": [np.inf, 0.2, 0.1, 2.5, 0.1],   # (its velocity is 0)
         "overflow": [-9.6e5, 1.1e12, 0, -2.5e18, 0]}   # (finite in FP64; its density is floored, so its velocity is 1e22)
# (cells, values) non-finite after one step and t after five, for meshes of 1, 2 and 3 dimensions
EXPECTED = {
    ("HLLC", "nan_energy"): [(1, 1, 2.3641e-2), (1, 1, 2.4036e-2), (1, 1, 2.7130e-2)],
    ("HLLC", "nan_density"): [(1, 1, 2.3641e-2), (1, 1, 2.4036e-2), (1, 1, 2.7130e-2)],
    ("HLLC", "nan_momentum"): [(1, 1, 2.3641e-2), (1, 1, 2.4036e-2), (1, 1, 2.7130e-2)],
    ("HLLC", "nan_transverse"): [(1, 1, 2.3641e-2), (1, 1, 2.4036e-2), (1, 1, 2.7130e-2)],
    ("HLLC", "inf_energy"): [(1, 1, 2.6913e-2), (1, 1, 2.6415e-2), (1, 1, 2.9171e-2)],
    ("HLLC", "inf_density"): [(1, 1, 2.3641e-2), (1, 1, 2.4036e-2), (1, 1, 2.7130e-2)],
    ("HLLC", "overflow"): [(3, 12, 2.4207e-2), (8, 22, 2.4056e-2), (13, 35, 2.6322e-2)],
    ("HLLC (Low-Mach Thornber)", "nan_energy"): [(1, 1, 2.3965e-2), (1, 1, 2.4744e-2), (1, 1, 2.7930e-2)],
    ("HLLC (Low-Mach Thornber)", "nan_density"): [(1, 1, 2.4699e-2), (1, 1, 2.4769e-2), (1, 1, 2.7930e-2)],
    ("HLLC (Low-Mach Thornber)", "nan_momentum"): [(1, 1, 2.4699e-2), (1, 1, 2.4769e-2), (1, 1, 2.7930e-2)],
    ("HLLC (Low-Mach Thornber)", "nan_transverse"): [(1, 1, 2.3986e-2), (1, 1, 2.4769e-2), (1, 1, 2.7909e-2)],
    ("HLLC (Low-Mach Thornber)", "inf_energy"): [(1, 1, 2.7106e-2), (1, 1, 2.6726e-2), (1, 1, 2.9391e-2)],
    ("HLLC (Low-Mach Thornber)", "inf_density"): [(1, 1, 2.4027e-2), (1, 1, 2.4769e-2), (1, 1, 2.7828e-2)],
    ("HLLC (Low-Mach Thornber)", "overflow"): [(3, 12, 2.5555e-2), (7, 24, 2.4573e-2), (11, 43, 2.7266e-2)],
}


def setup(dim, riemann):
    p = dict(nx=40, ny=(1, 32, 16)[dim - 1], Lx=1.0, Ly=1.0, gamma=1.4, riemann_solver=riemann, reconstruction="weno5",
             time_scheme="SSP Runge-Kutta 3", cfl=0.3)
    if dim == 3:
        p.update(nz=16, Lz=1.0)
    # a row of transmissive cells in a batch (the row kernel), periodic boxes (the marching kernels)
    p.update({f"bc_{a}{s}": "transmissive" if dim == 1 else "periodic" for a in "xyz"[:max(dim, 2)] for s in ("min", "max")})
    n = p["nx"] * p["ny"] * p.get("nz", 1)
    rng = np.random.default_rng(1)
    U = np.zeros((n, 5))
    U[:, 0] = 1 + 0.1 * rng.random(n)
    U[:, 1] = 0.2 * rng.random(n)
    U[:, 3] = 2.5 + 0.1 * rng.random(n)
    return p, U


@pytest.mark.parametrize("dim", [1, 2, 3])
@pytest.mark.parametrize("riemann,cell", list(EXPECTED), ids=["%s-%s" % (r.split()[-1].strip("()"), c) for r, c in EXPECTED])
def test_one_extreme_cell(riemann, cell, dim):
    p, U = setup(dim, riemann)
    U[len(U) // 2 + 11] = CELLS[cell]
    if dim < 3:
        U[:, 4] = 0.0
    run = Batch([p], [U], precision=1) if dim == 1 else Run(p, U, precision=1)
    run.run(1e30, max_steps=1)
    bad = ~np.isfinite(run.state())
    run.run(1e30, max_steps=1)
    run.run(1e30, max_steps=3)   # (no error: the run does not count the speeds it cannot tell)
    t = run.problem(0).t if dim == 1 else run.t
    cells, values, t5 = EXPECTED[riemann, cell][dim - 1]
    assert (int(bad.any(axis=1).sum()), int(bad.sum())) == (cells, values)
    assert abs(t - t5) <= 1e-3 * t5, (t, t5)


def test_tube_that_blows_up_goes_on():
    """A shock tube with a density that falls to 0 at its outflow side (WENO5-Z has no positivity limiter) blows up in the
    next step: its cells become NaN, no error is reported and the rest of the tube goes on with the speeds it has."""
    head = np.array([[0.05704540, 0.04510774, 0.0, -0.21930686], [1.60857304, 0.64209913, 0.0, 0.98746127], [1.86041959, 0.41713689, 0.0, 1.32649499],
                     [1.91548331, 0.45500305, 0.0, 1.36898056], [2.01336806, 0.50753157, 0.0, 1.42064297], [2.05756162, 0.54101918, 0.0, 1.45967688]])
    U = np.zeros((187, 5))
    U[:, :4] = [2.0, 0.52, 0.0, 1.46]
    U[:6, :4] = head
    p = dict(nx=187, ny=1, Lx=1.0, Ly=1.0 / 187, gamma=1.4, reconstruction="weno5", riemann_solver="HLLC", time_scheme="SSP Runge-Kutta 3", cfl=0.4,
             bc_xmin="transmissive", bc_xmax="transmissive", bc_ymin="transmissive", bc_ymax="transmissive")
    b = Batch([p], [U], precision=1)
    b.run(1e30, max_steps=1)
    t1 = b.problem(0).t
    b.run(1e30, max_steps=50)
    pr = b.problem(0)
    bad = ~np.isfinite(b.state()).all(axis=1)
    assert pr.status == 0 and pr.t > t1
    assert bad[:4].any() and not bad[8:].any()
