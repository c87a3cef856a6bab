"""The kernels at the edges of their tiles: meshes a cell smaller, equal and a cell larger than a tile or a marching CTA's
columns, and remainders along every axis.

The marching mixed kernels (32 x 8 columns in 3-D, 128 columns with 127 cells of their own in 2-D; the stage state formed as
it is read) against the same run in parts, whose tiled kernels solve every face and update every cell with the same explicitly
rounded operations: the same bits; gated by the sensor, against the same run with an immersed body outside the mesh, which the tiled
kernels serve (a face inside a CTA is solved once: only such a comparison shows which values it took). The FP64 kernels (8x8x8 tiles, 16 x 15 and 16 x 5 tiles, 14 x 14 MUSCL-Hancock tiles) against
the restatement of the reference: the same bits. The batched rows (63, 127 and 255 cells) against single runs: the same bits."""
import os

import numpy as np
import pytest

import cases
from fenice_b200 import Batch, Run, slabs
from fenice_b200.sensor import Sensor
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu

B = cases.bcs
PER = B("periodic", "periodic", "periodic", "periodic")
WALLS3 = B("wall", "transmissive", "outlet", "wall", z=("periodic", "periodic"))


def same_bits(a, b):
    return np.array_equal(np.ascontiguousarray(a).view(np.uint64), np.ascontiguousarray(b).view(np.uint64))


def march_planes(nx, ny, nz=1):
    """The planes a CTA of the marching kernels owns on a whole mesh; 0 where the mesh takes the tiles."""
    three = nz > 1
    n, cols = (nz, -(-nx // 32) * -(-ny // 8)) if three else (ny, -(-nx // 127))
    tiles = -(-nx // 8) * -(-ny // 8) * -(-nz // 8) if three else -(-nx // 16) * -(-ny // 15)
    fill, base, per, resident = (13.0, 2.4, 3.0, 2) if three else (8.0, 0.9, 0.77, 5)

    def us(lz):
        full, rest = divmod(cols * -(-n // lz), 148 * resident)
        return full * (fill + lz * (base + per * resident)) + (fill + lz * (base + per * -(-rest // 148)) if rest else 0.0)

    lz = min(range(1, n + 1), key=us)
    full, rest = divmod(tiles, 148 * (3 if three else 4))
    tiled = (0.0 if three else 1.0) + full * (35.0 if three else 12.0) + ((19.0 + 7.5 * -(-rest // 148) if three else 8.0 + 1.9 * -(-rest // 148)) if rest else 0.0)
    return lz if us(lz) < tiled else 0


# (the last one of each list: several planes or rows to a CTA)
@pytest.mark.parametrize("nx,ny,nz", [(31, 7, 8), (32, 8, 9), (33, 9, 16), (70, 17, 13), (161, 83, 37)])
@pytest.mark.parametrize("sides", ["periodic_viscous", "walls"])
def test_marching_3d(nx, ny, nz, sides):
    assert march_planes(nx, ny, nz) == (10 if nx == 161 else 1)
    params = dict(nx=nx, ny=ny, nz=nz, reconstruction="weno5", riemann_solver="lowmach", time_scheme="SSP Runge-Kutta 3", cfl=0.4)
    params.update(dict(PER, use_viscous=True, mu=0.01) if sides == "periodic_viscous" else WALLS3)
    U0 = cases.case_field(params, nx + ny)
    run = Run(params, U=U0, precision=1)
    assert run.run(1e30, max_steps=3) == 3
    U, steps, t = slabs.run_decomposed(params, U0, 2, 1e30, max_steps=3, precision=1)
    assert steps == 3 and t == run.t and same_bits(run.state(), U)


@pytest.mark.parametrize("nx,ny", [(126, 15), (127, 16), (128, 31), (260, 46), (1300, 203)])
@pytest.mark.parametrize("sides", [PER, B("transmissive", "wall", "wall", "transmissive")], ids=["periodic", "walls"])
def test_marching_2d(nx, ny, sides):
    assert march_planes(nx, ny) == (4 if nx == 1300 else 1)
    params = dict(nx=nx, ny=ny, reconstruction="weno5", time_scheme="SSP Runge-Kutta 3", cfl=0.4, **sides)
    U0 = cases.case_field(params, 3 * (nx // 3))   # (a seed whose field has a jump: the HLL blend)
    run = Run(params, U=U0, precision=1)
    assert run.run(1e30, max_steps=4) == 4
    U, steps, t = slabs.run_decomposed(params, U0, 2, 1e30, max_steps=4, precision=1)
    assert steps == 4 and t == run.t and same_bits(run.state(), U)


# (planes or rows a CTA owns: 1, then 10, 20, 4 and 6, several rows of tiles)
GATED = {(33, 9, 13): 1, (70, 17, 20): 1, (64, 24, 31): 1, (128, 31, 1): 1, (127, 46, 1): 1, (260, 46, 1): 1, (33, 100, 1): 1, (161, 83, 37): 10, (256, 128, 40): 20,
         (1300, 203, 1): 4, (700, 700, 1): 6}


@pytest.mark.parametrize("sides", ["periodic", "walls"])
@pytest.mark.parametrize("nx,ny,nz", list(GATED))
def test_gated_marching(nx, ny, nz, sides):
    assert march_planes(nx, ny, nz) == GATED[nx, ny, nz]
    p = dict(nx=nx, ny=ny, reconstruction="weno5", riemann_solver="lowmach" if nz > 1 else "HLLC", time_scheme="SSP Runge-Kutta 3", cfl=0.4)
    if nz > 1:
        p.update(nz=nz, Lz=1.0)
    p.update(PER if sides == "periodic" else WALLS3 if nz > 1 else B("transmissive", "wall", "wall", "transmissive"))
    if nz == 1:
        p = {k: v for k, v in p.items() if not k.startswith("bc_z")}
    # smooth flow with a block of other gas in it, off the middle, so that linear and WENO5-Z tiles meet on every axis
    z, y, x = np.meshgrid(*[(np.arange(n) + 0.5) / n for n in (nz, ny, nx)], indexing="ij")
    W = np.zeros((x.size, 5))
    wave = np.sin(2 * np.pi * x) * np.cos(2 * np.pi * y)
    W[:, 0] = (1.0 + 0.02 * wave).ravel()
    W[:, 1] = (0.3 + 0.02 * np.cos(2 * np.pi * y)).ravel()
    W[:, 2] = (-0.2 + 0.02 * np.sin(2 * np.pi * x)).ravel()
    W[:, 3] = (1.0 + 0.02 * wave).ravel()
    if nz > 1:
        W[:, 4] = (0.1 + 0.02 * np.sin(2 * np.pi * z)).ravel()
    block = ((x > 0.1) & (x < 0.25) & (y > 0.55) & (y < 0.8) & ((z > 0.6) if nz > 1 else True)).ravel()
    W[block, 0] *= 1.7
    W[block, 3] *= 1.4
    U0 = cases.prim_to_cons(W)
    sensor = Sensor.load(os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fenice_b200", "sensor_weights.npz"))
    got = []
    for body in ({}, dict(use_ibm=True, ibm_shape="Sphere" if nz > 1 else "Cylinder", ibm_radius=0.1, ibm_cx=-9.0, ibm_cy=-9.0)):
        run = Run(dict(p, **body), U=U0, precision=1)
        run.set_sensor(sensor, float(sensor.meta["threshold"]), every=2, radius=1)
        assert run.run(1e30, max_steps=5) == 5
        linear, evaluated = run.sensor_counts()
        got.append((run.state(), run.t, linear, evaluated))
    (a, ta, la, ea), (b, tb, lb, eb) = got
    assert 0 < la < ea and (la, ea, ta) == (lb, eb, tb)
    assert same_bits(a, b), f"{int((a != b).sum())} values differ"


FP64 = [
    # 14 x 14 MUSCL-Hancock tiles, each limiter (a symmetric one is evaluated once for both sides)
    *[(dict(nx=n, ny=m, reconstruction="muscl", muscl_limiter=lim, time_scheme="MUSCL-Hancock", **s), 5)
      for n, m, lim, s in [(13, 14, "Minmod", PER), (14, 15, "Van Leer", PER), (15, 29, "MC", B("vel_inlet", "transmissive", "wall", "outlet")),
                           (43, 13, "Koren", B("wall", "transmissive", "periodic", "periodic"))]],
    # 16 x 5 tiles up to 148 of 16 x 15 (222 x 149: 140), and those beyond (240 x 150: 150, 320 x 241: 340)
    *[(dict(nx=n, ny=m, reconstruction=r, time_scheme=ts, cfl=0.4, **s), 4)
      for n, m, r, ts, s in [(15, 4, "muscl", "SSP Runge-Kutta 2", PER), (16, 5, "weno5", "SSP Runge-Kutta 3", B("wall", "transmissive", "outlet", "wall")),
                             (17, 6, "weno3", "SSP Runge-Kutta 3", PER), (222, 149, "weno5", "SSP Runge-Kutta 3", B("wall", "transmissive", "outlet", "wall")),
                             (240, 150, "muscl", "SSP Runge-Kutta 2", PER), (320, 241, "weno5", "SSP Runge-Kutta 3", PER)]],
    # 8x8x8 tiles, the viscous box without and with wall rules; other gases (the quotient by gamma - 1)
    *[(dict(nx=7, ny=8, nz=9, reconstruction="weno5", riemann_solver="lowmach", time_scheme="SSP Runge-Kutta 3", use_viscous=True, mu=0.01, gamma=g, **s), 3)
      for g, s in [(1.4, PER), (5.0 / 3.0, PER), (1.1, B("no_slip", "wall", "periodic", "periodic", z=("moving_wall", "no_slip")))]],
    (dict(nx=17, ny=9, nz=8, reconstruction="weno3", time_scheme="SSP Runge-Kutta 3", gamma=2.0, **WALLS3), 3),
]


@pytest.mark.parametrize("params,steps", FP64, ids=[f"{p['nx']}x{p['ny']}x{p.get('nz', 1)}-{p['reconstruction']}-{p.get('muscl_limiter', p.get('gamma', ''))}" for p, _ in FP64])
def test_fp64_tiles(params, steps):
    U0 = cases.case_field(params, 4 + params["nx"])
    run = Run(params, U=U0)
    assert run.run(1e30, max_steps=steps) == steps
    U, t, _, _, _ = Oracle().run(params, U0, steps)
    assert t == run.t and same_bits(run.state(), U)


@pytest.mark.parametrize("precision", [0, 1])
def test_batch_rows(precision):
    plist = [dict(nx=n, ny=1, Ly=1.0 / n, reconstruction="weno5", time_scheme="SSP Runge-Kutta 3", cfl=0.4,
                  **B("transmissive", "transmissive", "transmissive", "transmissive")) for n in (62, 63, 64, 126, 127, 128, 254, 255, 256, 300)]
    states = [cases.case_field(p, 3 * p["nx"]) for p in plist]
    single = []
    for p, U in zip(plist, states):
        run = Run(p, U=U, precision=precision)
        assert run.run(1e30, max_steps=5) == 5
        single.append(run.state())
    for shape in range(3):
        b = Batch(plist, states, precision=precision)
        b.set_schedule(shape)
        b.run(1e30, max_steps=5)
        for got, want in zip(b.split(b.state()), single):
            assert same_bits(got, want), shape
