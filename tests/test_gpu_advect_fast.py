"""The 3D float advection's common case against the oracle, bit for bit, where
it can go wrong: positions around its limit of 2^22 cells and beyond, sides
above it, the last cells of every axis, samples that mix both forms."""
import numpy as np
import pytest

from conftest import rng
from test_gpu_ops import cells, faces, host, make_grid, same

pytestmark = pytest.mark.gpu


def check(pg, oracle, dims, vel, seed, dt=0.75):
    r = rng(seed)
    g = make_grid(pg, dims)
    q = r.standard_normal(dims).astype(np.float32)
    qf = r.standard_normal(vel.size).astype(np.float32)
    out = cells(pg, g, np.zeros(dims, np.float32))
    pg.advect(out, cells(pg, g, q), dt, faces(pg, g, vel))
    same(host(out), oracle.advect(q, dt, vel, dims))
    outf = faces(pg, g, np.zeros(vel.size, np.float32))
    pg.advect_mac(outf, faces(pg, g, qf), dt, faces(pg, g, vel))
    same(host(outf), oracle.advect_mac(qf, dt, vel, dims))


@pytest.mark.parametrize("dims", [(2, 2, 2), (3, 5, 4), (17, 2, 33), (9, 40, 65)])
@pytest.mark.parametrize("speed", [1.0, 5.6e6, 1e12])
def test_positions_near_and_past_the_limit(pg, oracle, dims, speed):
    """speed 5.6e6: back-traces of about 2^22 cells; a third of the faces
    slow, a few infinite or NaN."""
    r = rng(int(speed) % 997 + dims[2])
    vel = (speed * r.uniform(-1.0, 1.0, oracle.num_faces(dims))).astype(np.float32)
    vel[::3] = r.standard_normal(vel[::3].size)
    vel[5::17] = np.float32(0.5)
    if speed > 1e6:
        vel[7::41] = np.inf
        vel[11::53] = np.nan
    check(pg, oracle, dims, vel, 3)


@pytest.mark.parametrize("dims", [(2, 2, (1 << 22) + 9), (2, (1 << 22) + 1, 2), (2, 3, 1 << 22)])
def test_long_sides(pg, oracle, dims):
    r = rng(9)
    vel = (40.0 * r.standard_normal(oracle.num_faces(dims))).astype(np.float32)
    check(pg, oracle, dims, vel, 4)
