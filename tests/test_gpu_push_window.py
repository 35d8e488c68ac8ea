"""The mixed push's 32-bit shared sums at their limit: a cold blob of equal
particles in one cell that all leave it through one face, so that both segments
of every particle meet on one node, at the most particles a tile may hold for those sums and below.

With seed 0 the transverse move is tiny and its terms just below zero, where a part of a split value
was the largest; the other seeds draw the blob. Bars: a term's FP32 error is at most 4 * 2^-24 for a move of 0.15
cells, 2e-6 of the sums, against 2e-5 here; one unit charge lost of 16384 or
more such moves would be 1 / (0.15 * 32767) = 2e-4 or more."""
import numpy as np
import pytest

import pbpic_b200
from test_gpu_parity import new_sim

pytestmark = pytest.mark.gpu

FACES = [(1, 0), (-1, 0), (0, 1), (0, -1)]


def blob(oracle_mod, n, face, seed=0):
    """n electrons at one point of cell (11, 12) of a 24 x 24 grid, and the grid."""
    cva, d = 10.0, 0.1
    cfg = dict(mx=24, my=24, dx=d, dy=d, dt=0.5 * d / cva / np.sqrt(2.0), cva=cva, mime=25.0, in0=1.0,
               ybc=pbpic_b200.BC_PERIODIC)
    step = cfg["dt"] * cva / d  # cells a step at the speed of light
    rng = np.random.default_rng(seed)
    along, across = (0.15, 1e-6) if seed == 0 else (rng.uniform(0.1, 0.25), rng.uniform(-0.1, 0.1))
    pos = 0.45 if seed == 0 else 0.5 - along * rng.uniform(0.1, 0.9)
    side = 0.1 if seed == 0 else rng.uniform(-0.3, 0.3)
    x, v = np.array([side, side]), np.array([across, across])
    for k in range(2):
        if face[k]:
            x[k], v[k] = pos * face[k], along * face[k]
    v = np.append(v / step, 0.2)
    u = v / np.sqrt(1.0 - v @ v)
    p = np.zeros(n, dtype=oracle_mod.PARTICLE)
    p["dx"], p["dy"] = x
    for k, c in enumerate(("ux", "uy", "uz")):
        p[c] = u[k]
    p["grid"] = 11 * cfg["my"] + 12 + 1
    p["q"] = -1
    p["pid"] = np.arange(n)
    return cfg, p


def push(cfg, p):
    with new_sim(cfg, len(p), precision="fp32") as s:
        s.load_particles(p)
        s.load_fields(np.zeros((6, cfg["mx"], cfg["my"] + 1)))
        s.countingsort()
        start = s.particles()
        s.pusher()
        assert s.status() == 0
        return start, s.denjr()


@pytest.mark.parametrize("seed", [0, 1, 2])
@pytest.mark.parametrize("n", [16384, 20000, 30000, 32767])
@pytest.mark.parametrize("face", FACES)
def test_blob_through_one_face(gpu_lib, oracle_mod, face, n, seed):
    cfg, p = blob(oracle_mod, n, face, seed)
    start, j = push(cfg, p)
    o = oracle_mod.Oracle(**cfg)
    o.load_particles(start)
    o.set_fields(np.zeros((6, cfg["mx"], cfg["my"] + 1)))
    o.pusher()
    jo = o.current()
    assert (o.particles()["grid"] != start["grid"]).all()  # every particle left its cell
    assert np.abs(j[:2] - jo[:2]).max() <= 2e-5 * np.abs(jo[:2]).max()


@pytest.mark.parametrize("seed", [0, 1, 2])
@pytest.mark.parametrize("face", FACES)
def test_same_bits_as_the_64_bit_sums(gpu_lib, oracle_mod, face, seed):
    """Twice the particles of the largest such tile take the 64-bit sums: exactly twice its jx and jy."""
    cfg, p = blob(oracle_mod, 32767, face, seed)
    once, twice = push(cfg, p)[1], push(cfg, np.concatenate([p, p]))[1]
    assert np.array_equal(twice[:2], 2.0 * once[:2])
