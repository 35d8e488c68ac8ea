"""The push cell by cell (sorted input) at the sizes where it can go
wrong: particles per cell around the lane-group widths (16 and 32 lanes), more
passes in a cell than one chunk of sums, a last tile of few rows, both y
boundaries with fast particles (every lane's crossing branch), with and without
tracked ids, in place and through the sort's permutation.

Bars as in test_gpu_edges.py: particles within 2e-5 and the current within 2e-4 of
its maximum against the FP64 oracle started from the same FP32 state; the plain
form within 1e-12 (both)."""
import numpy as np
import pytest

import pbpic_b200
from test_gpu_edges import check_one_step, rows_of
from test_gpu_parity import assert_particles, new_sim, plasma, random_fields

pytestmark = pytest.mark.gpu

# pairs per cell: mixed 16 lanes from 16 particles a cell on, 32 lanes from 180 on; plain 32 lanes from 30 on
PPC = {"fp32": [8, 9, 16, 17, 89, 90, 140], "fp64": [15, 16, 17, 140]}
BOTH = [(p, k) for p, ks in PPC.items() for k in ks]


@pytest.mark.parametrize("ybc", [0, 1])
@pytest.mark.parametrize("precision,ppc", BOTH)
def test_in_place_step(gpu_lib, oracle_mod, precision, ppc, ybc):
    cfg, _, p, _ = plasma(oracle_mod, ybc, mx=5, my=67, ppc=ppc, vthe=0.4)
    check_one_step(oracle_mod, cfg, p, random_fields(cfg, 31 + ppc), precision)


@pytest.mark.parametrize("ybc", [0, 1])
@pytest.mark.parametrize("precision,ppc", BOTH)
def test_step_through_the_permutation(gpu_lib, oracle_mod, precision, ppc, ybc):
    cfg, _, p, _ = plasma(oracle_mod, ybc, mx=4, my=66, ppc=ppc, vthe=0.4)
    tol, jtol = (1e-12, 1e-12) if precision == "fp64" else (2e-5, 2e-4)
    with new_sim(cfg, len(p), precision=precision) as s:
        s.load_particles(p)
        s.load_fields(random_fields(cfg, 7 + ppc))
        s.step(1, sort_every=1)
        o = oracle_mod.Oracle(**cfg)
        o.load_particles(s.particles())
        o.set_fields(s.fields())
        o.pusher()
        s.pusher()
        assert_particles(s.particles(), o.particles(), tol)
        rows = rows_of(cfg)
        jg, jo = s.denjr()[:, :, :rows], o.current()[:, :, :rows]
        assert np.abs(jg - jo).max() <= jtol * np.abs(jo).max()
        grid = s.particles()["grid"]
        assert np.all(np.diff(grid) >= 0)  # the sort from the push's counts
        assert np.array_equal(s.cell_counts(), np.bincount(grid - 1, minlength=cfg["mx"] * cfg["my"]))
        assert s.status() == 0


@pytest.mark.parametrize("ppc", [9, 140])
def test_same_bits_with_and_without_ids_and_for_any_tile_rows(gpu_lib, oracle_mod, ppc):
    """A cell's sums do not depend on the tile it lies in, nor on the ids carried along."""
    cfg, _, p, _ = plasma(oracle_mod, 1, mx=6, my=50, ppc=ppc, vthe=0.4)
    yee = random_fields(cfg, 3)
    runs = []
    for ty, track in ((0, True), (0, False), (7, False), (33, True)):
        with pbpic_b200.Simulation.from_config(cfg, capacity=len(p), precision="fp32", tile_rows=ty,
                                               track_pid=track) as s:
            s.load_particles(p)
            s.load_fields(yee)
            s.step(3, sort_every=1)
            runs.append((s.particles(), s.fields(), s.denjr()))
    for q, f, j in runs[1:]:
        for c in ("grid", "dx", "dy", "ux", "uy", "uz", "q"):
            assert np.array_equal(q[c], runs[0][0][c]), c
        assert np.array_equal(f, runs[0][1]) and np.array_equal(j, runs[0][2])
