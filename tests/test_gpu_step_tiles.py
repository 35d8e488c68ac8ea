"""The one-launch field solve and the fused sort's tables at the sizes where they can
go wrong: grids around the field solve's 16 x 32 node tiles, narrower than
its halo, and sort tiles of one row, of one less than the rows allow, and that
leave one row over. Against the oracle: FP64 fields, node grid and energies
within 1e-12 (the current's sums differ in order), FP32 fields within 1e-5 of
their maximum; the sort order and counts exactly."""
import numpy as np
import pytest

import pbpic_b200
from pbpic_b200 import configs
from test_gpu_edges import rows_of
from test_gpu_parity import field_err, new_sim, plasma, random_fields

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("ybc", [0, 1])
@pytest.mark.parametrize("mx,my", [(3, 3), (3, 31), (15, 32), (16, 33), (17, 30), (33, 64), (5, 65), (2, 2)])
def test_field_solve(gpu_lib, oracle_mod, precision, ybc, mx, my):
    cfg, _, p, _ = plasma(oracle_mod, ybc, mx=mx, my=my, ppc=3)
    yee = random_fields(cfg, mx + 100 * my)
    with new_sim(cfg, len(p), precision=precision) as s:
        s.load_particles(p)
        s.load_fields(yee)
        o = oracle_mod.Oracle(**cfg)
        o.load_particles(s.particles())
        o.set_fields(s.fields())
        for _ in range(2):
            s.pusher()
            s.fieldsolver()
            s.countingsort()
            o.pusher()
            o.fieldsolver()
            o.countingsort()
        fo, rows = o.fields(), rows_of(cfg)
        tol = 1e-12 if precision == "fp64" else 1e-5
        assert field_err(s.fields(), fo, cfg) <= tol * np.abs(fo).max()
        go = o.emfgrid()
        assert np.abs(s.emfgrid() - go).max() <= tol * np.abs(go).max()
        assert np.allclose(s.energies(), o.energies(), rtol=tol)
        # rows that the boundary does not use keep what was loaded
        f = s.fields()
        assert np.array_equal(f[:, :, rows:], np.zeros_like(f[:, :, rows:]))
        # step (field solve beside the sort, energies in one row) equals the three calls
        with new_sim(cfg, len(p), precision=precision) as t:
            t.load_particles(p)
            t.load_fields(yee)
            t.step(2, sort_every=1)
            assert np.allclose(t.energy_history(), s.energy_history(), rtol=1e-12)
            if precision == "fp32":
                assert np.array_equal(t.fields(), s.fields()) and np.array_equal(t.denjr(), s.denjr())


@pytest.mark.parametrize("ybc,mx,my,ty", [(0, 3, 3, 1), (0, 3, 66, 64), (0, 4, 65, 1), (1, 3, 2, 1), (1, 3, 65, 64),
                                         (1, 4, 64, 64), (0, 5, 67, 64), (1, 6, 9, 2), (0, 33, 41, 13)])
def test_sort_tables(gpu_lib, oracle_mod, ybc, mx, my, ty):
    cfg, _, p, _ = plasma(oracle_mod, ybc, mx=mx, my=my, ppc=5, vthe=0.6)
    with new_sim(cfg, len(p), precision="fp32", tile_rows=ty, options=pbpic_b200.OPT_NO_AUTOSORT) as s:
        s.load_particles(p)
        s.load_fields(random_fields(cfg, 5, amp=0.2))
        s.countingsort()
        for _ in range(3):
            s.pusher()
            pre = s.particles()
            s.countingsort()
            post = s.particles()
            order = np.argsort(pre["grid"], kind="stable")
            assert np.array_equal(post["pid"], pre["pid"][order])
            assert np.array_equal(s.cell_counts(), np.bincount(pre["grid"] - 1, minlength=mx * my))
        assert s.status() == 0


@pytest.mark.parametrize("mx,my", [(31, 33), (32, 32), (25, 41), (64, 80), (4096, 2049)])
def test_sort_tables_chunks(gpu_lib, mx, my):
    """Cells one less than, equal to and one more than a chunk of the tables, several chunks, and more
    than one launch takes: the order and counts exactly, twice (the chunks' totals are cleared)."""
    rng = np.random.default_rng(mx * my)
    n = 20000
    p = np.zeros(n, dtype=pbpic_b200._lib.PARTICLE_F64)
    p["grid"] = rng.integers(0, mx * my, n) + 1
    p["q"] = np.where(np.arange(n) % 2, 1, -1)
    p["pid"] = np.arange(n)
    for c, w in (("dx", 0.49), ("dy", 0.49), ("ux", 0.8), ("uy", 0.8), ("uz", 0.8)):
        p[c] = rng.uniform(-w, w, n)
    cfg, _ = configs.uniform_c1(mx=mx, my=my)
    with new_sim(cfg, n, precision="fp32", options=pbpic_b200.OPT_NO_AUTOSORT) as s:
        s.load_particles(p)
        s.countingsort()
        for _ in range(2):
            s.pusher()
            pre = s.particles()
            s.countingsort()
            post = s.particles()
            assert (np.diff(pre["grid"]) < 0).any()
            assert np.array_equal(post["pid"], pre["pid"][np.argsort(pre["grid"], kind="stable")])
            assert np.array_equal(s.cell_counts(), np.bincount(pre["grid"] - 1, minlength=mx * my))
        assert s.status() == 0
