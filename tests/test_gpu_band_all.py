"""A band of every row (pbpic_band_extract over [0, my)): the records of the whole
domain in cell order, equal to the stored particles bit for bit, at counts
around the block of 256 records, with the sort's permutation pending and
without, with shifted rows, into aligned and (FP32) 4-byte aligned buffers."""
import ctypes

import numpy as np
import pytest

import pbpic_b200
from pbpic_b200 import _lib as L
from test_gpu_parity import new_sim, plasma

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("n", [0, 1, 255, 256, 257, 3000])
@pytest.mark.parametrize("steps", [0, 2])
def test_all_rows(gpu_lib, oracle_mod, precision, n, steps):
    import torch
    cfg, _, p, yee = plasma(oracle_mod, 0, mx=10, my=15, ppc=10)
    rec = L.PARTICLE_F32 if precision == "fp32" else L.PARTICLE_F64
    with new_sim(cfg, max(n, 1), precision=precision) as s:
        s.load_particles(p[:n].copy())
        s.load_fields(yee)
        s.countingsort()
        if steps:
            s.step(steps, sort_every=1)
        want = s.particles(rec)
        for shift in (0, 4) if precision == "fp32" else (0,):
            buf = torch.full((n * rec.itemsize + 64,), 255, dtype=torch.uint8, device="cuda")
            got = ctypes.c_int64()
            L.check(L.lib().pbpic_band_extract(s.handle, 0, s.my, s.my + 3, 2, ctypes.c_void_p(buf.data_ptr() + shift),
                                               n, ctypes.byref(got)))
            assert got.value == n
            host = buf.cpu().numpy()
            out = host[shift:shift + n * rec.itemsize].copy().view(rec)
            assert np.all(host[shift + n * rec.itemsize:] == 255) and np.all(host[:shift] == 255)
            g = want["grid"] - 1
            assert np.array_equal(out["grid"], (s.my + 3) * (g // s.my) + g % s.my + 3)
            for c in ("dx", "dy", "ux", "uy", "uz", "q", "pid"):
                assert np.array_equal(out[c], want[c]), c
        if n:
            with pytest.raises(pbpic_b200.PbpicError) as e:
                L.check(L.lib().pbpic_band_extract(s.handle, 0, s.my, s.my, 0, ctypes.c_void_p(buf.data_ptr()), n - 1,
                                                   ctypes.byref(got)))
            assert e.value.code == L.ERR_CAPACITY and got.value == n
