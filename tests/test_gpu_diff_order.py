"""The differentiable form's cell order: gradients do not depend on where the
checkpoints lie (a recomputed segment's particles may come back in another
order than the checkpoint after it), nor on whether the last segment's states
are still there (a second backward call recomputes them); sizes around a warp
and a block of particles, sparse and dense cells.

Bars: the same FP64 terms added in another order, over 6 steps: 1e-10 of the
largest gradient entry (FP64), 1e-5 where the adjoint's state is stored in FP32."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

P = dict(psi0=0.1, nb=0.2, ti_te=5.0)


@pytest.mark.parametrize("loss", ["magnetic", "jdote"])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("mx,my,ppc", [(3, 3, 1), (5, 7, 2), (16, 8, 1), (33, 21, 3), (8, 6, 90)])
def test_checkpoints_do_not_matter(gpu_lib, precision, loss, mx, my, ppc):
    from pbpic_b200.autograd import DiffEngine
    tol = 1e-10 if precision == "fp64" else 1e-5
    ref = None
    for every in (6, 1, 2, 4):
        with DiffEngine(mx, my, ppc, nsteps=6, checkpoint_every=every, precision=precision, loss=loss) as e:
            value = e.forward(**P)
            g = [np.array(e.backward()), np.array(e.backward())]
        if ref is None:
            ref = (value, g[0])
        assert abs(value - ref[0]) <= 1e-12 * abs(ref[0])
        for x in g:
            assert np.all(np.isfinite(x))
            assert np.all(np.abs(x - ref[1]) <= tol * np.abs(ref[1]).max())
