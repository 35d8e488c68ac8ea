"""What the differentiable form keeps: a gradient takes no more device memory
than states of cell words, offsets and momenta (24 bytes a particle in FP32, 44 in FP64), one a checkpoint
and one a step of a segment and two more, with two sets of particle adjoints; and its
states, some of which are formed again when they are needed, give the same gradient
for segments of every length."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

P = dict(psi0=0.1, nb=0.2, ti_te=5.0)


@pytest.mark.parametrize("precision,nsteps,every", [("fp32", 4, 1), ("fp32", 6, 3), ("fp32", 64, 8), ("fp64", 12, 4),
                                                    ("fp64", 3, 20)])
def test_memory_of_a_gradient(gpu_lib, precision, nsteps, every):
    import torch

    from pbpic_b200.autograd import DiffEngine
    mx, my, ppc = 256, 128, 64
    n, real = 2 * mx * my * ppc, 4 if precision == "fp32" else 8
    state = n * (4 + 5 * real) + 6 * mx * (my + 1) * real
    nseg = -(-nsteps // every)
    planes = 20 * mx * (my + 1) * 8 + (mx + 1) * (my + 1) * 8 * (real + 8)
    allowed = (nseg + every + 2) * state + 10 * real * n + planes
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    with DiffEngine(mx, my, ppc, nsteps=nsteps, checkpoint_every=every, precision=precision):
        used = before - torch.cuda.mem_get_info()[0]
    # (each allocation is rounded up to at most 2 MB; two a state and 20 more)
    assert used <= allowed + (2 << 20) * (2 * (nseg + every) + 20), (used, allowed)


@pytest.mark.parametrize("loss", ["magnetic", "jdote"])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("nsteps", [1, 2, 5, 7])
def test_segments_of_every_length(gpu_lib, precision, loss, nsteps):
    """One segment, more steps a segment than there are, a last segment of one step, segments of one step: the
    gradient from kept and from recomputed states (bars of test_gpu_diff_order.py)."""
    from pbpic_b200.autograd import DiffEngine
    tol = 1e-10 if precision == "fp64" else 1e-5
    ref = None
    for every in (nsteps, nsteps + 3, 1, 2, 3, 4):
        with DiffEngine(17, 9, 5, nsteps=nsteps, checkpoint_every=every, precision=precision, loss=loss) as e:
            value = e.forward(**P)
            g = [np.array(e.backward()), np.array(e.backward())]
            assert abs(e.forward(**P) - value) <= 1e-12 * abs(value)
            g.append(np.array(e.backward()))
        ref = ref or (value, g[0])
        assert abs(value - ref[0]) <= 1e-12 * abs(ref[0])
        for x in g:
            assert np.all(np.abs(x - ref[1]) <= tol * np.abs(ref[1]).max())
