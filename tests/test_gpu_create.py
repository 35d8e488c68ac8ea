"""What a domain's arrays take on the device."""
import pytest

import pbpic_b200
from pbpic_b200 import configs

pytestmark = pytest.mark.gpu


def test_a_domain_takes_what_its_arrays_add_up_to(gpu_lib):
    """The arrays of a domain are parts of one allocation. By themselves, those of a megabyte or more would each be
    mapped in pages of their own (2 MB): 86 MB here in place of 76, and 4.4 ms to create it in place of 0.7 ms."""
    import torch
    side, ppc = 128, 32
    n, cells = 2 * side * side * ppc, side * side
    # a particle: two buffers of cell word, offsets and momenta, keys and values of the general sort, its counters;
    # a cell: two sets of planes, node grid, gather record, two currents, counts and offsets, charge, tile tables
    arrays = n * (2 * (24 + 8) + 1) + cells * (12 * 4 + 32 + 96 + 64 + 8 + 8 + 32)
    cfg, _ = configs.uniform_c1(mx=side, my=side, ppc=ppc)
    pbpic_b200.Simulation.from_config(cfg, precision="fp32", capacity=1).close()  # (the library's code is on the device)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    with pbpic_b200.Simulation.from_config(cfg, precision="fp32", capacity=n):
        used = before - torch.cuda.mem_get_info()[0]
    assert used <= arrays + 2 * (2 << 20), (used, arrays)  # the block's rounding, and the energy history's
