"""Options that a build of the CUDA sources may set (-DPBPIC_...)."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pbpic_b200", "csrc")


def test_one_layout_of_gather_records():
    """The kernels that write the mixed form's gather records (k_cell_records, k_field_step) and those that read them
    (k_push, k_push_cells) agree on bilinear coefficients: an option that only some of them
    follow would give wrong fields."""
    for name in os.listdir(CSRC):
        for option in re.findall(r"#\s*ifndef\s+(PBPIC_\w+)", open(os.path.join(CSRC, name)).read()):
            assert "COEF" not in option, (name, option)
