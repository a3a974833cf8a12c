"""The cubic that stands in for some exponentials of the attention forward kernels (no GPU needed)."""
import os
import re

import numpy as np

HEADER = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gpt_moe_b200", "csrc", "attention", "attn_math.cuh")


def test_error_of_the_polynomial():
    text = open(HEADER).read()
    c1, c2, c3 = (np.float32(re.search(rf"POLY_C{i} = ([0-9.]+)f", text).group(1)) for i in (1, 2, 3))
    f = np.linspace(-0.5, 0.5, 100001).astype(np.float32)
    value = ((c3 * f + c2) * f + c1) * f + np.float32(1.0)
    error = value / np.exp2(f.astype(np.float64)) - 1
    assert np.abs(error).max() < 1.03e-4                    # the bound that the header states
    assert value[50000] == 1.0                              # 2^0
