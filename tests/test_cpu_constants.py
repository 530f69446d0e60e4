"""Constants folded from several are the floats nearest to their exact products (a product of rounded factors can be a
unit in the last place off, which a product of hundreds of factors turns into a bias)."""

from __future__ import annotations

import math
import re
from pathlib import Path

import numpy as np

CSRC = Path(__file__).resolve().parents[1] / "ultrasound-3d-reconstruction_b200" / "csrc"


def test_scanline_quadrature_constants():
    text = (CSRC / "ultragray.cu").read_text()
    for name, exact in (("kNegLog2eOuter", -5.0 / 9.0 / math.log(2.0)), ("kNegLog2eMiddle", -8.0 / 9.0 / math.log(2.0))):
        value = np.float32(re.search(name + r" = (-[\d.]+)f", text).group(1))
        assert value == np.float32(exact)
    forward = text[text.index("forward_ckpt_kernel("):text.index("backward_ckpt_kernel(")]
    assert "dup2(kNegLog2eOuter)" in forward and "dup2(kNegLog2eMiddle)" in forward
