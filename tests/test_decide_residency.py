"""The CTA decide kernels are sized for two 1024-thread (eight 256-thread) CTAs per
SM: the register bound that keeps them there is part of the declaration, since
the compiler's own choice changes with the body."""
import os
import re

from conftest import PKG


def test_cta_kernels_bound_their_registers():
    with open(os.path.join(PKG, "csrc", "phase1.cu")) as f:
        text = f.read()
    m = re.search(r"__launch_bounds__\(([^)]*)\) k_decide_cta\(", text)
    block, blocks = [x.strip() for x in m.group(1).split(",")]
    assert block == "BLOCK"
    for b in (256, 512, 1024):
        assert eval(blocks.replace("/", "//"), {"BLOCK": b}) * b == 2048
