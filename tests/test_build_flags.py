"""How the kernels are compiled: for sm_100a alone, without fused multiply-add contraction (the FP64
paths reproduce the reference's operations), and every file as one unit: split compilation chooses
other registers, which cost the shake 18% and the detector 10 to 25%."""
import os

MAKEFILE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                        "pyopenlpt_b200", "csrc", "Makefile")


def test_flags():
    with open(MAKEFILE) as f:
        text = "".join(line for line in f if not line.lstrip().startswith("#"))
    assert "arch=compute_100a,code=sm_100a" in text
    assert "--fmad=false" in text
    assert "split-compile" not in text
