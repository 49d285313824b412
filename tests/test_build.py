"""The build: a kernel's code must not depend on what else its unit holds."""
import os

from nissa_b200 import build


def test_units_are_compiled_whole():
    split = [os.path.basename(s) for s in build.sources() if "--split-compile" in build.unit_flags(s)]
    assert split == ["tms_cg_half.cu"]
    # which holds one solver's instantiation and nothing else
    code = [x for x in open(os.path.join(build.CSRC, split[0])).read().splitlines() if not x.startswith("//")]
    assert sum("template" in x for x in code) == 1 and len(code) < 8
    for s in build.sources():
        assert "-shared" not in build.unit_flags(s) and "arch=compute_100a,code=sm_100a" in build.unit_flags(s)
