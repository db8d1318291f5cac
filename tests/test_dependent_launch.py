"""Every kernel launched with the dependent-launch attribute (pdl, chasqui_b200/csrc/chq_common.cuh)
waits for the kernel before it as its first statement: what an earlier kernel wrote is visible to a
grid only once that grid itself has waited. Checked on the sources."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "chasqui_b200", "csrc")


def test_every_dependent_kernel_waits_first():
    text = "".join(open(f).read() for f in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))))
    text = re.sub(r"//[^\n]*", "", text)
    launched = set()
    for call in re.findall(r"\bpdl\(([^;]*);", text):
        launched |= set(re.findall(r"\b(\w+_(?:kernel|batched))\b", call.split("grid", 1)[0]))
    bodies = dict(re.findall(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\((?:[^()]|\([^()]*\))*\))*\)\s*)?"
                             r"(\w+)\([^{;]*\)\s*\{\s*([^;]*;)", text))
    assert len(launched) > 35 and launched <= set(bodies), sorted(launched - set(bodies))
    late = {k: bodies[k] for k in launched if bodies[k] != "pdl_begin();"}
    assert not late, late
