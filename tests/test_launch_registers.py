"""A kernel that raises registers with setmaxnreg can only draw on what its CTA was launched with: beyond that the raise never
returns.  So every launch of such a kernel asks first how many registers the build gave it.  Read from the sources, since the case
itself is not one to bring about on a GPU."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "megafold_b200", "csrc")


def raising_kernels():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = open(path).read()
        starts = [(m.start(), m.group(1)) for m in re.finditer(r"__global__[^;{]*?\b(\w+_kernel)\(", text)]
        for (at, kernel), (end, _) in zip(starts, starts[1:] + [(len(text), "")]):
            if "setmaxnreg.inc" in text[at:end]:
                yield os.path.basename(path), kernel, text


CASES = list(raising_kernels())


def test_the_kernels_are_found():
    assert {k for _, k, _ in CASES} >= {"evo_fwd_ws_kernel", "evo_bwd_ws_kernel", "evo_dbias_ws_kernel", "lnl_fwd_tc_kernel", "lnl_bwd_tc_kernel",
                                        "transition_fwd_tc_kernel", "transition_bwd_tc_kernel"}


@pytest.mark.parametrize("name,kernel,text", CASES, ids=[k for _, k, _ in CASES])
def test_every_launch_checks_the_registers(name, kernel, text):
    launches = re.findall(rf"constexpr auto kern = {kernel}<[^;]*;(.*?)kern<<<", text, re.S)
    assert launches and len(launches) == len(re.findall(rf"\b{kernel}<", text))
    for between in launches:
        assert re.search(r"opt_in_smem<kern>\(\w+, k\w*LaunchRegs\)", between), between
