"""A CTA whose bounded wait has expired leaves early.  Copies into its shared memory that are still under way then have to be
awaited by whoever requested them: read from the sources, since the case itself is not one to bring about on a GPU."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "megafold_b200", "csrc")


def kernels():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = open(path).read()
        if "mbar_expect_tx(" in text:
            yield os.path.basename(path), text


@pytest.mark.parametrize("name,text", list(kernels()), ids=[n for n, _ in kernels()])
def test_every_requested_copy_is_awaited_before_exit(name, text):
    pointers = re.findall(r"uint64_t\* (\w+) = &bar\.(\w+)", text)

    def barriers(pattern):
        names = set(re.findall(pattern + r"\(&?(?:bar\.)?(\w+)", text))
        return {n for n in names if n not in dict(pointers)} | {b for p, b in pointers if p in names}

    requested, awaited = barriers("mbar_expect_tx"), barriers("(?:drain\\w*|mbar_wait)")
    assert requested and requested <= awaited, sorted(requested - awaited)
