"""The kernel sets of the model families (a checkout without the full library compiles only one of them)."""
import re

import pytest

from minisgl.ops import build


@pytest.mark.parametrize("name", list(build.KERNEL_SETS))
def test_projections_are_in_every_set(name):
    """Sizes decide which kernel a projection runs on, so a set has all that ``ops/gemm.py`` calls."""
    called = set(re.findall(r'nv\.call\("(\w+)"', (build.HERE / "gemm.py").read_text()))
    here = "".join((build.CSRC / f"{n}.cu").read_text() for n in build.KERNEL_SETS[name])
    missing = {c for c in called if f"dsv4_{c}(" not in here}
    assert len(called) > 5 and not missing, missing
