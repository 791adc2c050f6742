"""Bulk loads go to the issuing CTA alone. The library runs unchanged on every rank of
a job over several GPUs, where a load that writes the shared memory of other CTAs of
its cluster is not to be used; the kernels' clusters exchange values by plain stores."""
import pathlib
import re

import pytest

CSRC = pathlib.Path(__file__).resolve().parent.parent / "vardyn_gb300" / "csrc"


@pytest.mark.parametrize("path", sorted(CSRC.glob("*.cu*")), ids=lambda p: p.name)
def test_no_multicast_form(path):
    code = re.sub(r"//[^\n]*", "", path.read_text())
    assert "multicast" not in code
