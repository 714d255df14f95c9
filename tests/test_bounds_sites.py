"""Every site that the bounds-check build can name is checked somewhere in the
kernels, and the index arithmetic of the list passes, the octree and the adjoint
goes through it."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "meshtrex_b200", "csrc")


def _uses():
    uses = {}
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cu", ".cuh")):
            text = open(os.path.join(CSRC, f)).read()
            for m in re.finditer(r"\bMTX_BC\(", text):
                site = re.search(r"\bkBc\w+", text[m.end():m.end() + 400])
                if site:
                    uses.setdefault(site.group(0), set()).add(f)
    return uses


def test_every_site_is_used():
    enum = re.findall(r"^\s+(kBc\w+) = \d+,", open(os.path.join(CSRC, "mtx_device.cuh")).read(), re.M)
    assert len(enum) > 10
    assert sorted(enum) == sorted(s for s in _uses() if s in enum)


@pytest.mark.parametrize("site,where", [
    ("kBcJobs", "pmb_lists.cuh"), ("kBcVertex", "pmb_lists.cuh"), ("kBcIndex", "pmb_lists.cuh"),
    ("kBcContext", "pmb_lists.cuh"), ("kBcList", "pmb_lists.cuh"), ("kBcVoxTab", "pmb_lists.cuh"),
    ("kBcOctree", "minmax_device.cuh"), ("kBcVolume", "minmax_device.cuh"), ("kBcTerms", "adjoint.cu"),
    ("kBcTile", "adjoint.cu"), ("kBcPartial", "adjoint.cu"), ("kBcField", "adjoint.cu")])
def test_site_is_checked_in(site, where):
    assert where in _uses().get(site, ())
