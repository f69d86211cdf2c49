"""Warp-wide exchanges name the lanes that take part.  A mask of the lanes that happen
to be converged (``__activemask``) makes a shuffle's result depend on how the
compiler scheduled the branches before it."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "jax_cosmo_gb300", "csrc")


def test_masks_are_known_by_construction():
    found = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        with open(path) as f:
            found += [f"{os.path.basename(path)}:{i}" for i, line in enumerate(f, 1) if re.search(r"__activemask\s*\(", line)]
    assert not found, found
