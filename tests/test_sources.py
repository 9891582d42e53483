"""Properties of the CUDA sources that no run on one GPU shows."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pot_gb300", "csrc")


def _sources():
    out = {}
    for f in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        with open(f) as h:
            out[os.path.basename(f)] = h.read()
    return out


def test_no_multicast_loads():
    """The library also runs with one process per GPU on several GPUs, where
    bulk copies into more than one CTA are not used."""
    for name, text in _sources().items():
        for line in text.splitlines():
            assert not re.search(r"cp\.async\.bulk[^\"]*multicast", line), name
