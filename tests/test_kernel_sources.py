"""Rules of the CUDA sources that no run can show to be broken."""
import glob
import os

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pydiskann_b200", "csrc")


def test_no_exchange_among_whichever_lanes_are_active():
    """__activemask() names the lanes that happen to run together, not those
    that must take part: an exchange under it may leave a partner out."""
    for f in glob.glob(os.path.join(CSRC, "*.cu*")):
        with open(f) as h:
            assert "__activemask" not in h.read(), os.path.basename(f)
