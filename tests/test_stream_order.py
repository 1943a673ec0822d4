"""A context's stream does not wait for the default stream, so nothing in the
library may fill a device buffer there: a clear that is still under way would
overlap what the context's next launch writes. (cudaMemset takes the default
stream and returns before it is done.)"""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "phantom_gb300", "csrc")


def test_no_clear_on_the_default_stream():
    found = []
    for f in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = re.sub(r"//[^\n]*", "", open(f).read())
        found += [(os.path.basename(f), m.group(0)) for m in re.finditer(r"\bcudaMemset\w*\s*\([^;]*;", text)
                  if not re.match(r"cudaMemsetAsync\s*\(.*(\bst\b|->stream|\bstream)\)\s*;", m.group(0), re.S)]
    assert not found
