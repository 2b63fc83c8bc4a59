"""Device tables are written through table_upload, which orders the copy behind
queued work that may still read a reused pool buffer: no other source writes
device memory on the legacy stream, which does not wait for the library's.  No
GPU."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "jvsip_gb300", "csrc")


def test_no_copy_on_the_legacy_stream():
    for path in glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")):
        src = re.sub(r"//[^\n]*", "", open(path).read())
        assert not re.search(r"\bcudaMem(cpy|set)(ToSymbol|2D|3D)?\s*\(", src), os.path.basename(path)
