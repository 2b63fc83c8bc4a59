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


def test_the_buffer_of_gathered_tables_goes_back_last():
    """A plan's tables lie in one buffer that starts at d_tw.  Once that is back in the
    pool another thread can get memory at a pointer into it, which freeing that
    pointer would then take away: d_tw is freed after the others, in one place."""
    src = open(os.path.join(CSRC, "jv_plan.cu")).read()
    frees = re.findall(r"dfree\(\w+->(d_\w+)\)", src)
    tables = [f for f in frees if f in ("d_tw", "d_thalf", "d_twp", "d_twg", "d_pc")]
    assert sorted(tables) == ["d_pc", "d_thalf", "d_tw", "d_twg", "d_twp"] and tables[-1] == "d_tw"
