"""k-omega of few sensors at the lengths where the R2C rows change kernels (4, 40
sensors; 256 to 8192 samples), column-major spectrum: tapered data bit for bit,
power, imaginary part and gram against numpy in 64 bits (tolerances of the
pipeline: rel-L2 1e-6 log2 of the sizes, twice that for squares)."""
import pytest

from test_gpu_dif import test_komega_column_major as check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns,nt", [(2, 8192), (3, 256), (4, 512), (4, 1024), (5, 512), (5, 4096), (8, 2000), (40, 256),
                                   (40, 2048), (40, 3000), (42, 2048), (42, 256)])
def test_few_sensors(ns, nt):
    check(ns, nt)
