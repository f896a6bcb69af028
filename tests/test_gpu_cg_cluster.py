"""FP64 CG in one thread-block cluster (needs a B200) at the edges of its
shapes: 256, 512 and 1024 threads per CTA, 1 to 16 CTAs, one row more (the last
CTA nearly empty; above 16,384 rows the grid's kernel), rows whose neighbours
lie in other CTAs, full rows of 8 entries' room; checks and tolerances of the
larger form's test."""
import pytest

from test_gpu_cg_rows import test_rows_cg_matches_oracle as check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,offsets", [
    (300, [1, 150, 290]), (512, [1, 256]), (513, [1, 256]),
    (4096, [1, 64]), (4097, [1, 64, 4000]),
    (8192, [1, 128]), (8193, [1, 512, 8000]),
    (16384, [1, 8192, 15000]), (16385, [1, 128]),
])
def test_cluster_cg_matches_oracle(mf, n, offsets):
    check(mf, n, offsets)
