"""The download's ways (a plane at a time, chunks by one thread, by three to
eight) at the sizes where the rule changes, by rows and by columns."""
import pytest

from coldplate_solver_b200 import cps
from test_download_gpu import test_download_returns_the_uploaded_fields as check

pytestmark = pytest.mark.gpu


# planes of 382 and 386 KB; eight fields just below and above 4, 5, 10 and 15 MB
@pytest.mark.parametrize("M,N", [(190, 255), (191, 256), (255, 255), (256, 257), (286, 284), (287, 287), (404, 404),
                                 (405, 406), (495, 495), (496, 497)])
@pytest.mark.parametrize("layout", [cps.CPS_ROW_MAJOR, cps.CPS_COL_MAJOR])
def test_download_at_the_rule_s_edges(M, N, layout):
    check(M, N, layout)
