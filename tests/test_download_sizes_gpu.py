"""The download's ways (a plane at a time, chunks by one thread, by four, by
eight) at the sizes where the rule changes, by rows and by columns."""
import pytest

from coldplate_solver_b200 import cps
from test_download_gpu import test_download_returns_the_uploaded_fields as check

pytestmark = pytest.mark.gpu


# planes of 382 and 386 KB; eight fields of 11.9, 12.2, 23.97 and 24.3 MB
@pytest.mark.parametrize("M,N", [(190, 255), (191, 256), (443, 440), (444, 448), (626, 626), (630, 632)])
@pytest.mark.parametrize("layout", [cps.CPS_ROW_MAJOR, cps.CPS_COL_MAJOR])
def test_download_at_the_rule_s_edges(M, N, layout):
    check(M, N, layout)
