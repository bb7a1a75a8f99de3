"""Ghost-fluid fixes of many cells in one pass on a mesh of several runs of cells (32 blocks collect the
flagged cells, a run each; here 8,192 cells a run): the case and bars of test_gpu_m5_crossings on
262,144 cells, and on 32,768 cells, where most blocks have none."""
import pytest

import test_gpu_m5_crossings as crossings

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("level,at_least", [(5, 10000), (6, 80000)])
def test_many_runs_match_oracle(level, at_least, built_lib, oracle_lib):
    crossings.test_many_crossings_match_oracle(level, at_least, built_lib, oracle_lib)
