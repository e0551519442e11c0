"""What a user gets without pinning anything: the tests of the pinned engines (every table and score against
the reference's recorded ones and the oracle's, the reference's best triplets of the full-size workloads) on
contexts of the library's own choice, and of FP4 without a tuning option."""
import pytest

import epik2
from test_gpu_parity import *  # noqa: F401,F403
from test_gpu_tiles import test_every_table_across_many_tiles_vs_oracle  # noqa: F401
from test_gpu_workloads import (test_best_triplet_identical_to_reference,  # noqa: F401
                                test_planted_triplet_tables_sum_to_class_sizes)

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[epik2.ENGINE_AUTO, epik2.ENGINE_TC_FP4], ids=["auto", "fp4-free"])
def ctx(request):
    c = epik2.Context(0, engine=request.param)
    c.config = (request.param, 0, 0, 0)
    yield c
    c.close()
