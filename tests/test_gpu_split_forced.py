"""The genotype-split search at sizes and on data where the library would take other kernels (small searches,
constant SNPs): its own edge tests, and the tests of the pinned engines (recorded tables and scores of the
reference, the oracle's), on a context that takes it wherever its counts fit."""
import pytest

import epik2
from test_gpu_parity import *  # noqa: F401,F403
from test_gpu_split import *  # noqa: F401,F403
from test_gpu_tiles import test_every_table_across_many_tiles_vs_oracle  # noqa: F401
from test_gpu_precision import test_top32_fp64_matches_oracle  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = epik2.Context(0)
    c.config = (0, 0, 0, 0)
    c.test_always_split()
    yield c
    c.close()


@pytest.fixture(scope="module")
def auto(ctx):
    return ctx
