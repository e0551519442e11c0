"""The bounded-wait error path of the genotype-split search.  The first stage of one CTA waits for an arrival
that never comes, before any matrix product is issued, with the wait limit shortened to about 10 ms: every
role of the pair must leave its loop, the search must return EPIK2_E_TIMEOUT, and the same context must
then search correctly (its tensor memory was released).  Nothing faults: the waits simply run out."""
import numpy as np
import pytest

import epik2
import oracle as O
from conftest import f32_bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("odd", [False, True], ids=["even", "odd"])
@pytest.mark.parametrize("form", ["scan", "topk", "batch", "replicates", "dump"])
def test_expired_wait_returns_timeout_and_context_recovers(odd, form):
    g, p = O.gen_hwe(121, 2000, 200, 1000, planted=[(5, 33, 171)], effects=[0.8])
    ref = O.scan(g, p)
    with epik2.Context(0) as c:
        did = c.load(g, p)

        def call():
            if form == "scan":
                return c.scan(did)
            if form == "topk":
                return c.scan_topk(did, 32, rescore_fp64=1)[0]
            if form == "batch":
                return c.scan_batch([did, did], rescore_fp64=1)[1]
            if form == "replicates":
                return c.scan_replicates(did, np.stack([1 - p, p]))[1]
            return c.dump_tables(did)
        if form != "dump":
            before = call()
            assert before.ijk == ref["ijk"] and f32_bits(before.score) == f32_bits(ref["score"])
        c.set_wait_limit(20_000_000)  # about 10 ms
        c.test_withhold_odd_arrival() if odd else c.test_withhold_arrival()
        with pytest.raises(epik2.Epik2Error) as e:
            call()
        assert e.value.status == epik2.E_TIMEOUT
        for limit in (20_000_000, 0):  # one-shot; the same short limit still holds
            c.set_wait_limit(limit)
            b = call()
            if form != "dump":
                assert b.ijk == ref["ijk"] and f32_bits(b.score) == f32_bits(ref["score"])
            b = c.scan(did)
            assert b.ijk == ref["ijk"] and f32_bits(b.score) == f32_bits(ref["score"])
        c.unload(did)
