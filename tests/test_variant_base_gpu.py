"""The ablation switches' round kernel with every technique on, the base that the
switches are compared with: the oracle's forest, and no fewer atomics without
its guards."""
import numpy as np
import pytest

import ecl_mst as E
import oracle_lib as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [6, 14, 17])
@pytest.mark.parametrize("kw", [dict(), dict(mode=E.THRESH_NONE)])
def test_variant_base(scale, kw):
    g = E.gen_rmat(scale, 16, 0.57, 0.19, 0.19, scale, 1 << 20)
    with E.Context(g.nodes, g.edges) as c:
        atomics = {}
        for flags in (E.FLAG_VARIANT_BASE, E.FLAG_NO_GUARDS):
            got, st = c.run_host(g, E.make_opts(flags=flags | E.FLAG_STATS, **kw))
            want, weight, _ = O.oracle_mst(g.nindex, g.nlist, g.eweight, st["threshold"], st["filtered"])
            assert st["status"] == 0 and np.array_equal(got, want) and st["forest_weight"] == weight
            atomics[flags] = st["atomics"]
    assert 0 < atomics[E.FLAG_VARIANT_BASE] <= atomics[E.FLAG_NO_GUARDS]
