"""The threaded tree walk and list grouping against the oracle's sequential ones
(CPU): the same lists in the same order at a size that is walked in shares."""
import numpy as np
import pytest

import cabi


@pytest.mark.parametrize("waters,ncrit", [(1300, 16), (8000, 64)])
def test_lists_and_order(port, waters, ncrit):
    from cppe_gb300 import synthetic
    b = synthetic.water_box(waters, seed=3)
    info, m2l, p2p = cabi.tree_lists(b.xyz, ncrit=ncrit, theta=0.5)
    ref = port.tree_lists(b.xyz, ncrit=ncrit, theta=0.5)
    np.testing.assert_array_equal(p2p, ref["p2p"])  # walk order
    rm = ref["m2l"]
    assert (np.diff(m2l[:, 0]) >= 0).all()  # by source, ties in walk order
    np.testing.assert_array_equal(m2l, rm[np.argsort(rm[:, 0], kind="stable")])
    nvec, ne = cabi.tree_vectors(b.xyz, ncrit=ncrit, theta=0.5)
    c = ref["cells"][:, :3]
    u = 0.5 * ref["cells"][:, 3].min()
    d = np.rint((c[m2l[:, 1]] - c[m2l[:, 0]]) / u).astype(np.int64)
    assert ne == len(m2l) and nvec == len(np.unique(d, axis=0))
