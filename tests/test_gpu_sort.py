"""The launched radix sort (systems above the one-launch build, and batches) at the edges of its
tiles, on a GPU: the tree of 32,769 and more bodies equals the oracle's, part-filled tiles and
several rows of the digit table, and keys that share most of their digits."""
import numpy as np
import pytest

from conftest import bits_equal, make_ctx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,spread", [(32769, 1.0), (34815, 1.0), (34816, 1.0), (34817, 1.0),
                                      (40000, 1e-6), (40000, 1e3), (263000, 1.0)])
def test_tree_equals_the_oracle(n, spread):
    from milkywayathome_client_b200 import NBodyState, models
    from oracle import bindings as ob
    pos, vel, mass, _ = models.plummer_plummer_dwarf(n, seed=n)
    pos = pos.mean(0) + spread * (pos - pos.mean(0))
    ctx = make_ctx(n, theta=1.0)
    want = ob.tree(ctx.struct, pos, mass, ctx.treeRSize)
    with NBodyState.create(ctx, pos, vel, mass, gravmap=False) as st:
        assert st.makeTree(ctx) == want["status"]
        if want["status"]:
            return
        got = st.tree()
    for k in ("next", "body", "depth"):
        assert np.array_equal(got[k], want[k]), k
    for k in ("pos", "mass", "rcrit2", "quad"):
        assert bits_equal(got[k], want[k]), k
