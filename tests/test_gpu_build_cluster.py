"""The one-launch build of small systems at the edges of its split, on a GPU: fewer bodies than
blocks, part-filled blocks and rounds, both sides of its line, chains deeper than the sort key,
test particles, node arrays that have to grow.  Trees equal the oracle's bit for bit; the two
sides of the line meet on the same bodies."""
import numpy as np
import pytest

from conftest import bits_equal, make_ctx

pytestmark = pytest.mark.gpu


def _tree_equal(ctx, pos, vel, mass):
    from milkywayathome_client_b200 import NBodyState
    from oracle import bindings as ob
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


@pytest.mark.parametrize("n", [1, 2, 3, 7, 8, 9, 255, 257, 1023, 1025, 8191, 8193, 16385, 32767, 32768,
                               32769])
def test_tree_equals_the_oracle(n):
    from milkywayathome_client_b200 import models
    pos, vel, mass, _ = models.plummer_plummer_dwarf(n, seed=n)
    _tree_equal(make_ctx(max(n, 2), theta=0.7), pos, vel, mass)


@pytest.mark.parametrize("case", ["deep chains", "equal keys", "test particles", "all massless",
                                  "coincident", "one octant", "growing root"])
def test_unusual_systems(case):
    from milkywayathome_client_b200 import models
    n = 2000
    pos, vel, mass, _ = models.plummer_plummer_dwarf(n, seed=5)
    mass = mass.copy()
    if case == "deep chains":
        pos = np.round(pos * 2.0) / 2.0 + np.arange(n)[:, None] * 2.0 ** -41
    elif case == "equal keys":
        pos = pos.copy()
        pos[1::2] = pos[::2] + 1e-12 * (1.0 + np.arange(n // 2))[:, None] / n
    elif case == "test particles":
        mass[::5] = 0.0
    elif case == "all massless":
        mass[:] = 0.0
    elif case == "coincident":
        pos = pos.copy()
        pos[17] = pos[1400]
    elif case == "one octant":
        pos = np.abs(pos)
    else:
        pos = pos * 1e6
    _tree_equal(make_ctx(n, theta=0.8), pos, vel, mass)
