"""The octree build on a GPU: the one-launch build of small systems at the edges of its split (fewer
bodies than blocks, part-filled blocks and rounds, both sides of its line), and unusual systems in it
and in the launched phases above the line: chains deeper than the sort key, runs of equal keys, test
particles, node arrays that have to grow, bodies too close to part.  Trees equal the oracle's bit for
bit."""
import numpy as np
import pytest

from conftest import bits_equal, make_ctx

pytestmark = pytest.mark.gpu


def _tree_equal(ctx, pos, vel, mass, fails=False):
    from milkywayathome_client_b200 import NBodyState
    from oracle import bindings as ob
    want = ob.tree(ctx.struct, pos, mass, ctx.treeRSize)
    assert (want["status"] != 0) == fails
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


@pytest.mark.parametrize("n", [2000, 32771])        # the one-launch build; the launched phases
@pytest.mark.parametrize("case", ["deep chains", "equal keys", "long runs", "too close", "test particles",
                                  "all massless", "coincident", "one octant", "growing root"])
def test_unusual_systems(case, n):
    from milkywayathome_client_b200 import models
    pos, vel, mass, _ = models.plummer_plummer_dwarf(n, seed=5)
    pos, mass = pos.copy(), mass.copy()
    k = np.arange(n)
    if case == "deep chains":                   # more than the 2 n + 64 nodes there are at first
        pos = np.round(pos * 2.0) / 2.0 + k[:, None] * 2.0 ** -41
    elif case == "equal keys":                  # pairs closer than the key's cells of 6e-5
        pos[1::2] = pos[:n - 1:2] + 1e-9 * (1.0 + k[1::2])[:, None] / n
    elif case == "long runs":                   # of 50 bodies, in falling order
        pos = pos[k // 50 * 50] + 1e-7 * (50 - k % 50)[:, None] * np.array([1.0, -1.0, 0.5])
    elif case == "too close":                   # apart on the grid, below the smallest cell
        pos[17], pos[1400] = 3e-17, 6e-17
    elif case == "test particles":
        mass[::5] = 0.0
    elif case == "all massless":
        mass[:] = 0.0
    elif case == "coincident":
        pos[17] = pos[1400]
    elif case == "one octant":
        pos = np.abs(pos)
    else:
        pos = pos * 1e6
    _tree_equal(make_ctx(n, theta=0.8), pos, vel, mass, fails=case in ("too close", "coincident"))
