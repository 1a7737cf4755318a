"""The bottom-up moments (eight lanes a cell, four cells a warp) on a GPU where they can go wrong:
fewer cells than a warp holds, cells of two to eight children, long chains of single-child cells (tight
pairs), massless bodies, cells of every criterion with and without quadrupoles.  The accelerations
of a walk that opens almost nothing equal the oracle's bit for bit."""
import numpy as np
import pytest

from conftest import bits_equal, make_ctx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 3, 9, 40, 257, 4001])
@pytest.mark.parametrize("cfg", [dict(criterion="TreeCode"), dict(criterion="SW93"),
                                 dict(criterion="BH86"), dict(useQuad=False)],
                         ids=["treecode", "sw93", "bh86", "noquad"])
@pytest.mark.parametrize("pairs", [False, True])
def test_moments_equal_the_oracle(n, cfg, pairs):
    from milkywayathome_client_b200 import NBodyState, models
    from oracle import bindings as ob
    pos, vel, mass, _ = models.plummer_plummer_dwarf(n, seed=n)
    if pairs:
        pos[1::2] = pos[:2 * (n // 2):2] + 1e-8
        mass = mass.copy()
        mass[::5] = 0.0
    ctx = make_ctx(n, theta=1.0, allowIncest=True, **cfg)
    rc, want, _, _ = ob.grav_map(ctx.struct, pos, mass, ctx.treeRSize)
    with NBodyState.create(ctx, pos, vel, mass, gravmap=False) as st:
        got_rc = st.gravMap(ctx)
        got = st.accels()
    assert got_rc == rc
    assert bits_equal(got, want)
