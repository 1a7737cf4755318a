"""The Exact criterion's direct sum at the edges of its split, on a GPU: part-filled groups of
sources, one, two and four lanes a body (the lines lie at 4,736 and 9,472 bodies on 148 SMs), and
operands its shared reciprocals leave to the operators; bit for bit the oracle's."""
import numpy as np
import pytest

from conftest import bits_equal, make_ctx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 15, 17, 31, 32, 33, 63, 65, 4735, 4736, 4737, 9472, 9473])
def test_sizes_equal_the_oracle(n):
    from milkywayathome_client_b200 import NBodyState, models
    from oracle import bindings as ob
    pos, vel, mass, _ = models.plummer_plummer_dwarf(n, seed=70 + n)
    ctx = make_ctx(max(n, 2), criterion="Exact")
    rc, want, _, _ = ob.grav_map(ctx.struct, pos, mass, ctx.treeRSize)
    with NBodyState.create(ctx, pos, vel, mass, gravmap=False) as st:
        assert st.gravMap(ctx) == rc
        assert bits_equal(st.accels(), want)


@pytest.mark.parametrize("eps2,scale", [(0.0, 1.0), (2.0 ** -120, 1.0), (0.01, 2.0 ** -715),
                                        (0.01, 2.0 ** 705), (0.01, 0.0)])
def test_operands_outside_the_shared_ranges(eps2, scale):
    from milkywayathome_client_b200 import NBodyState, models
    from oracle import bindings as ob
    pos, vel, mass, _ = models.plummer_plummer_dwarf(300, seed=3)
    ctx = make_ctx(300, criterion="Exact", eps2=eps2, potential=None)
    mass = mass * scale
    rc, want, _, _ = ob.grav_map(ctx.struct, pos, mass, ctx.treeRSize)
    with NBodyState.create(ctx, pos, vel, mass, gravmap=False) as st:
        assert st.gravMap(ctx) == rc
        assert np.array_equal(st.accels(), want, equal_nan=True)


@pytest.mark.parametrize("every", [1, 3, 8])
def test_test_particles(every):
    """Massless sources of either sign of zero beside massive ones, a subnormal mass among them."""
    from milkywayathome_client_b200 import NBodyState, models
    from oracle import bindings as ob
    n = 1003
    pos, vel, mass, _ = models.plummer_plummer_dwarf(n, seed=4)
    mass = mass.copy()
    mass[::every] = 0.0
    mass[::2 * every] = -0.0
    mass[500:502] = 5e-324, -3e-310
    ctx = make_ctx(n, criterion="Exact")
    rc, want, _, _ = ob.grav_map(ctx.struct, pos, mass, ctx.treeRSize)
    with NBodyState.create(ctx, pos, vel, mass, gravmap=False) as st:
        assert st.gravMap(ctx) == rc
        assert bits_equal(st.accels(), want)


@pytest.mark.parametrize("criterion,form", [("Exact", 0), ("TreeCode", 0), ("TreeCode", 1)])
def test_operands_next_to_midpoints(criterion, form):
    """Two bodies so close that s = |dr|^2 + eps^2 is eps^2: the softened distances whose root or
    reciprocal lies next to a midpoint of two doubles (tests/test_rdiv.py), with the device's own
    reciprocal estimate."""
    from milkywayathome_client_b200 import NBodyState
    from test_rdiv import HARD_RECIPROCALS, hard_roots
    d = 2.0 ** -30
    pos, vel = np.array([[0.0, 0.0, 0.0], [d, 0.0, 0.0]]), np.zeros((2, 3))
    rng = np.random.default_rng(1)
    for s in hard_roots() + HARD_RECIPROCALS:
        for k in (0, 1, 9):
            eps2 = s * 4.0 ** k
            mass = 1.0 + rng.integers(0, 1 << 52, 2) * 2.0 ** -52
            ctx = make_ctx(2, criterion=criterion, theta=0.5, eps2=eps2, potential=None)
            assert d * d + eps2 == eps2
            with NBodyState.create(ctx, pos, vel, mass, gravmap=False) as st:
                st.set_walk_form(form)
                assert st.gravMap(ctx) == 0
                acc = st.accels()
            want = ((mass[::-1] / np.sqrt(eps2)) / eps2) * np.array([d, -d])
            assert bits_equal(acc[:, 0], want) and not acc[:, 1:].any(), (s, k)
