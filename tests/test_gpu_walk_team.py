"""The team walk (form 0 of the FP64 walk) at the sizes where it can go wrong, on a GPU: fewer
bodies than a team, remainders, both sides of its lines, and operands its shared reciprocals
leave to the operators; the choice of the form, by rule and by timing.  The accelerations equal the oracle's (small sizes) and the per-lane
walk's bit for bit."""
import numpy as np
import pytest

from conftest import bits_equal, make_ctx

pytestmark = pytest.mark.gpu


def _acc(ctx, pos, vel, mass, form):
    from milkywayathome_client_b200 import NBodyState
    with NBodyState.create(ctx, pos, vel, mass, gravmap=False) as st:
        st.set_walk_form(form)
        rc = st.gravMap(ctx)
        return rc, st.accels()


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 7, 8, 9, 15, 17, 31, 33, 1000, 1025])
@pytest.mark.parametrize("cfg", [dict(theta=0.5), dict(theta=1.0, criterion="SW93"),
                                 dict(theta=0.8, useQuad=False), dict(theta=0.0)],
                         ids=["t0.5", "sw93", "noquad", "t0"])
def test_small_sizes_equal_the_oracle(n, cfg):
    from milkywayathome_client_b200 import models
    from oracle import bindings as ob
    pos, vel, mass, _ = models.plummer_plummer_dwarf(n, seed=40 + n)
    ctx = make_ctx(max(n, 2), **cfg)
    rc, want, _, _ = ob.grav_map(ctx.struct, pos, mass, ctx.treeRSize)
    got_rc, got = _acc(ctx, pos, vel, mass, 0)
    assert got_rc == rc and bits_equal(got, want)


@pytest.mark.parametrize("n", [12288, 12289, 24576, 24577])
@pytest.mark.parametrize("quad", [True, False])
def test_the_automatic_choice_equals_every_form(n, quad):
    """Both sides of its lines, with and without quadrupoles."""
    from milkywayathome_client_b200 import models
    pos, vel, mass, _ = models.plummer_plummer_dwarf(n, seed=6)
    ctx = make_ctx(n, theta=0.9, useQuad=quad)
    rc, want = _acc(ctx, pos, vel, mass, 1)
    assert rc == 0
    for form in (-1, 0, 2):
        rc, got = _acc(ctx, pos, vel, mass, form)
        assert rc == 0 and bits_equal(got, want), form


@pytest.mark.parametrize("n,quad,theta,evaluations", [
    (1500, True, 0.0, 6), (1500, False, 0.19, 6), (12289, True, 0.15, 6), (24576, True, 0.19, 6),
    (24577, True, 0.49, 6), (12289, False, 0.3, 6), (32769, True, 0.4, 6), (24577, True, 0.5, 4),
    (12289, False, 0.5, 4)])
def test_the_timed_choice(n, quad, theta, evaluations):
    """Where no rule decides, the first evaluations do, with form 0 among the forms below theta 0.5."""
    from milkywayathome_client_b200 import NBodyState, models
    pos, vel, mass, _ = models.plummer_plummer_dwarf(n, seed=6)
    ctx = make_ctx(n, theta=theta, useQuad=quad)
    _, want = _acc(ctx, pos, vel, mass, 1)
    with NBodyState.create(ctx, pos, vel, mass, gravmap=False) as st:
        for k in range(evaluations):
            assert st.walk_form() == -1
            assert st.gravMap(ctx) == 0 and bits_equal(st.accels(), want)
        assert st.walk_form() in ((0, 1, 2) if evaluations == 6 else (1, 2))


@pytest.mark.parametrize("n,quad,theta", [(1500, True, 0.04), (12288, True, 0.05), (12289, True, 0.2),
                                          (24576, True, 0.2), (12288, False, 0.2)])
def test_the_team_walk_by_rule(n, quad, theta):
    from milkywayathome_client_b200 import NBodyState, models
    pos, vel, mass, _ = models.plummer_plummer_dwarf(n, seed=6)
    ctx = make_ctx(n, theta=theta, useQuad=quad)
    _, want = _acc(ctx, pos, vel, mass, 1)
    with NBodyState.create(ctx, pos, vel, mass, gravmap=False) as st:
        assert st.gravMap(ctx) == 0 and st.walk_form() == 0
        assert bits_equal(st.accels(), want)


@pytest.mark.parametrize("sizes,theta,quad", [
    ((3100, 2900, 3200, 3088), 0.5, True), ((3100, 2900, 3200, 3088), 0.0, True),   # 12,288 in all
    ((3100, 2900, 3201, 3088), 0.5, True), ((3100, 2900, 3201, 3088), 0.25, True),
    ((3100, 2900, 3201, 3088), 0.5, False), ((2467, 31, 2503, 4999) * 3, 0.2, True),
    ((2467, 31, 2503, 4999) * 3, 0.6, True), ((30011, 9990, 60000), 0.3, True),
    ((30011, 9990, 60000), 0.3, False)])
def test_the_batch_rule_equals_the_per_lane_walk(sizes, theta, quad):
    """Both sides of the lines of a batch's rule: teams, unions (of warps that hold bodies of two
    dwarfs, too) and both per-lane walks."""
    from milkywayathome_client_b200 import NBodyBatch, models
    dwarfs = [models.plummer_plummer_dwarf(n, seed=k)[:3] for k, n in enumerate(sizes)]
    ctx = make_ctx(sizes[0], theta=theta, useQuad=quad)
    with NBodyBatch([(n, ctx.eps2 * (1 + k), ctx.timestep, ctx.treeRSize)
                     for k, n in enumerate(sizes)]) as bt:
        got = []
        for form in (0, 1, 2):
            bt.set_walk_form(form)
            bt.set_bodies(*(np.concatenate([d[c] for d in dwarfs]) for c in range(3)))
            assert bt.gravMap(ctx) == 0
            got.append(bt.accels())
    assert bits_equal(got[0], got[1]) and bits_equal(got[2], got[1])


def test_the_automatic_choice_follows_the_context():
    """A state's evaluations with and without quadrupoles each take the form of their own: the
    team walk by its line (20,000 lies between the two), the timed choice kept for its kind."""
    from milkywayathome_client_b200 import NBodyState, models
    n = 20000
    pos, vel, mass, _ = models.plummer_plummer_dwarf(n, seed=6)
    quad, mono = make_ctx(n, theta=0.9), make_ctx(n, theta=0.9, useQuad=False)
    with NBodyState.create(quad, pos, vel, mass, gravmap=False) as st:
        assert st.walk_form() == -1
        seen = []
        for ctx in (quad, mono, mono, quad, mono, mono, quad, mono):
            assert st.gravMap(ctx) == 0
            seen.append(st.walk_form())
        assert [seen[k] for k in (0, 3, 6)] == [0, 0, 0]
        assert [seen[k] for k in (1, 2, 4)] == [-1, -1, -1]     # four evaluations decide
        assert seen[5] in (1, 2) and seen[7] == seen[5]


@pytest.mark.parametrize("n,theta", [(32767, 0.9), (32768, 0.9), (32769, 0.9), (12288, 0.1),
                                     (12289, 0.03), (12289, 0.05), (20001, 0.12), (20001, 0.14)])
def test_both_sides_of_the_line_equal_the_per_lane_walk(n, theta):
    """Form 0: the team walk on one side of its lines, the union of a warp's paths on the other."""
    from milkywayathome_client_b200 import models
    pos, vel, mass, _ = models.plummer_plummer_dwarf(n, seed=5)
    ctx = make_ctx(n, theta=theta)
    a, b = (_acc(ctx, pos, vel, mass, f) for f in (0, 1))
    assert a[0] == b[0] == 0 and bits_equal(a[1], b[1])


@pytest.mark.parametrize("case", ["no softening", "tiny masses", "huge masses", "tiny sizes",
                                  "massless bodies", "near ones"])
def test_operands_outside_the_shared_ranges(case):
    from milkywayathome_client_b200 import _lib, models
    from oracle import bindings as ob
    n = 700
    pos, vel, mass, _ = models.plummer_plummer_dwarf(n, seed=8)
    over = dict(theta=0.7, potential=None, allowIncest=True)
    if case == "no softening":
        over["eps2"] = 0.0
    elif case == "tiny masses":
        mass = mass * 2.0 ** -715
    elif case == "huge masses":
        mass = mass * 2.0 ** 705
    elif case == "tiny sizes":
        over["eps2"] = 2.0 ** -120
    elif case == "massless bodies":
        mass = mass.copy()
        mass[::9] = 0.0
    else:
        # softened distances next to powers of two: s = 4 - 2^-k and neighbours
        pos = np.round((pos - pos.mean(0)) * 2.0) / 2.0
        pos += np.arange(n)[:, None] * 2.0 ** -40
        over["eps2"] = 4.0 - 2.0 ** -50
    ctx = make_ctx(n, **over)
    rc, want, _, _ = ob.grav_map(ctx.struct, pos, mass, ctx.treeRSize)
    for form in (0, 1, 2):
        got_rc, got = _acc(ctx, pos, vel, mass, form)
        assert got_rc == rc, form
        if not _lib.status_is_fatal(rc):
            assert np.array_equal(got, want, equal_nan=True), form
