"""The one-launch coarsest solve (a thread-block cluster per problem) against
the fill-based colour passes with the sweep check after each sweep: the same
sweep counts and the same bits, over the shapes the cluster form accepts."""
import numpy as np
import pytest

from samrai_b200 import configs, fac
from samrai_b200.fac import E, R

pytestmark = pytest.mark.gpu


def _level0(dim, n, cuts, var_d, c_kind, seed):
    """One-level problem of n cells per axis, cut at the given indices."""
    n = tuple(n) + (1,) * (3 - len(n))
    runs = [[(a, b - 1) for a, b in zip((0,) + tuple(cut), tuple(cut) + (m,))]
            for cut, m in zip(tuple(cuts) + ((),) * (3 - len(cuts)), n)]
    boxes = [[x[0], y[0], z[0], x[1], y[1], z[1]] for z in runs[2] for y in runs[1]
             for x in runs[0]]
    p = configs.Problem(dim=dim, n0=n, xlo=(0.0, 0.0, 0.0), xup=(1.0, 1.3, 0.7),
                        levels=[configs.Level((1, 1, 1), np.array(boxes, dtype=np.int32))])
    rng = np.random.default_rng(seed)
    p.c_kind, p.c_const = c_kind, -3.0
    if var_d:
        p.d_variable = True
        # a face that two patches share holds one value on both
        p.d = [configs.fill_side_field(p, 0, lambda X, Y, Z: np.exp(np.sin(7 * X + 5 * Y - 3 * Z)))]
    if c_kind == 2:
        p.c = [-1.0 - rng.random(configs.field_size(p, 0, 0))]
    return p


ROBIN = (np.array([1.0, 2.0, 1.0, 0.5, 1.5, 1.0]), np.array([0.5, 1.0, 0.25, 1.0, 0.0, 0.3]),
         np.zeros(6))

CASES = [
    # dim, cells, cuts, variable D, C kind, Robin, sweeps, tolerance
    (2, (1, 1), (), False, 0, False, 5, 0.0),
    (2, (3, 5), (), True, 0, True, 30, 1e-6),
    (2, (64, 64), (), False, 0, False, 40, 1e-300),
    (2, (57, 76), (), True, 2, True, 40, 1e-2),
    (2, (97, 131), (), True, 1, False, 12, 1e-300),
    (2, (40, 36), ((20,), (12, 24)), False, 1, True, 25, 1e-300),
    (3, (8, 8, 8), (), True, 0, False, 60, 1e-3),
    (3, (16, 16, 16), (), False, 2, False, 30, 1e-300),
    (3, (13, 7, 9), (), True, 2, True, 25, 1e-1),
    (3, (32, 32, 32), ((16,), (16,), (16,)), True, 0, False, 8, 1e-300),
    (3, (40, 40, 40), ((16, 32), (16, 32), (16, 32)), False, 0, False, 6, 1e-300),
    (3, (20, 12, 30), ((8,), (), (10, 20)), True, 1, True, 40, 5e-1),
]


def _run(probs, bc, fused, sweeps, tol, data):
    g = fac.FacContext(probs, bc=bc)
    g.set_fused(fused)
    for i, (e, r) in enumerate(data):
        g.upload(E, i, 0, e)
        g.upload(R, i, 0, r)
    n0 = fac.kernel_launches()
    n = g.smooth(E, R, 0, sweeps, tol)
    # the sweeps in one launch, or two colour passes and more for each
    launches = fac.kernel_launches() - n0
    assert launches <= 4 if fused else launches > 2 * int(n.max())
    out = [g.download(E, i, 0) for i in range(len(probs))]
    g.close()
    return n, out


@pytest.mark.parametrize("case", CASES, ids=lambda c: f"{c[0]}d_{'x'.join(map(str, c[1]))}")
def test_one_launch_matches_passes(case, require_gpu):
    dim, n, cuts, var_d, c_kind, robin, sweeps, tol = case
    p = _level0(dim, n, cuts, var_d, c_kind, 3)
    rng = np.random.default_rng(5)
    data = [(rng.standard_normal(configs.field_size(p, 0, 1)),
             rng.standard_normal(configs.field_size(p, 0, 0)))]
    bc = ROBIN if robin else None
    na, a = _run([p], bc, True, sweeps, tol, data)
    nb, b = _run([p], bc, False, sweeps, tol, data)
    assert np.array_equal(na, nb)
    assert np.array_equal(a[0], b[0])


def test_batch_of_sizes_stops_per_problem(require_gpu):
    probs = [_level0(3, (8 + 2 * i,) * 3, (), True, 0, i) for i in range(5)]
    rng = np.random.default_rng(9)
    data = [(0.1 * rng.standard_normal(configs.field_size(p, 0, 1)),
             10.0 ** -i * rng.standard_normal(configs.field_size(p, 0, 0)))
            for i, p in enumerate(probs)]
    na, a = _run(probs, None, True, 200, 1e-2, data)
    nb, b = _run(probs, None, False, 200, 1e-2, data)
    assert np.array_equal(na, nb) and len(set(na.tolist())) > 1
    for x, y in zip(a, b):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("lo, n", [(-5, (64, 40)), (-4, (33, 97))])
def test_negative_lower_index(lo, n, require_gpu):
    """A 2-D level 0 may start below zero along x: one launch for all sweeps,
    which are those of passes of a fixed count.  (Where the row sums that start
    the colouring turn negative and odd, both passes update the same cells; such
    levels keep to passes.)"""
    p = _level0(2, n, (), False, 0, 0)
    p.n0 = (n[0] + lo, n[1], 1)
    p.levels = [configs.Level((1, 1, 1), np.array([[lo, 0, 0, n[0] + lo - 1, n[1] - 1, 0]],
                                                  dtype=np.int32))]
    rng = np.random.default_rng(2)
    data = [(fid, rng.standard_normal(configs.field_size(p, 0, g))) for fid, g in ((E, 1), (R, 0))]
    g = fac.FacContext([p])
    g.set_staged(False)  # passes that take the Robin value of a face cell where they read it
    sweeps, outs = 20, []
    for tol in (1e-300, -1.0):
        for fid, x in data:
            g.upload(fid, 0, 0, x)
        n0 = fac.kernel_launches()
        assert g.smooth(E, R, 0, sweeps, tol)[0] == sweeps
        outs.append((fac.kernel_launches() - n0, g.download(E, 0, 0)))
    assert outs[0][0] < sweeps < outs[1][0]
    assert np.array_equal(outs[0][1], outs[1][1])
    g.close()


def test_profile_keeps_the_one_launch_solve_apart(require_gpu):
    """Its values stay on the chip: it is no colour pass over the level's
    arrays, and its bytes do not grow with the sweeps."""
    probs = [_level0(3, (8, 8, 8), (), True, 2, 0), _level0(3, (12, 8, 8), (), True, 2, 1)]
    g = fac.FacContext(probs)
    faces = sum(configs.side_size(p, 0) for p in probs)
    cells = sum(configs.field_size(p, 0, 0) for p in probs)
    for i, p in enumerate(probs):
        g.upload(R, i, 0, np.ones(configs.field_size(p, 0, 0)))
    for sweeps in (5, 50):
        g.profile(True)
        g.smooth(E, R, 0, sweeps, 1e-300)
        n, ms, by = g.profile_read(6)
        assert (n, by) == (1, 8.0 * (faces + 4 * cells)) and ms > 0.0
        assert g.profile_read(0) == (0, 0.0, 0.0)
        g.profile(True)
        g.smooth(E, R, 0, sweeps, -1.0)
        assert g.profile_read(6)[0] == 0 and g.profile_read(0)[0] == 2 * sweeps
    g.profile(False)
    with pytest.raises(fac.FacError):
        g.profile_read(7)
    g.close()
