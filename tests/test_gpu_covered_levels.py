"""Solves on hierarchies whose first levels lie wholly under finer ones.

Such a level holds no part of the composite problem (weights 0), so a solve
leaves u, the operator and the residual on it until its end, skips flux sums
and fix-ups of covered cells, and keeps Krylov vectors only where cells are
uncovered.  (Only the first levels can be like this: a level that covers the
next coarser one has no coarse-fine boundary, so it covers the domain.)  Here
u with all its ghost values and the residual on every level after a solve are
those of the level operators, which work on whole levels, bit for bit, and so
are the residual norms of every cycle.
"""
import numpy as np
import pytest

from samrai_b200 import configs, fac
from samrai_b200.fac import E, F, R, U

pytestmark = pytest.mark.gpu

# a caller's coefficient object: the solve leaves boundary ghosts as last filled
ROBIN = (np.array([1.0, 2.0, 1.0, 0.5, 1.5, 1.0]), np.array([0.5, 1.0, 0.25, 1.0, 0.0, 0.3]),
         np.array([0.1, -0.2, 0.05, 0.3, 0.2, -0.1]))


def _grid(dim, lo, hi, cuts):
    """Boxes of [lo, hi] cut into `cuts` runs per axis."""
    b = np.linspace(lo, hi + 1, cuts + 1).astype(int)
    runs = [(x, y - 1) for x, y in zip(b[:-1], b[1:])]
    zs = runs if dim == 3 else [(0, 0)]
    return np.array([[x[0], y[0], z[0], x[1], y[1], z[1]] for z in zs for y in runs for x in runs],
                    dtype=np.int32)


def _problem(dim, n, levels, seed, var_d=True):
    """levels: (first cell, last cell, cuts) per axis and level, at ratio 2."""
    lv = []
    for ln, (lo, hi, cuts) in enumerate(levels):
        r = 1 if ln == 0 else 2
        lv.append(configs.Level((r, r, r if dim == 3 else 1), _grid(dim, lo, hi, cuts)))
    p = configs.Problem(dim=dim, n0=(n, n, n if dim == 3 else 1), xlo=(0.0,) * 3, xup=(1.0,) * 3,
                        levels=lv)
    rng = np.random.default_rng(seed)
    p.f = [rng.standard_normal(configs.field_size(p, ln, 0)) for ln in range(p.nlev)]
    p.u0 = [0.01 * rng.standard_normal(configs.field_size(p, ln, 1)) for ln in range(p.nlev)]
    if var_d:
        p.d_variable = True
        p.d = [configs.fill_side_field(p, ln, lambda X, Y, Z: np.exp(np.sin(5 * X + 4 * Y + 3 * Z)))
               for ln in range(p.nlev)]
    return p


# name: (problems, levels of the library's extension)
HIERARCHIES = {
    "2d_one_covered": lambda: ([_problem(2, 32, [(0, 31, 1), (0, 63, 2), (40, 95, 2)], 1)], 0),
    "2d_two_covered": lambda: ([_problem(2, 16, [(0, 15, 1), (0, 31, 1), (0, 63, 2),
                                                 (32, 79, 3)], 2, False)], 0),
    "2d_covered_in_one_problem": lambda: ([_problem(2, 32, [(0, 31, 1), (0, 63, 2), (40, 95, 2)], 3),
                                           _problem(2, 24, [(0, 23, 1), (8, 39, 2), (24, 63, 2)],
                                                    4)], 0),
    "3d_one_covered": lambda: ([_problem(3, 16, [(0, 15, 1), (0, 31, 2), (16, 47, 2)], 5)], 0),
    "3d_extension": lambda: ([_problem(3, 32, [(0, 31, 2), (16, 47, 2)], 6),
                              _problem(3, 16, [(0, 15, 1), (8, 23, 1)], 7)], 2),
    "3d_extension_of_covered": lambda: ([_problem(3, 16, [(0, 15, 1), (0, 31, 2),
                                                          (24, 55, 2)], 8)], 1),
}

# (staged passes, one-pass residual)
PATHS = [(True, -1), (False, True), (False, False)]
PRM = dict(coarse_tol=1e-300, coarse_max_it=12, max_cycles=5, relative_residual_tol=1e-300)


def _context(probs, ext, path, **kw):
    g = fac.FacContext(probs, params=PRM, bc=ROBIN, coarse_extension=ext, **kw)
    g.set_staged(path[0])
    g.set_fused_residual(path[1])
    return g


def _composite_residual(g):
    """computeFullCompositeResidual over whole levels, finer u restricted first."""
    top = g.nlev - 1
    for ln in range(top - 1, -1, -1):
        g.restrict_solution(U, ln)
    g.comp_residual(R, U, F, top, False)
    for ln in range(top - 1, -1, -1):
        g.restrict_solution(U, ln)
        g.comp_residual(R, U, F, ln, False)
        g.restrict(R, R, ln)
    return g.rms_norm(R)


def _state(g):
    return {(fid, i, ln): g.download(fid, i, ln) for fid in (U, R) for i in range(g.nprob)
            for ln in range(g.nlev)}


def _assert_same(a, b):
    for key, x in a.items():
        assert np.array_equal(x, b[key]), key


@pytest.mark.parametrize("path", PATHS, ids=["staged", "one_pass", "flux_arrays"])
@pytest.mark.parametrize("name", HIERARCHIES)
def test_solve_equals_whole_level_operators(name, path, require_gpu):
    probs, ext = HIERARCHIES[name]()
    g, ref = (_context(probs, ext, path) for _ in range(2))
    g.solve()
    if ext:
        assert fac.load_library().fac_extend_coefficients(ref.h) == 0
    norms = [_composite_residual(ref)]
    for _ in range(PRM["max_cycles"]):
        ref.zero(E)
        ref.fac_cycle()
        ref.vec_linear_sum(U, 1.0, U, 1.0, E)
        norms.append(_composite_residual(ref))
    for i in range(g.nprob):
        assert np.array_equal(g.residual_history(i), [n[i] for n in norms])
    _assert_same(_state(g), _state(ref))
    g.close()
    ref.close()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("krylov", [0, 3])
@pytest.mark.parametrize("name", HIERARCHIES)
def test_levels_after_a_solve_are_restrictions(name, krylov, precision, require_gpu):
    """FGMRES (restarted within the solve) and the mixed precision too: every
    level as the composite residual over whole levels leaves it, also in a
    second solve that starts from the first one's fields."""
    probs, ext = HIERARCHIES[name]()
    g = _context(probs, ext, (True, -1), precision=precision)
    g.set_krylov(krylov)
    for _ in range(2):
        g.solve()
        after = _state(g)
        _composite_residual(g)
        _assert_same(after, _state(g))
        assert all(np.isfinite(x).all() for x in after.values())
    g.close()


@pytest.mark.parametrize("krylov", [0, 4])
@pytest.mark.parametrize("level", [1, 2, 3])
def test_learned_level_below_at_and_above_the_first(level, krylov, require_gpu):
    """The learned correction on a covered level, on the first uncovered one
    and on a finer one: R is the composite residual of U, and u on the covered
    levels its restriction, to the rounding of the correction's own updates."""
    probs = [_problem(3, 32, [(0, 31, 2), (16, 47, 2)], 6)]
    g = _context(probs, 2, (True, -1))
    net = fac.CNN(max_batch=64, seed=5)
    g.set_learned(net, level)
    g.set_krylov(krylov)
    g.solve()
    after = _state(g)
    _composite_residual(g)
    scale = {fid: max(np.abs(x).max() for (f, *_), x in after.items() if f == fid) for fid in (U, R)}
    for key, x in _state(g).items():
        assert np.abs(x - after[key]).max() <= 1e-11 * max(scale[key[0]], 1.0), key
    g.close()
    net.close()
