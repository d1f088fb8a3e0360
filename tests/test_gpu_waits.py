"""Bounded device waits.

Every wait of the staged colour pass (a unit's copies landing in shared
memory, a stage coming free) and of the coarsest solve (another block's values)
gives up after a bound and sets the context's device error flag instead of
hanging the GPU; the next norm or dot product reports FAC_ERR_CUDA and the
context stays usable.  Here they are made to wait on an mbarrier nothing arrives on, with a
1e6-cycle bound: the call must end with the error, and after the flag is
cleared the same context must smooth exactly as before.
"""
import numpy as np
import pytest

from samrai_b200 import configs, fac
from oracle.oracle import E, Oracle, R

pytestmark = pytest.mark.gpu

FAC_ERR_CUDA = 3
FAC_ERR_DEVICE = 6


def test_bounded_wait_runs_out_and_context_recovers(require_gpu):
    p = configs.small_3d(seed=7)
    prm = dict(coarse_tol=1e-10, max_cycles=2)
    g = fac.FacContext([p], params=prm)
    o = Oracle(p, params=prm)
    ln = p.nlev - 1
    rng = np.random.default_rng(11)
    vals = {fid: rng.standard_normal(o.size(fid, ln)) for fid in (E, R)}
    for l2 in range(p.nlev):
        for fid in (E, R):
            v = vals[fid] if l2 == ln else np.zeros(o.size(fid, l2))
            g.upload(fid, 0, l2, v)
            o.set(fid, l2, v)
    L = fac.load_library()
    assert L.fac_set_wait_test(g.h, 1_000_000, 1) == 0
    g.smooth(E, R, ln, 1)
    with pytest.raises(fac.FacError) as err:
        g.rms_norm(R)
    assert err.value.code == FAC_ERR_CUDA
    # back to the default bound: the context works and matches the oracle
    assert L.fac_set_wait_test(g.h, 4_000_000_000, 0) == 0
    assert L.fac_clear_device_error(g.h) == 0
    for fid in (E, R):
        g.upload(fid, 0, ln, vals[fid])
    g.smooth(E, R, ln, 2)
    o.smooth(E, R, ln, 2)
    assert np.array_equal(g.download(E, 0, ln), o.get(E, ln))
    g.rms_norm(R)
    g.close()


@pytest.mark.parametrize("nprob", [1, 2])
@pytest.mark.parametrize("nx", [64, 97])
def test_coarsest_solve_wait_runs_out(nprob, nx, require_gpu):
    """One launch of several blocks per problem.  In problem 0 a single thread
    (not the one that arms the mbarriers) gives up, in problem 1 every thread:
    the flag is set, all blocks stop together long before the last sweep, and
    the context then solves like one that never failed."""
    def problem():
        return configs.Problem(dim=2, n0=(nx, nx, 1), xlo=(0.0,) * 3, xup=(1.0,) * 3,
                               levels=[configs.Level((1, 1, 1), np.array(
                                   [[0, 0, 0, nx - 1, nx - 1, 0]], dtype=np.int32))])

    rng = np.random.default_rng(nx)
    data = [{fid: rng.standard_normal(configs.field_size(problem(), 0, 1 if fid == E else 0))
             for fid in (E, R)} for _ in range(nprob)]

    def fresh():
        ctx = fac.FacContext([problem() for _ in range(nprob)])
        load(ctx)
        return ctx

    def load(ctx):
        for i, d in enumerate(data):
            for fid in (E, R):
                ctx.upload(fid, i, 0, d[fid])

    sweeps = 200
    a, b = fresh(), fresh()
    n0 = fac.kernel_launches()
    want = b.smooth(E, R, 0, sweeps, 1e-300)
    assert fac.kernel_launches() - n0 < sweeps  # all sweeps in one launch
    assert np.all(want == sweeps)
    L = fac.load_library()
    for _ in range(2):
        assert L.fac_set_wait_test(a.h, 1_000_000, 1) == 0
        # the first wait runs out in sweep 0, whose outcome stops sweep 1
        assert np.all(a.smooth(E, R, 0, sweeps, 1e-300) == 1)
        with pytest.raises(fac.FacError) as err:
            a.rms_norm(R)
        assert err.value.code == FAC_ERR_CUDA
        assert L.fac_set_wait_test(a.h, 4_000_000_000, 0) == 0
        assert L.fac_clear_device_error(a.h) == 0
        load(a)
        assert np.array_equal(a.smooth(E, R, 0, sweeps, 1e-300), want)
        a.rms_norm(R)
        for i in range(nprob):
            assert np.array_equal(a.download(E, i, 0), b.download(E, i, 0))
    a.close()
    b.close()


@pytest.mark.parametrize("coarsest", [False, True])
def test_composite_reductions_report_the_flag(coarsest, require_gpu):
    """Every reduction over a field reports it, not the RMS norm alone."""
    g = fac.FacContext([configs.config1() if coarsest else configs.small_3d(seed=7)])
    L = fac.load_library()
    assert L.fac_set_wait_test(g.h, 1_000_000, 1) == 0
    if coarsest:
        g.upload(R, 0, 0, np.ones(g.size(R, 0, 0)))
        g.solve_coarsest()
    else:
        g.smooth(E, R, g.nlev - 1, 1)
    for norm in (lambda: g.vec_l2_norm(R), lambda: g.vec_max_norm(R), lambda: g.vec_dot(R, E),
                 lambda: g.rms_norm(R)):
        with pytest.raises(fac.FacError) as err:
            norm()
        assert err.value.code == FAC_ERR_CUDA
    assert L.fac_set_wait_test(g.h, 4_000_000_000, 0) == 0
    assert L.fac_clear_device_error(g.h) == 0
    g.vec_l2_norm(R)
    g.vec_max_norm(R)
    g.vec_dot(R, E)
    g.close()


@pytest.mark.parametrize("n", [1, 60])
def test_convolution_wait_runs_out(n, require_gpu):
    """Batches of one slab a block and of several: the call reports the wait,
    the blocks leave once their multiplications are done, and the network then
    gives the bits of before."""
    import torch
    S = fac.CNN_BOX
    net = fac.CNN(max_batch=n, seed=2)
    x = torch.randn((n, S, S, S), generator=torch.Generator().manual_seed(n)).cuda()
    want, y = torch.zeros_like(x), torch.zeros_like(x)
    net.forward(x.data_ptr(), n, want.data_ptr())
    L = fac.load_library()
    for _ in range(2):
        assert L.fac_cnn_set_wait_test(net.h, 1_000_000, 1) == 0
        with pytest.raises(fac.FacError) as err:
            net.forward(x.data_ptr(), n, y.data_ptr())
        assert err.value.code == FAC_ERR_DEVICE
        assert L.fac_cnn_set_wait_test(net.h, 4_000_000_000, 0) == 0
        net.forward(x.data_ptr(), n, y.data_ptr())
        assert torch.equal(y, want)
    net.close()
