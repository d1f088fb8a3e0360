"""The regrid step on the device (fac_tag_gradient, fac_cluster_tags)
against the reference's own tagging and Berger-Rigoutsos clustering.

tests/golden/ref_br_<case>.npz hold the tags of the FAC_adaptive test's
AdaptivePoisson estimate and the boxes of mesh::BergerRigoutsos for the
cases of tests/br_cases.py (oracle/_ref/br_ref_driver).  The device tags
must equal them bit for bit and the boxes as a set; several problems in one
context are tagged and clustered each on its own and all at once
(fac_cluster_tags_all).
"""
import os

import numpy as np
import pytest

import br_cases
from samrai_b200 import fac
from oracle.oracle import U

pytestmark = pytest.mark.gpu

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden")


def _fixture(name):
    fx = np.load(os.path.join(GOLDEN, f"ref_{name}.npz"))
    tags = np.unpackbits(fx["tags_packed"])[:int(fx["ntags"][0])]
    return fx, tags


@pytest.mark.parametrize("name", list(br_cases.CASES))
def test_device_regrid_matches_reference(name, require_gpu):
    fx, want = _fixture(name)
    c = br_cases.CASES[name]
    p = br_cases.problem(name)
    g = fac.FacContext([p])
    g.upload(U, 0, 0, p.u0[0])
    cnt = g.tag_gradient(U, 0, c["threshold"])
    assert int(cnt[0]) == int(fx["tagged"][0])
    assert np.array_equal(g.download_tags(0, 0), want)
    boxes = g.cluster_tags(0, 0, br_cases.bound_boxes(name), c["min_box"], c["max_box"],
                           c["efficiency"], c["combine"])
    assert np.array_equal(br_cases.sorted_boxes(boxes), br_cases.sorted_boxes(fx["boxes"]))
    g.close()


def test_batched_problems_tag_and_cluster_each(require_gpu):
    names = ["br_3d", "br_3d_eff"]
    probs = [br_cases.problem(n) for n in names]
    g = fac.FacContext(probs)
    for i, p in enumerate(probs):
        g.upload(U, i, 0, p.u0[0])
    thr = br_cases.CASES[names[0]]["threshold"]
    cnt = g.tag_gradient(U, 0, thr)
    for i, n in enumerate(names):
        c = br_cases.CASES[n]
        fx, want = _fixture(n)
        if c["threshold"] == thr:
            assert int(cnt[i]) == int(fx["tagged"][0])
            assert np.array_equal(g.download_tags(i, 0), want)
    # per problem with its own threshold: retag and cluster
    for i, n in enumerate(names):
        c = br_cases.CASES[n]
        fx, want = _fixture(n)
        cnt = g.tag_gradient(U, 0, c["threshold"])
        assert int(cnt[i]) == int(fx["tagged"][0])
        boxes = g.cluster_tags(i, 0, br_cases.bound_boxes(n), c["min_box"], c["max_box"],
                               c["efficiency"], c["combine"])
        assert np.array_equal(br_cases.sorted_boxes(boxes), br_cases.sorted_boxes(fx["boxes"]))
    g.close()


def test_cluster_all_problems_at_once(require_gpu):
    """fac_cluster_tags_all over problems of different sizes and parameters
    sharing one threshold: the same boxes, in the same order, as
    fac_cluster_tags problem by problem, and the reference's boxes where the
    fixture's threshold is the one used."""
    names = ["br_3d", "br_3d_eff"]
    probs = [br_cases.problem(n) for n in names]
    g = fac.FacContext(probs)
    for i, p in enumerate(probs):
        g.upload(U, i, 0, p.u0[0])
    c0 = br_cases.CASES[names[0]]
    g.tag_gradient(U, 0, c0["threshold"])
    bounds = [br_cases.bound_boxes(n) for n in names]
    one = [g.cluster_tags(i, 0, bounds[i], c0["min_box"], c0["max_box"], c0["efficiency"],
                          c0["combine"]) for i in range(len(names))]
    allb = g.cluster_tags_all(0, bounds, c0["min_box"], c0["max_box"], c0["efficiency"],
                              c0["combine"])
    assert len(allb) == len(names)
    for a, b in zip(one, allb):
        assert np.array_equal(a, b)
    fx, _ = _fixture(names[0])
    assert np.array_equal(br_cases.sorted_boxes(allb[0]), br_cases.sorted_boxes(fx["boxes"]))
    g.close()


@pytest.mark.parametrize("n, bounds", [
    # rows of 1 to 1024 tags, bounds whose first cell lies on every byte of a word
    ((1024, 3), [[0, 0, 1023, 2]]),
    ((700, 9), [[1, 0, 350, 8], [351, 2, 698, 8]]),
    ((37, 2100), [[2, 0, 36, 2099]]),
    ((130, 8, 5), [[3, 1, 0, 127, 7, 4], [128, 0, 0, 129, 7, 4]]),
    ((5, 70, 40), [[0, 0, 0, 4, 69, 39]]),
])
def test_histograms_of_long_and_ragged_rows(n, bounds, require_gpu):
    """Node boxes at the edges of the histogram kernel's split (words of four
    tags, lanes per row, rows per block): the boxes of the CPU restatement."""
    from oracle import br_oracle
    from samrai_b200 import configs
    dim = len(n)
    m = tuple(n) + (1,) * (3 - dim)
    p = configs.Problem(dim=dim, n0=m, xlo=(0.0,) * 3, xup=(1.0,) * 3,
                        levels=[configs.Level((1, 1, 1), np.array([[0, 0, 0] + [x - 1 for x in m]],
                                                                  dtype=np.int32))])
    rng = np.random.default_rng(sum(m))
    shape = [x + 2 for x in m[:dim]][::-1]
    u = np.zeros(shape)
    for _ in range(12):  # spikes tag their neighbourhoods
        u[tuple(rng.integers(0, s) for s in shape)] = 1.0
    ctx = fac.FacContext([p])
    ctx.upload(U, 0, 0, u.reshape(-1))
    ctx.tag_gradient(U, 0, 0.4)
    tags = ctx.download_tags(0, 0).reshape(m[::-1])
    full = [b if dim == 3 else [b[0], b[1], 0, b[2], b[3], 0] for b in bounds]
    got = ctx.cluster_tags(0, 0, full, [2] * dim)
    cl = br_oracle.Clusterer(tags if dim == 3 else tags[0], [0, 0, 0], dim, [2] * dim, None, 0.8, 0.8)
    boxes = cl.cluster(full)
    pad = [0] * (3 - dim)
    want = np.array([list(lo) + pad + list(hi) + pad for lo, hi in boxes], dtype=np.int64)
    assert len(want) > 0
    assert np.array_equal(br_cases.sorted_boxes(got), br_cases.sorted_boxes(want))
    ctx.close()
