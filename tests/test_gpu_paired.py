"""Paired orientations of the split-BF16 contraction (in-plane angles half a turn apart share an operand
row) against the general path, which takes every orientation by itself: the same problem with the
matrices of one half moved by 1e-10, far below what the projections resolve and enough that they are no
longer each other's exact half turn.  Both against the FP64 oracle at the coarse pass's 1e-5, for
resident and chunked operands (chunks of no whole tile), at batches on each side of a column tile;
and a model whose x = 0 plane is not Hermitian, which has to take the general path."""
import numpy as np
import pytest

import problems

pytestmark = pytest.mark.gpu


def coarse(pb, chunk, which):
    es = pb["product"](orientation_chunk=chunk)
    P = pb["parts"]
    res = es.expectation(P["fimg"], P["ctf"], P["minv"], P["scalars"])
    d2 = [es.coarse_diff2(b).astype(np.float64).reshape(-1) for b in which]
    es.close()
    return res, d2


@pytest.mark.parametrize("name,classes,chunk,n", [("refine_o1_ovs", 1, 0, 1), ("refine_o1_ovs", 1, 0, 9),
                                                  ("refine_o1_ovs", 2, 0, 10), ("refine_o1_ovs", 2, 700, 9),
                                                  ("class2d", 3, 0, 20), ("refine_o2", 1, 0, 3)])
def test_paired_contraction_matches_the_general_one(name, classes, chunk, n):
    pb = problems.build(name, n_particles=n, seed=31, nr_classes=classes, diff2_mode=1)
    which = sorted({0, n // 2, n - 1})
    paired, dp = coarse(pb, chunk, which)
    E = np.asarray(pb["samp"]["eul_coarse"]).reshape(-1, 9)
    npsi = E.shape[0] // pb["samp"]["n_dir"]
    assert npsi % 2 == 0
    late = np.arange(E.shape[0]) % npsi >= npsi // 2
    assert np.max(np.abs(E[late, :6] + E[~late, :6])) < 1e-13
    E[late, :6] += 1e-10
    pb["samp"]["eul_coarse"] = E.reshape(np.asarray(pb["samp"]["eul_coarse"]).shape)
    general, dg = coarse(pb, chunk, which)
    for b, p, g in zip(which, dp, dg):
        ref = np.asarray(pb["prob"].coarse_diff2(pb["oparts"], b)[0]).reshape(-1)
        ok = ref >= 0
        assert np.array_equal(ok, p >= 0) and np.array_equal(ok, g >= 0)
        for d in (p, g):
            assert np.max(np.abs(d[ok] - ref[ok]) / ref[ok]) <= 1e-5
    assert np.all(paired["status"] == 0) and np.array_equal(paired["pose"], general["pose"])


def test_model_of_no_real_map():
    pb = problems.build("refine_o1_ovs", n_particles=3, seed=5, diff2_mode=1)
    m = pb["maps"][0]
    rng = np.random.default_rng(3)
    amp = np.abs(m).max()
    m[..., 0] += (1e-2 * amp * (rng.standard_normal(m.shape[:-1]) + 1j * rng.standard_normal(m.shape[:-1]))).astype(m.dtype)
    prob = pb["oracle_problem"]()
    _, d2 = coarse(pb, 0, [0, 2])
    for b, d in zip([0, 2], d2):
        ref = np.asarray(prob.coarse_diff2(pb["oparts"], b)[0]).reshape(-1)
        assert np.max(np.abs(d - ref) / ref) <= 1e-5
