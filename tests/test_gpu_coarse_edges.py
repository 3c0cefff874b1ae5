"""The coarse pass where no size is a multiple of its tiles: 3 x 997 in-plane orientations x 29 shifts
(86,739 hypotheses a particle, so that from the second particle on no row is 16-byte aligned), at
particle counts on each side of the plain FP32 kernels' tile choices.

The oracle (FP64) gives the coarse diff2 (1e-5 relative, as everywhere) and, from the product's own
diff2, the sum of the weights, the threshold and the number of significant hypotheses: FP64 sums in
another order, 1e-10, and the threshold itself 1e-12."""
import numpy as np
import pytest

import problems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,mode", [(1, 0), (8, 0), (9, 0), (33, 0), (65, 0), (1, 1), (9, 1)])
def test_coarse_pass_at_ragged_sizes(n, mode):
    pb = problems.build("class2d_odd", n_particles=n, seed=11, nr_classes=3, diff2_mode=mode)
    es, prob, op, P = pb["product"](), pb["prob"], pb["oparts"], pb["parts"]
    assert prob.O == 997 and prob.T == 29
    res = es.expectation(P["fimg"], P["ctf"], P["minv"], P["scalars"])
    assert np.all(res["status"] == 0)
    for b in {0, n // 2, n - 1}:
        ref, _ = prob.coarse_diff2(op, b)
        d2 = es.coarse_diff2(b).astype(np.float64)
        ref = np.asarray(ref).reshape(d2.shape)
        ok = ref >= 0
        assert np.array_equal(ok, d2 >= 0)
        assert np.max(np.abs(d2[ok] - ref[ok]) / ref[ok]) <= 1e-5
        rc, w, sw, sig, ns = prob.weights(op, b, 0, d2.reshape(-1), np.arange(d2.size), d2[ok].min())
        assert rc == 0
        assert res["coarse_sum_weight"][b] == pytest.approx(sw, rel=1e-10)
        assert res["coarse_sig_weight"][b] == pytest.approx(sig, rel=1e-12)
        assert res["nr_sign"][b] == ns
        assert res["n_coarse_sig"][b] == int(np.sum(w >= sig))
    es.close()
