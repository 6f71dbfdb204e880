"""A served request's scores do not depend on the requests it is merged with:
bit for bit those of the request alone.  Image 64, where a small batch of its
own would split its long k-loops; 1 to 40 particles (below five, a batch's norms
have a kernel of their own), on the texture and on the linear projector."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("interp", ["TEXTURE", "LINEAR"])
@pytest.mark.parametrize("precision", ["TF32", "BF16X3"])
def test_merged_equals_alone(pkg, synth, cuda, precision, interp):
    rng = np.random.default_rng(5)
    prob = synth.make_problem("c2", P=40)
    proj = pkg.Projector(prob.projector, use_texture=2)
    view = proj.view(prob.imgX, prob.imgY, prob.imgMaxR, interp=getattr(pkg, "INTERP_" + interp))
    srv = pkg.Server(slots=1, hbm_budget=8 << 30, precision=getattr(pkg, "PREC_" + precision))
    ref = srv.add_reference(view, prob.eulers, prob.N_img)
    reqs = []
    for P, O, rad in [(1, 300, 3), (4, 90, 2), (3, 800, 4), (9, 257, 3), (20, 500, 2), (2, 4608, 1), (40, 130, 3)]:
        ps = np.sort(rng.choice(prob.P, P, replace=False))
        orient = np.sort(rng.choice(prob.O, O, replace=False)).astype(np.int32)
        sh = synth.translation_grid(rad * rad)
        t = np.ascontiguousarray((-2 * np.pi * sh / prob.projector.ori_size).astype(np.float32).T)
        reqs.append((tuple(np.ascontiguousarray(a[ps]) for a in (prob.fimg_re, prob.fimg_im, prob.corr)), orient, t))

    def submit(imgs, orient, t):
        out = np.zeros((len(imgs[0]), orient.size, t.shape[1]), np.float32)
        mn, am = np.zeros(len(imgs[0])), np.zeros(len(imgs[0]), np.int64)
        return srv.submit(ref, *imgs, orient, t[0].copy(), t[1].copy(), out, mn, am), out, mn, am

    # a long request holds the one slot, so that the others queue and merge
    full = np.arange(prob.O, dtype=np.int32)
    long_out = np.zeros((prob.P, prob.O, prob.T), np.float32)
    t_long = srv.submit(ref, prob.fimg_re, prob.fimg_im, prob.corr, full, prob.trans_x, prob.trans_y, long_out,
                        np.zeros(prob.P), np.zeros(prob.P, np.int64))
    merged = [submit(*r) for r in reqs]
    assert all(srv.wait(t)[0] == 0 for t in (t_long, *(m[0] for m in merged)))
    assert srv.stats()["merged_requests"] >= 2
    srv.set_merging(1)
    for r, (_, out, mn, am) in zip(reqs, merged):
        t, out1, mn1, am1 = submit(*r)
        assert srv.wait(t)[0] == 0
        np.testing.assert_array_equal(out, out1)
        np.testing.assert_array_equal(mn, mn1)
        np.testing.assert_array_equal(am, am1)
    srv.close()
    proj.close()
