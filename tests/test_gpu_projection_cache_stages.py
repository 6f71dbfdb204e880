"""The one-particle call on the tensor cores takes its norms from the same kernels
whether the projection cache is on or off, so that every sum is the same: with
the cache on it launches the check of the Euler matrices besides, nothing else,
and the scores are equal bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["BF16X3", "TF32"])
def test_same_stages(pkg, synth, cuda, prec):
    torch = cuda
    pr = synth.make_problem("c2", P=2)  # 4608 orientations x 1600 pixels: above the 2^20 samples that are kept
    proj = pkg.Projector(pr.projector, use_texture=1)
    view = proj.view(pr.imgX, pr.imgY, pr.imgMaxR)
    dev = lambda a: torch.as_tensor(np.ascontiguousarray(a, np.float32), device="cuda")  # noqa: E731
    eul, tx, ty = dev(pr.eulers.reshape(-1)), dev(pr.trans_x), dev(pr.trans_y)
    re, im, co = dev(pr.fimg_re), dev(pr.fimg_im), dev(pr.corr)

    def call(p):
        out = torch.zeros(pr.O * pr.T, device="cuda")
        n0 = pkg.launch_count()
        pkg.run_diff2_kernel_coarse(view, tx, ty, co[p], re[p], im[p], eul, out, pr.O, pr.T, pr.N_img,
                                    precision=getattr(pkg, "PREC_" + prec))
        torch.cuda.synchronize()
        return pkg.launch_count() - n0, out

    try:
        pkg.set_projection_cache(1)
        on = [call(p) for p in (0, 1, 1)]  # projected, kept, and kept again
        pkg.set_projection_cache(0)
        off = [call(p) for p in (0, 1, 1)]
    finally:
        pkg.set_projection_cache(1)
    for (n1, a), (n0, b) in zip(on, off):
        assert n1 == n0 + 1
        assert torch.equal(a, b)
    proj.close()
