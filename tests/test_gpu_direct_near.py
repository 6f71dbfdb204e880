"""Images that almost equal a projection, on the CUDA cores.  FP32 diff2 scales
the projection and the image by sqrt(corr/2) and rounds before it subtracts;
where the score is small against the image's power the differences are taken
first, so that the smallest score keeps its relative accuracy.

The image is the library's own projection of one orientation, perturbed by a
relative 1e-5 or 1e-6, so that at zero shift every A - S is exact in FP32.  The
score is then a sum of K = 2000 or so positive terms of four roundings each, in
one sequence per cluster CTA: relative error at most (K + 4) 2^-24 = 1.2e-4 in
the worst case and sqrt(K) 2^-24 = 2.7e-6 for roundings without a sign; 1e-5
holds for the FP32 drop-in.  Scaling first would put 2^-23 sqrt(2) into every
term's difference: 2e-2 / sqrt(K) = 4e-4 at 1e-5 and ten times that at 1e-6."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P", [1, 40])  # clusters that share the pixels; CTAs on their own
@pytest.mark.parametrize("T", [1, 29, 113])
@pytest.mark.parametrize("delta", [1e-5, 1e-6])
def test_near_equal_image(pkg, synth, cuda, T, P, delta):
    torch = cuda
    pr = synth.make_problem("c2", P=1)
    proj = pkg.Projector(pr.projector, use_texture=1)
    view = proj.view(pr.imgX, pr.imgY, pr.imgMaxR)
    N, O = pr.N_img, 640
    eul = torch.as_tensor(np.ascontiguousarray(pr.eulers.reshape(-1, 9)[:O].reshape(-1)), device="cuda")
    i = torch.arange(N, device="cuda", dtype=torch.int32)
    x, y = i % view.imgX, i // view.imgX
    y = torch.where(y > view.maxR, y - view.imgY, y).int().contiguous()
    re, im = (torch.empty(O * N, device="cuda") for _ in range(2))
    pkg.project_pixels(view, eul, x.int().contiguous(), y, re, im, O, N)
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    best = 77
    a = torch.stack([re.reshape(O, N)[best], im.reshape(O, N)[best]])
    img = a * (1 + delta * torch.randn(2, N, generator=g, device="cuda"))
    co = torch.rand(N, generator=g, device="cuda") + 0.5
    tx, ty = (torch.as_tensor(v[:T].copy(), device="cuda") for v in (pr.trans_x, pr.trans_y))
    tx[0] = ty[0] = 0.0
    dr, di = (img - a).double()
    want = (co.double() / 2 * (dr * dr + di * di)).sum().item()
    power = (co.double() / 2 * (img.double() ** 2).sum(0)).sum().item()
    assert 0 < want < 1e-8 * power
    out = torch.empty((P, O, T), device="cuda")
    imgs = [v.expand(P, N).contiguous() for v in (img[0], img[1], co)]
    b = pkg.make_batch(eul, tx, ty, *imgs, out, O=O, T=T, P=P, N_img=N)
    pkg.diff2_coarse_batch(view, b, pkg.PREC_FP32)
    assert ((out[:, best, 0].double() - want).abs() / want).max().item() <= 1e-5
    f64 = torch.zeros(O * T, device="cuda", dtype=torch.float64)
    pkg.run_diff2_kernel_coarse_double(view, tx, ty, co, img[0].contiguous(), img[1].contiguous(), eul, f64, O, T, N)
    # the FP64 form subtracts first as well: (K + 8) 2^-53, 3e-13
    assert abs(f64.reshape(O, T)[best, 0].item() - want) <= 1e-12 * want
    proj.close()
