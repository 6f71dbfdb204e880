"""FP32 batches on the CUDA cores, diff2 and CC, over the translation counts at
which the tile's shape changes and over enough particles to take the 256-thread
tiles as well as the clusters, on both projectors.

Reference: the FP64 form of the same score, one particle at a time; 1e-5
relative for diff2 as documented for the FP32 drop-in, and for CC, which changes
sign, relative to the particle's largest score."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def setup(pkg, synth, cuda):
    import importlib
    healpix = importlib.import_module("relion_b200.healpix")
    pr = synth.make_problem("tiny", P=4)
    proj = pkg.Projector(pr.projector, use_texture=2)
    eul, _ = healpix.orientation_grid(2, 24)
    yield pr, proj, np.ascontiguousarray(eul)
    proj.close()


@pytest.mark.parametrize("interp", ["TEXTURE", "LINEAR"])
@pytest.mark.parametrize("score", ["DIFF2", "CC"])
@pytest.mark.parametrize("P,O", [(1, 129), (3, 300), (30, 385), (75, 65)])
@pytest.mark.parametrize("T", [1, 16, 17, 32, 33, 49, 113])
def test_fp32_batch(pkg, cuda, setup, T, P, O, score, interp):
    torch = cuda
    pr, proj, eul = setup
    view = proj.view(pr.imgX, pr.imgY, pr.imgMaxR, interp=getattr(pkg, "INTERP_" + interp))
    rng = np.random.default_rng(T * 1009 + P)
    dev = lambda a: torch.as_tensor(np.ascontiguousarray(a, np.float32), device="cuda")  # noqa: E731
    N = pr.N_img
    tx, ty = dev(rng.uniform(-0.6, 0.6, T)), dev(rng.uniform(-0.6, 0.6, T))
    e = dev(eul[rng.integers(0, len(eul), O)].reshape(-1))
    which = rng.integers(0, pr.P, P)
    re, im, co = dev(pr.fimg_re[which]), dev(pr.fimg_im[which]), dev(pr.corr[which] * rng.uniform(0.5, 2, (P, 1)))
    out = torch.full((P, O, T), float("nan"), device="cuda")
    b = pkg.make_batch(e, tx, ty, re, im, co, out, O=O, T=T, P=P, N_img=N, score=getattr(pkg, "SCORE_" + score))
    pkg.diff2_coarse_batch(view, b, pkg.PREC_FP32)
    f64 = pkg.run_diff2_kernel_coarse_double if score == "DIFF2" else pkg.run_diff2_kernel_coarse_cc_double
    for p in sorted({0, P // 2, P - 1}):
        ref = torch.zeros(O * T, device="cuda", dtype=torch.float64)
        f64(view, tx, ty, co[p], re[p], im[p], e, ref, O, T, N)
        scale = ref.abs() if score == "DIFF2" else ref.abs().max()
        assert ((out[p].reshape(-1).double() - ref).abs() / scale).max().item() <= 1e-5, p
