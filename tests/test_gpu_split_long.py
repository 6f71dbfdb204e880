"""Contractions split over k at sizes where every requested split is launched and
every CTA of its cluster wraps its ring: 81 to 230 k-blocks of 64 bytes at image
64.  Each split (also the odd ones, and 8), both tile widths and row widths, the
operands generated in the contraction, and plans that take an explicit split.

A split adds FP32 partial sums in FP64 and rounds once: 1e-5 relative for BF16x3
and 1e-3 for TF32 against the FP64 kernel, as unsplit."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = {"BF16X3": 1e-5, "TF32": 1e-3}
ELEM = {"BF16X3": 2, "TF32": 4}


@pytest.fixture(scope="module")
def setup(pkg, synth, cuda):
    torch = cuda
    pr = synth.make_problem("c2", P=3)
    proj = pkg.Projector(pr.projector, use_texture=1)
    view = proj.view(pr.imgX, pr.imgY, pr.imgMaxR)
    O, T = 300, 37
    dev = lambda a: torch.as_tensor(np.ascontiguousarray(a, np.float32), device="cuda")  # noqa: E731
    eul = dev(pr.eulers.reshape(-1, 9)[:O].reshape(-1))
    tx, ty = dev(pr.trans_x[:T]), dev(pr.trans_y[:T])
    re, im, corr = dev(pr.fimg_re), dev(pr.fimg_im), dev(pr.corr)
    ref = []
    for p in range(pr.P):
        r = torch.zeros(O * T, device="cuda", dtype=torch.float64)
        pkg.run_diff2_kernel_coarse_double(view, tx, ty, corr[p], re[p], im[p], eul, r, O, T, pr.N_img)
        ref.append(r)
    x, y = (np.arange(pr.N_img) % pr.imgX, np.arange(pr.N_img) // pr.imgX)
    y = np.where(y > pr.imgMaxR, y - pr.imgY, y)
    listed = int((x * x + y * y <= pr.imgMaxR ** 2).sum())
    yield pr, view, O, T, eul, tx, ty, re, im, corr, torch.stack(ref).reshape(pr.P, O, T), listed
    proj.close()


def _check(out, ref, prec):
    assert ((out.double() - ref).abs() / ref).max().item() <= TOL[prec]


@pytest.mark.parametrize("gen", [0, 1])
@pytest.mark.parametrize("rb,tn", [(64, 256), (64, 128), (128, 256), (128, 128)])
@pytest.mark.parametrize("split", [2, 3, 5, 7, 8])
@pytest.mark.parametrize("prec", ["BF16X3", "TF32"])
def test_batch(pkg, cuda, setup, prec, split, rb, tn, gen):
    torch = cuda
    pr, view, O, T, eul, tx, ty, re, im, corr, ref, listed = setup
    assert listed * 2 * ELEM[prec] // rb >= 4 * split  # no clamp: every CTA has k-blocks to wrap its ring with
    out = torch.full((pr.P, O, T), float("nan"), device="cuda")
    b = pkg.make_batch(eul, tx, ty, re, im, corr, out, O=O, T=T, P=pr.P, N_img=pr.N_img)
    code = getattr(pkg, "PREC_" + prec)
    pkg.set_operand_gen(gen)
    pkg.set_gemm_variant(rb, tn, split, 2)
    try:
        ws = torch.empty(pkg.batch_workspace_bytes(view, b, code), device="cuda", dtype=torch.uint8)
        pkg.diff2_coarse_batch(view, b, code, ws)
        torch.cuda.synchronize()
    finally:
        pkg.set_gemm_variant(0, 0, 0, 0)
        pkg.set_operand_gen(0)
    assert pkg.workspace_status(ws) == 0
    _check(out, ref, prec)


@pytest.mark.parametrize("split", [3, 8])
@pytest.mark.parametrize("tn", [128, 256])
def test_plan(pkg, cuda, setup, split, tn):
    """Uneven particles in a plan that is not autotuned and so takes the set split."""
    torch = cuda
    pr, view, O, T, _, _, _, re, im, corr, ref, _ = setup
    rng = np.random.default_rng(split)
    subsets = [np.sort(rng.choice(O, n, replace=False)).astype(np.int32) for n in (40, 300, 129)]
    Ts = (5, 37, 20)
    outs = [torch.full((o.size, t), float("nan"), device="cuda") for o, t in zip(subsets, Ts)]
    parts = [dict(real=re[p], imag=im[p], corr=corr[p], diff2=outs[p], orient=subsets[p],
                  trans_x=pr.trans_x[:Ts[p]].copy(), trans_y=pr.trans_y[:Ts[p]].copy()) for p in range(3)]
    d_eul = torch.as_tensor(np.ascontiguousarray(pr.eulers.reshape(-1, 9)[:O].reshape(-1)), device="cuda")
    pkg.set_gemm_variant(128, tn, split, 2)
    try:
        plan = pkg.Plan(view, d_eul, O, pr.N_img, parts, precision=pkg.PREC_BF16X3, flags=0)
        assert plan.info()["split"] == split
        plan.run()
        torch.cuda.synchronize()
    finally:
        pkg.set_gemm_variant(0, 0, 0, 0)
    for p in range(3):
        o = torch.as_tensor(subsets[p], device="cuda").long()
        _check(outs[p], ref[p][o][:, :Ts[p]], "BF16X3")
    plan.close()


def test_set_split_does_not_reach_full_grids(pkg, cuda, setup):
    """A set split is for grids that leave SMs idle: where the tiles fill the GPU
    none is taken (a plan says so), and the CTA pairs that were asked for run."""
    torch = cuda
    pr, view, _, _, _, tx, ty, re, im, corr, _, _ = setup
    O, T, P = 4608, 113, 30
    eul = torch.as_tensor(np.ascontiguousarray(pr.eulers.reshape(-1, 9)[:O].reshape(-1)), device="cuda")
    which = [p % pr.P for p in range(P)]
    out = torch.empty((P, O, T), device="cuda")
    parts = [dict(real=re[w], imag=im[w], corr=corr[w], diff2=out[p], orient=None, O=O, trans_x=pr.trans_x[:T].copy(),
                  trans_y=pr.trans_y[:T].copy()) for p, w in enumerate(which)]
    pkg.set_gemm_variant(128, 256, 4, 1)
    try:
        plan = pkg.Plan(view, eul, O, pr.N_img, parts, precision=pkg.PREC_BF16X3, flags=0)
        info = plan.info()
    finally:
        pkg.set_gemm_variant(0, 0, 0, 0)
    assert (info["split"], info["pair"]) == (1, 1)
    plan.run()
    r = torch.zeros(O * T, device="cuda", dtype=torch.float64)
    t = [torch.as_tensor(np.ascontiguousarray(a[:T]), device="cuda") for a in (pr.trans_x, pr.trans_y)]
    pkg.run_diff2_kernel_coarse_double(view, *t, corr[0], re[0], im[0], eul, r, O, T, pr.N_img)
    _check(out[0].reshape(-1), r, "BF16X3")
    plan.close()
