"""Give-up paths: when a bounded device-side wait runs out, nothing that depends
on it is stored.  The limit is cut by the test hook; the kernels drain what
they have in flight and return, the status reads B200D2_ERR_TIMEOUT, and the
next call with the default limit is correct in the same workspace.

Scores that were written all the same must be the right ones: 1e-5 relative
against the FP64 kernel, plus 6e-8 for the addition onto the initial value."""
from __future__ import annotations

import numpy as np
import pytest

from gpu_util import DeviceProblem

pytestmark = pytest.mark.gpu
TIMEOUT = 5  # B200D2_ERR_TIMEOUT


@pytest.fixture(scope="module")
def c2(pkg, synth, cuda):
    pr = synth.make_problem("c2", P=2)
    proj = pkg.Projector(pr.projector, use_texture=2)
    # the linear projector's norms have a kernel without waits
    view = proj.view(pr.imgX, pr.imgY, pr.imgMaxR, interp=pkg.INTERP_LINEAR)
    dp = DeviceProblem(cuda, pr)
    ref = []
    for p in range(pr.P):
        d = cuda.zeros(pr.O * pr.T, device="cuda", dtype=cuda.float64)
        pkg.run_diff2_kernel_coarse_double(view, dp.tx, dp.ty, dp.corr[p], dp.re[p], dp.im[p], dp.eulers, d, pr.O,
                                           pr.T, pr.N_img)
        ref.append(d)
    yield pr, proj, view, dp, cuda.stack(ref).reshape(pr.P, pr.O, pr.T)
    proj.close()


@pytest.mark.parametrize("split", [2, 3, 8])
def test_split_tile_that_gave_up_is_not_written(pkg, cuda, c2, split):
    """A 1 us limit runs out in the epilogue's wait for the accumulator (tens of
    k-blocks per CTA of the cluster): added scores stay as they were."""
    torch = cuda
    pr, _, view, dp, ref = c2
    init = (2.0 ** torch.floor(torch.log2(ref))).float()  # of the score's size: the sum rounds once more
    out = init.clone()
    b = pkg.make_batch(dp.eulers, dp.tx, dp.ty, dp.re, dp.im, dp.corr, out, O=pr.O, T=pr.T, P=pr.P, N_img=pr.N_img,
                       accumulate=True)
    ws = torch.empty(pkg.batch_workspace_bytes(view, b, pkg.PREC_BF16X3), device="cuda", dtype=torch.uint8)
    pkg.set_gemm_variant(128, 128, split, 2)
    try:
        pkg.set_wait_limit_ns(1000)
        try:
            pkg.diff2_coarse_batch(view, b, pkg.PREC_BF16X3, ws)
            torch.cuda.synchronize()
        finally:
            pkg.set_wait_limit_ns(0)
        assert pkg.workspace_status(ws) == TIMEOUT
        untouched = out == init
        want = ref + init.double()
        good = (out.double() - want).abs() <= (1e-5 + 6e-8) * want
        assert bool((untouched | good).all()) and bool(untouched.any())
        out.copy_(init)
        pkg.diff2_coarse_batch(view, b, pkg.PREC_BF16X3, ws)
        torch.cuda.synchronize()
        assert pkg.workspace_status(ws) == 0
        assert ((out.double() - want).abs() / want).max().item() <= 1e-5 + 6e-8
    finally:
        pkg.set_gemm_variant(0, 0, 0, 0)


@pytest.mark.parametrize("pair", [1, 2])  # CTA pairs and single CTAs: neither may score what is missing
def test_projection_that_gave_up_is_not_scored(pkg, cuda, c2, pair):
    """The projection kernel that takes the norms along (texture) waits for its
    ring for microseconds: with a 1 us limit no score is written or added."""
    torch = cuda
    pr, proj, _, dp, _ = c2
    view = proj.view(pr.imgX, pr.imgY, pr.imgMaxR)
    init = torch.rand(pr.P, pr.O, pr.T, device="cuda") + 1.0
    out = init.clone()
    b = pkg.make_batch(dp.eulers, dp.tx, dp.ty, dp.re, dp.im, dp.corr, out, O=pr.O, T=pr.T, P=pr.P, N_img=pr.N_img,
                       accumulate=True)
    ws = torch.empty(pkg.batch_workspace_bytes(view, b, pkg.PREC_BF16X3), device="cuda", dtype=torch.uint8)
    pkg.set_gemm_variant(0, 256, 1, pair)
    try:
        pkg.diff2_coarse_batch(view, b, pkg.PREC_BF16X3, ws)
        torch.cuda.synchronize()
        assert pkg.workspace_status(ws) == 0
        scores = out.clone()
        pkg.set_wait_limit_ns(1000)
        out.copy_(init)
        try:
            pkg.diff2_coarse_batch(view, b, pkg.PREC_BF16X3, ws)
            torch.cuda.synchronize()
        finally:
            pkg.set_wait_limit_ns(0)
        assert pkg.workspace_status(ws) == TIMEOUT
        assert torch.equal(out, init)
        pkg.diff2_coarse_batch(view, b, pkg.PREC_BF16X3, ws)
        torch.cuda.synchronize()
        assert pkg.workspace_status(ws) == 0 and torch.equal(out, scores)
    finally:
        pkg.set_gemm_variant(0, 0, 0, 0)
