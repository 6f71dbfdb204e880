"""Batches around the sizes at which the projection kernel takes the norms along
and at which its tiles change: one wave of 8-, 16- and 32-orientation CTAs (148
SMs), orientations padded past a wave, and few particles.  Every batch agrees
with the FP64 kernel to the BF16x3 bound of 1e-5, and needs one launch less
where projection and norms are one kernel."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def setup(pkg, synth, cuda):
    import importlib
    healpix = importlib.import_module("relion_b200.healpix")
    pr = synth.make_problem("tiny", P=8)
    proj = pkg.Projector(pr.projector, use_texture=1)
    eul, _ = healpix.orientation_grid(3, 12)
    yield pr, proj, np.ascontiguousarray(eul)
    proj.close()


@pytest.mark.parametrize("P,O,fused", [(5, 1184, True), (5, 1185, True), (8, 1152, True), (64, 1300, True), (20, 2368, True),
                                       (20, 2369, True), (66, 1000, False), (66, 1200, True), (1, 1600, False),
                                       (4, 2369, False), (1, 2360, True), (4, 3200, True), (1, 3200, False), (2, 4608, True)])
def test_batch(pkg, cuda, setup, P, O, fused):
    torch = cuda
    pr, proj, eul = setup
    view = proj.view(pr.imgX, pr.imgY, pr.imgMaxR)
    rng = np.random.default_rng(P + O)
    N, T = pr.N_img, 3
    dev = lambda a: torch.as_tensor(np.ascontiguousarray(a, np.float32), device="cuda")  # noqa: E731
    which = rng.integers(pr.P, size=P)
    re, im, corr = dev(pr.fimg_re[which]), dev(pr.fimg_im[which]), dev(pr.corr[which] * rng.uniform(0.5, 2, (P, 1)))
    d_eul = dev(eul[:O].reshape(-1))
    tx, ty = dev(pr.trans_x[:T]), dev(pr.trans_y[:T])
    out = torch.full((P, O, T), float("nan"), device="cuda")
    b = pkg.make_batch(d_eul, tx, ty, re, im, corr, out, O=O, T=T, P=P, N_img=N)
    ws = torch.empty(pkg.batch_workspace_bytes(view, b, pkg.PREC_BF16X3), device="cuda", dtype=torch.uint8)
    ws.fill_(0x7f)  # padding rows of the operands are written by the call
    n0 = pkg.launch_count()
    pkg.diff2_coarse_batch(view, b, pkg.PREC_BF16X3, ws)
    torch.cuda.synchronize()
    # pixel list, phase tables (two kernels), normX, A, contraction and the projection with the norms or before them
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    if sms == 148:
        assert pkg.launch_count() - n0 == (7 if fused else 8)
    assert pkg.workspace_status(ws) == 0
    for p in sorted({0, P // 2, P - 1}):
        ref = torch.zeros(O * T, device="cuda", dtype=torch.float64)
        pkg.run_diff2_kernel_coarse_double(view, tx, ty, corr[p], re[p], im[p], d_eul, ref, O, T, N)
        assert ((out[p].reshape(-1).double() - ref).abs() / ref).max().item() <= 1e-5
