"""The kernels counted for a graph (a plan's, a repeated batch's) are those that
its capture recorded, whatever other threads launch meanwhile."""
from __future__ import annotations

import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_graphs_captured_beside_other_launches(pkg, synth, cuda):
    torch = cuda
    pr = synth.make_problem("tiny", P=4)
    proj = pkg.Projector(pr.projector, use_texture=1)
    view = proj.view(pr.imgX, pr.imgY, pr.imgMaxR)
    dev = lambda a: torch.as_tensor(np.ascontiguousarray(a, np.float32), device="cuda")  # noqa: E731
    eul, re, im, corr = dev(pr.eulers.reshape(-1)), dev(pr.fimg_re), dev(pr.fimg_im), dev(pr.corr)
    tx, ty = dev(pr.trans_x), dev(pr.trans_y)
    orient = np.arange(pr.O, dtype=np.int32)

    def plan_launches():
        outs = torch.empty((pr.P, pr.O, pr.T), device="cuda")
        parts = [dict(real=re[p], imag=im[p], corr=corr[p], diff2=outs[p], orient=orient, trans_x=pr.trans_x,
                      trans_y=pr.trans_y) for p in range(pr.P)]
        return pkg.Plan(view, eul, pr.O, pr.N_img, parts, precision=pkg.PREC_TF32, flags=pkg.PLAN_GRAPH)

    def batch():
        out = torch.empty((pr.P, pr.O, pr.T), device="cuda")
        b = pkg.make_batch(eul, tx, ty, re, im, corr, out, O=pr.O, T=pr.T, P=pr.P, N_img=pr.N_img)
        ws = torch.empty(pkg.batch_workspace_bytes(view, b, pkg.PREC_TF32), device="cuda", dtype=torch.uint8)
        return lambda: pkg.diff2_coarse_batch(view, b, pkg.PREC_TF32, ws), (out, ws)

    def counted(f):
        n0 = pkg.launch_count()
        f()
        return pkg.launch_count() - n0

    quiet = plan_launches()
    want = counted(quiet.run)
    call, keep = batch()
    want_batch = counted(call)
    stop = threading.Event()
    scores, mn = torch.rand(64, device="cuda"), torch.empty(1, device="cuda", dtype=torch.float64)
    am, side = torch.empty(1, device="cuda", dtype=torch.int64), torch.cuda.Stream()

    def other():
        while not stop.is_set():
            pkg.minloc(scores, 64, 1, mn, am, stream=side)

    threads = [threading.Thread(target=other) for _ in range(2)]
    for t in threads:
        t.start()
    plans, batches = [], []
    for _ in range(8):
        plans.append(plan_launches())
        batches.append(batch())
        for _ in range(2):  # the second call captures
            batches[-1][0]()
    stop.set()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert [counted(p.run) for p in plans] == [want] * 8
    assert [counted(c) for c, _ in batches] == [want_batch] * 8
    for p in (quiet, *plans):
        p.close()
    proj.close()
