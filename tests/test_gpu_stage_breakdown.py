"""The stages that a breakdown reports are those that launch something."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("minima", [False, True])
@pytest.mark.parametrize("interp", ["TEXTURE", "LINEAR"])
def test_reported_stages(pkg, synth, cuda, interp, minima):
    torch = cuda
    pr = synth.make_problem("c1", P=8)
    proj = pkg.Projector(pr.projector, use_texture=2)
    view = proj.view(pr.imgX, pr.imgY, pr.imgMaxR, interp=getattr(pkg, "INTERP_" + interp))
    dev = lambda a: torch.as_tensor(np.ascontiguousarray(a, np.float32), device="cuda")  # noqa: E731
    args = [dev(a) for a in (pr.eulers.reshape(-1), pr.trans_x, pr.trans_y, pr.fimg_re, pr.fimg_im, pr.corr)]
    out, mn = torch.empty((pr.P, pr.O, pr.T), device="cuda"), torch.empty(pr.P, device="cuda", dtype=torch.float64)
    b = pkg.make_batch(*args, out, O=pr.O, T=pr.T, P=pr.P, N_img=pr.N_img, out_min=mn if minima else None)
    ws = torch.empty(pkg.batch_workspace_bytes(view, b, pkg.PREC_BF16X3), device="cuda", dtype=torch.uint8)
    per = pkg.kernel_breakdown(view, b, pkg.PREC_BF16X3, ws)["per_kernel_ms"]
    names = pkg.stage_names(pkg.PREC_BF16X3)
    # with the texture these 8 particles' norms are taken in the projection kernel
    absent = {n for n in names if ("project_kernel" in n and interp == "TEXTURE") or ("finalize" in n and not minima)}
    assert set(per) == set(names) - absent and all(v > 0 for v in per.values())
    proj.close()
