"""Minima that a caller keeps inside the weights' workspace, whose contents the
call ignores: they are read before the workspace is written.  The weights are bit
for bit those with the minima elsewhere."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 256, 512])  # the minima, the chunk sums, the counters
@pytest.mark.parametrize("normalize", [False, True])
def test_minima_in_the_workspace(pkg, cuda, offset, normalize):
    torch = cuda
    P, O, T = 3, 3500, 20  # three chunks of samples
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    d2 = torch.randn(P, O, T, generator=g, device="cuda") * 5 + 400
    mn = d2.reshape(P, -1).min(1).values.double()
    nbytes = pkg.lib().b200d2_coarse_weights_workspace(P, O * T)
    got = []
    for inside in (False, True):
        ws = torch.zeros(max(nbytes, offset + 8 * P), device="cuda", dtype=torch.uint8)
        m = mn.clone()
        if inside:
            m = ws[offset:offset + 8 * P].view(torch.float64)
            m.copy_(mn)
        w, s = torch.empty((P, O, T), device="cuda", dtype=torch.float64), torch.empty(P, device="cuda", dtype=torch.float64)
        pkg.coarse_weights(d2, P, O, T, out_min=m, weights=w, sums=s, workspace=ws, normalize=normalize)
        torch.cuda.synchronize()
        got.append((w, s))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
