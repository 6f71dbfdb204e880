"""The fine pass at the largest images whose columns, phase tables and sums fit in
one CTA's shared memory (194 KB), and the first that do not: the checks, the
reference and the tolerance of the column kernel's test."""
from __future__ import annotations

import pytest

import test_gpu_fine_rows as rows

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cc", [False, True], ids=["diff2", "cc"])
@pytest.mark.parametrize("interp", ["TEXTURE", "LINEAR"])
@pytest.mark.parametrize("imgX,imgY,R,cut", [(94, 186, 32, 0), (98, 194, 32, 37), (100, 197, 32, 0), (102, 200, 32, 0),
                                             (288, 60, 30, 0)])
def test_large_images(pkg, synth, cuda, imgX, imgY, R, cut, interp, cc):
    rows.test_fine_rows(pkg, synth, cuda, imgX, imgY, R, cut, 1.0, interp, cc)
