"""Where the reference's own kernels are not built, the tests that compare with
them are skipped, and those that only share their fixtures still run."""
from __future__ import annotations

import types

import pytest

from conftest import skip_without_reference_kernels
from gpu_util import RefKernels


def _oracle(available):
    def ref_lib():
        if not available:
            raise OSError("libref_diff2.so: cannot open shared object file")
        return "library"
    return skip_without_reference_kernels(types.SimpleNamespace(ref_available=lambda: available, ref_lib=ref_lib))


def test_absent_kernels_skip():
    ref = RefKernels(_oracle(False), None)  # a fixture shared with tests that do not use them
    with pytest.raises(pytest.skip.Exception):
        ref.L
    with pytest.raises(pytest.skip.Exception):
        ref.h
    ref.close()


def test_present_kernels_load():
    assert RefKernels(_oracle(True), None).L == "library"
