"""Shared fixtures: the package (loaded from t2-relion-kernel_b200/ as
`relion_b200`), the oracle, and the `gpu` marker."""
from __future__ import annotations

import importlib.util
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG_DIR = os.path.join(ROOT, "t2-relion-kernel_b200")
sys.path.insert(0, os.path.join(ROOT, "oracle"))


def load_package():
    if "relion_b200" in sys.modules:
        return sys.modules["relion_b200"]
    spec = importlib.util.spec_from_file_location(
        "relion_b200", os.path.join(PKG_DIR, "__init__.py"), submodule_search_locations=[PKG_DIR])
    mod = importlib.util.module_from_spec(spec)
    sys.modules["relion_b200"] = mod
    spec.loader.exec_module(mod)
    return mod


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200, sm_100a)")


@pytest.fixture(scope="session")
def pkg():
    return load_package()


@pytest.fixture(scope="session")
def synth(pkg):
    import importlib
    return importlib.import_module("relion_b200.synth")


def skip_without_reference_kernels(o):
    """The reference project's own GPU kernels can only be built where its
    sources are: without them, a test that asks for them is skipped."""
    if not o.ref_available():
        def ref_lib():
            pytest.skip("the reference's own kernels (oracle/_ref) are not built here")
        o.ref_lib = ref_lib
    return o


@pytest.fixture(scope="session")
def oracle():
    import oracle as o
    o.lib()
    return skip_without_reference_kernels(o)


@pytest.fixture(scope="session")
def cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch
