"""The C-ABI library loads and exports every entry point that include/pdgpu.h declares (no GPU needed)."""
import os
import re

import pytest

from conftest import ROOT, gpu_available


def declared_functions():
    with open(os.path.join(ROOT, "include", "pdgpu.h")) as f:
        text = f.read()
    return sorted(set(re.findall(r"^\s*(?:int|const char \*)\s*(pdg_\w+)\s*\(", text, re.M)))


def test_header_declares_entry_points():
    names = declared_functions()
    assert "pdg_fock_two_electron" in names and "pdg_scf_run" in names


def test_library_exports_every_declared_symbol():
    from pdynamo3_b200 import lib
    L = lib.load()
    for name in declared_functions():
        assert hasattr(L, name), name
    assert set(declared_functions()) <= set(lib.EXPORTS) | set(declared_functions())


def test_version_and_error_string():
    from pdynamo3_b200 import lib
    L = lib.load()
    assert L.pdg_version() >= 100
    assert isinstance(L.pdg_last_error(), bytes)


@pytest.mark.skipif(gpu_available(), reason="needs a machine without a device")
def test_purification_without_a_place_for_its_cluster():
    """Where eight CTAs of the one-launch purification cannot run together (here: no device), the library says
    so, and an SCF takes the GEMM form, instead of failing in the launch."""
    from pdynamo3_b200 import lib
    L = lib.load()
    assert [L.pdg_purify_clusters(m) for m in (1, 64, 128, 129)] == [0, 0, 0, 0]
