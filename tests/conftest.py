import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
sys.path.insert(0, os.path.join(ROOT, "oracle"))


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200)")


# GPU tests against libraries built from the reference's own sources
# (oracle/_ref), which exist only where its tree was at hand for the build
FROM_REFERENCE = ("test_adiabatic_bit_exact_short", "test_adiabatic_matches_reference", "test_dropin_reproduces_reference",
                  "test_dust_diffusion_bit_exact_short", "test_dust_diffusion_matches_reference",
                  "test_dat_files_equal_the_references_own_writer", "test_fp64_full_size_matches_reference",
                  "test_stock_step_loop_on_the_b200", "test_outputs_and_host_writes_follow_the_freshness_protocol")


def pytest_collection_modifyitems(items):
    """Where those libraries are missing, the tests that fail for it run after
    all others, so that a run that stops at the first failure has made the
    others' checks."""
    ref = os.path.join(ROOT, "oracle", "_ref")
    if not (os.path.isdir(ref) and any(f.endswith(".so") for f in os.listdir(ref))):
        items.sort(key=lambda it: it.name.split("[")[0] in FROM_REFERENCE)


def gpu_available() -> bool:
    try:
        import torch
        return torch.cuda.is_available()
    except Exception:
        return False


@pytest.fixture(scope="session")
def oracle_lib():
    import pyoracle
    pyoracle.build()
    return pyoracle
