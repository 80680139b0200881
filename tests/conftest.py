import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200) and the built native library")


# compare with the reference's own code, compiled from its sources: skipped,
# like the tests that say so themselves, where that library has not been built
NEED_REFERENCE = {"test_localizer_fit_emitters_matches_reference_pipeline", "test_workload_full_size_against_reference"}


def pytest_collection_modifyitems(items):
    from oracle import oracle
    if oracle.ref_available():
        return
    for item in items:
        if getattr(item, "originalname", item.name) in NEED_REFERENCE:
            item.add_marker(pytest.mark.skip(reason="reference build absent"))
