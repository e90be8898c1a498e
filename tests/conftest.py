"""Shared test set-up: the `gpu` marker, import paths and the oracle build."""
import os
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
if str(ROOT) not in sys.path:
    sys.path.insert(0, str(ROOT))

# CPU tests that check the table generators against the reference's data read it from the checkout
# the build recipe uses (VT_REFERENCE_ROOT); where it is absent they skip.
from __graft_entry__ import REFERENCE_DEFAULT  # noqa: E402

os.environ.setdefault("VT_REFERENCE_ROOT", REFERENCE_DEFAULT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (runs on the B200)")


# Where the generated data files are missing, GPU and oracle share closed-form stand-ins, and what compares
# against the reference's data or its own BSDF library skips.
from oracle import openpbr_ref, stand_in  # noqa: E402

STAND_INS = stand_in.install()
NEEDS_DATA = {"test_bsdf_matches_the_reference", "test_grid_builds_once_with_small_residuals",
              "test_grid_nodes_equal_the_reference_generator", "test_every_code_round_trips_within_half_a_step",
              "test_grid_lines_match_the_reference_generator", "test_sampled_codes_round_trip_within_half_a_step",
              "test_refined_cells_are_the_badly_interpolated_ones"}
if not openpbr_ref.available():
    openpbr_ref.load = lambda: pytest.skip(f"{openpbr_ref.LIB} is not built (it needs the reference checkout)")


def pytest_collection_modifyitems(items):
    for item in items:
        if STAND_INS and getattr(item, "originalname", item.name) in NEEDS_DATA:
            item.add_marker(pytest.mark.skip(reason="needs the generated data files (from the reference checkout)"))


@pytest.fixture(scope="session")
def oracle():
    from oracle import vt_oracle
    vt_oracle.load()
    return vt_oracle


@pytest.fixture(scope="session")
def ctx():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from metal_vibe_tracer_b200 import Context
    c = Context(0)
    yield c
    c.close()
