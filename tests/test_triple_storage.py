"""The shared memory the triple kernels take with the autotuner's candidates and the chosen values: a staged neighbor is
two float4, an index and (damped) three floats, and the fast kernel stages twice IX_TUNE_ATM_FAST for each of 4 warps."""
import re

import pytest

import build_lib
import tune

SOURCE = (build_lib.CSRC / "ix_atm.cuh").read_text()
ENTRY = 16 + 16 + 4 + 12


def _candidates():
    return [dict(tune.DEFAULTS, **build_lib.tuned_values())] + [dict(tune.DEFAULTS, **o) for _, options in tune.GROUPS
                                                                for o in options]


def test_storage_is_as_counted_here():
    assert "constexpr int kAtmFastStaged = 2 * kAtmFast;" in SOURCE and "constexpr int kAtmFastWarps = 4;" in SOURCE
    body = re.search(r"struct TripleStorage \{(.*?)\};", SOURCE, re.S).group(1)
    assert [" ".join(line.split()) for line in body.strip().splitlines()] == [
        "float4 pos[N];", "float4 par[N];", "int site[N];", "SiteDamping damp[DAMP ? N : 1];"]


@pytest.mark.parametrize("values", _candidates(), ids=lambda v: f"{v['IX_TUNE_ATM_FAST']}x{v['IX_TUNE_ATM_MIN_BLOCKS']}")
def test_fast_kernel_fits(values):
    block = 4 * 2 * values["IX_TUNE_ATM_FAST"] * ENTRY
    assert block < 48 * 1024
    assert (block + 1024) * values["IX_TUNE_ATM_MIN_BLOCKS"] <= 228 * 1024


def test_limits_are_checked_where_the_kernels_are_compiled():
    for storage in ("kAtmFastWarps * sizeof(TripleStorage<true, kAtmFastStaged>)",
                    "kAtmWarps * sizeof(TripleStorage<true, kAtmMaxStaged>)"):
        assert re.search(r"static_assert\(\(?" + re.escape(storage), SOURCE)
