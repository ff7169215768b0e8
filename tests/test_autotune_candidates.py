"""The tuner's default candidates are launches that differ: a cap on the resident
blocks per SM lies below what the step's kernels hold anyway, and the exact form,
which has one set of kernels, is timed as one form."""
import os
import re

from romspath_b200 import autotune

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "romspath_b200", "csrc")


def test_candidates_differ_in_what_they_launch():
    text = open(os.path.join(CSRC, "rp_internal.h")).read()
    held = {k: int(re.search(rf"#define {k} (\d+)", text).group(1)) for k in ("RP_MIXED_MIN_BLOCKS", "RP_VTURB_MIN_BLOCKS")}
    most = min(held["RP_MIXED_MIN_BLOCKS"], held["RP_VTURB_MIN_BLOCKS"] // 4)     # k_vturb's blocks are one warp of four
    c = autotune.DEFAULT_CANDIDATES
    assert len(set(c)) == len(c)
    assert all(bps == 0 or bps < most for _, bps in c)


def test_exact_form_is_one_form():
    """launch_step takes no form: the exact step's kernels are the same under every one"""
    decl = re.search(r"cudaError_t launch_step\(([^;]*)\);", open(os.path.join(CSRC, "rp_internal.h")).read()).group(1)
    assert "variant" not in decl and "form" not in decl and "split" not in decl
    assert len(autotune.EXACT_FORMS) == 1
