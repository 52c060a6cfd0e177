"""The drop-in `run(...)` where no GPU is needed: how it sets up and shares its handles."""
import re
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_option_matches_the_header(pkg):
    txt = (ROOT / "include" / "moe_fp8_b200.h").read_text()
    value = re.search(r"MOE_FP8_B200_OPT_SCALES_IN_PLACE\s*=\s*(\d+)", txt).group(1)
    assert int(value) == pkg._lib.OPT_SCALES_IN_PLACE
