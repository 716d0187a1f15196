"""What bench.py says of a march: the form that ran and the bytes of that form (CPU)."""
import sys
from pathlib import Path

import pytest

sys.path.insert(0, str(Path(__file__).resolve().parent.parent))
import bench  # noqa: E402
from cupyram_b200 import _lib  # noqa: E402

CODES = {"plain": _lib.CR_PLAIN_C128, "chosen": _lib.CR_CHOSEN_C64R, "fast": _lib.CR_CHOSEN_C64,
         "refined": _lib.CR_C64_REFINED}


@pytest.mark.parametrize("asked,ran,tiles", [("plain", "plain", 0), ("refined", "plain", 0), ("refined", "refined", 9),
                                             ("chosen", "chosen", 9), ("fast", "plain", 9)])
def test_record_describes_the_form_that_ran(asked, ran, tiles):
    st = {"precision_used": CODES[ran], "n_tiles": tiles}
    assert bench.form_marched(asked, st) == ran
    assert ran in bench.FORM_DESC
    r = bench.roofline(2e9, 0.5, asked, st, 1000.0, None)
    assert r["bytes_per_point_update"] == bench.B_ALG[ran]
    assert r["achieved"] == pytest.approx(2e9 * bench.B_ALG[ran] / 0.5 / 1e9)
    assert r["frac"] == pytest.approx(r["achieved"] / 1000.0)
    assert ("note" in r) == (tiles == 0)
    assert bench.roofline(2e9, 0.5, asked, st, 1000.0, 70.0)["traffic"] == pytest.approx(1.4e11)
