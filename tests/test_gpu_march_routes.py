"""Which kernel marches what, by cr_stats and cr_cluster_stats, and the routes that the register
march leaves to the others, against the oracle.

Bars as in test_gpu_parity: TL line 1e-3 dB, complex pressure 1e-6 relative.
"""
import pytest

from cupyram_b200 import _lib
from cupyram_b200.engine import Engine
from test_gpu_reg import _batch

pytestmark = pytest.mark.gpu


# (form, depth, rays, CUPYRAM_B200_COL, CUPYRAM_B200_SUM) -> (rays on clusters, of these in registers, form used)
@pytest.mark.parametrize("form,nz,rays,col,summed,on_clusters,in_registers,used", [
    ("plain", 300, 40, None, None, 40, 40, "CR_PLAIN_C128"),
    ("refined", 300, 40, None, None, 40, 40, "CR_PLAIN_C128"),
    ("plain", 300, 40, "1", None, 40, 40, "CR_PLAIN_C128"),
    ("plain", 300, 40, "0", None, 0, 0, "CR_PLAIN_C128"),
    ("refined", 300, 40, "0", None, 0, 0, "CR_C64_REFINED"),
    ("chosen", 300, 40, "0", None, 0, 0, "CR_CHOSEN_C64R"),
    ("chosen", 300, 40, "1", None, 40, 0, "CR_CHOSEN_C64R"),
    ("fast", 300, 40, "1", None, 40, 0, "CR_CHOSEN_C64"),
    ("plain", 6145, 2, "1", None, 2, 0, "CR_PLAIN_C128"),
    ("refined", 6145, 2, "1", None, 2, 0, "CR_PLAIN_C128"),
    ("refined", 300, 40, None, "0", 0, 0, "CR_PLAIN_C128"),
])
def test_statistics_name_what_marches(cuda_device, monkeypatch, form, nz, rays, col, summed, on_clusters, in_registers,
                                      used):
    for name, v in (("CUPYRAM_B200_COL", col), ("CUPYRAM_B200_SUM", summed)):
        monkeypatch.delenv(name, raising=False)
        if v is not None:
            monkeypatch.setenv(name, v)
    b = _batch(nz, 4, rays, False)
    with Engine(b, precision=form) as eng:
        laid = eng.stats()
        assert laid["cluster_launches"] == laid["cluster_register_launches"] == 0  # nothing marched yet
        eng.run()
        st = eng.stats()
    assert (st["cluster_rays"], st["cluster_register_rays"]) == (on_clusters, in_registers)
    assert st["precision_used"] == getattr(_lib, used)
    assert (st["n_tiles"] == 0) == (on_clusters == rays)
    assert (st["cluster_launches"] > 0) == (on_clusters > 0)
    assert (st["cluster_register_launches"] > 0) == (in_registers > 0)
    if on_clusters == rays:
        assert st["kernel_launches"] == st["cluster_launches"]
