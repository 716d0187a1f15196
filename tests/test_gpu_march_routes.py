"""Which kernel marches what, by cr_stats and cr_cluster_stats, and the routes that the register
march leaves to the others, against the oracle.

Bars as in test_gpu_parity: TL line 1e-3 dB, complex pressure 1e-6 relative.
"""
import numpy as np
import pytest

from cupyram_b200 import _lib, workloads
from cupyram_b200 import batch as B
from cupyram_b200.engine import Engine
from oracle import oracle
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


def _close(out, ref, n):
    assert np.abs(out["tll"][:n] - ref["tll"][:n]).max() < 1e-3
    assert np.abs(out["cpl"][:n] - ref["cpl"][:n]).max() < 1e-6 * np.abs(ref["cpl"][:n]).max()


# one row more than the register march takes, an uneven split over 16 CTAs, deeper
@pytest.mark.parametrize("nz", [6145, 6400, 7001])
@pytest.mark.parametrize("npd", [1, 2, 3, 6])
def test_column_kernel_in_complex128_beyond_the_register_march(cuda_device, monkeypatch, nz, npd):
    monkeypatch.setenv("CUPYRAM_B200_COL", "1")
    b = _batch(nz, npd, 2, True)
    with Engine(b) as eng:
        out = eng.run()
        st = eng.stats()
    assert (st["cluster_rays"], st["cluster_register_rays"], st["rays_failed"]) == (2, 0, 0)
    ref = oracle.run(b, "plain")
    _close(out, ref, b.line_len)
    g = b.grid_len
    assert np.abs(out["cpg"][:g] - ref["cpg"][:g]).max() < 1e-6 * np.abs(ref["cpg"][:g]).max()


@pytest.mark.parametrize("form", ["plain", "refined"])
@pytest.mark.parametrize("nz,npd", [(300, 5), (6200, 1), (6200, 6), (6144, 8)])
def test_batched_tiles_beside_the_default_march(cuda_device, monkeypatch, form, nz, npd):
    """The batched kernels of both FP64-accurate forms, against the oracle, and against the
    cluster march of the same rays: another kernel."""
    b = _batch(nz, npd, 40, True)
    monkeypatch.setenv("CUPYRAM_B200_COL", "0")
    with Engine(b, precision=form) as eng:
        out = eng.run()
        st = eng.stats()
    assert st["n_tiles"] > 0 and st["cluster_rays"] == 0 and st["precision_used"] == (3 if form == "refined" else 0)
    monkeypatch.setenv("CUPYRAM_B200_COL", "1")
    with Engine(b) as eng:
        other = eng.run()
        assert eng.stats()["n_tiles"] == 0
    one = _batch(nz, npd, 1, True)
    ref = oracle.run(one, "plain")
    n, g = one.line_len, one.grid_len
    for o in (out, other):
        _close(o, ref, n)
        assert np.abs(o["cpg"][:g] - ref["cpg"][:g]).max() < 1e-6 * np.abs(ref["cpg"][:g]).max()


def _mixed():
    """66 deep rays of 60 steps, 2 of 600, 30 shallow ones, interleaved; flat bottoms."""
    kind = (["deep"] * 2 + ["shallow"]) * 30 + ["deep"] * 6 + ["long"] * 2
    depth = [190.0 if k == "shallow" else 6240.0 for k in kind]
    rmax = np.array([15025.0 if k == "long" else 1525.0 for k in kind])
    n = len(kind)
    args = [np.full(n, 100.0), 50.0 + np.arange(n) % 7, np.full(n, 60.0),
            [np.array([0.0, 0.3 * d, d]) for d in depth], [np.array([0.0])] * n,
            [np.array([[1500.0], [1492.0 + i % 5], [1505.0]]) for i in range(n)],
            [np.array([0.0, 10.0])] * n, [np.array([0.0])] * n, [np.array([[1600.0], [1700.0]])] * n,
            [np.array([[1.4], [1.6]])] * n, [np.array([[0.3], [0.5]])] * n,
            [np.array([[0.0, 0.97 * d], [r, 0.97 * d]]) for d, r in zip(depth, rmax)]]
    kw = dict(batch_size=n, per_ray=True, rmax=rmax, dr=25.0, dz=1.0, np=5, lyrw=0.5, c0=np.full(n, 1500.0))
    envs, p, zs, zr, pr = B.prepare(*args, kw)
    b = B.build_batch(envs, p, zs, zr, pr, False)
    assert [k for k, nz in zip(kind, b.nz) if nz > 6144] == [k for k in kind if k != "shallow"]
    return b


@pytest.mark.parametrize("form", ["plain", "refined"])
def test_tiles_column_and_register_clusters_together(cuda_device, monkeypatch, form):
    """All three marches of one batch at once: columns too deep for registers in batched tiles,
    the two long ones of them on the column kernel, the shallow rays in registers.  Two marches
    agree to the last bit, and every ray with the oracle."""
    monkeypatch.delenv("CUPYRAM_B200_COL", raising=False)
    # costs that put a ray on the column kernel when it takes 1.25 times the batch's mean steps
    monkeypatch.setenv("CUPYRAM_B200_COSTS", "1e-9,1e8,0")
    b = _mixed()
    outs = []
    for _ in range(2):
        with Engine(b, precision=form) as eng:
            outs.append(eng.run())
            st = eng.stats()
    assert st["n_tiles"] > 0 and st["rays_failed"] == 0
    assert st["cluster_register_rays"] == 30 and st["cluster_rays"] == 32
    assert st["cluster_launches"] > st["cluster_register_launches"] > 0
    assert st["kernel_launches"] > st["cluster_launches"]
    n = b.line_len
    for key in ("tll", "cpl"):
        assert np.array_equal(outs[0][key][:n], outs[1][key][:n]), key
    ref = oracle.run(b, "plain")
    r = b.rays
    for i in range(b.n_rays):
        s = slice(int(r["line_off"][i]), int(r["line_off"][i] + r["nvr"][i]))
        assert np.abs(outs[0]["tll"][s] - ref["tll"][s]).max() < 1e-3, i
        assert np.abs(outs[0]["cpl"][s] - ref["cpl"][s]).max() < 1e-6 * np.abs(ref["cpl"][s]).max(), i


def test_chosen_tiles_beside_clusters_are_deterministic(cuda_device, monkeypatch):
    """The uneven wedge batch in the form that still splits it: a stale row read by a bulk copy
    beside the clusters would show as two marches that differ."""
    monkeypatch.delenv("CUPYRAM_B200_COL", raising=False)
    b = workloads.build(*workloads.wedge_batch(2000, seed=2024), compute_grids=False)
    outs = []
    for _ in range(2):
        with Engine(b, precision="chosen") as eng:
            outs.append(eng.run())
            st = eng.stats()
    assert st["n_tiles"] > 0 and st["cluster_launches"] > 0, st
    assert np.array_equal(outs[0]["tll"][:b.line_len], outs[1]["tll"][:b.line_len])
