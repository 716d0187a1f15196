"""Pade sets of different lengths on the register march (cr_set_pade), against the oracle.

A ray marches four sets in turn: the self-starter's, the ip=2 step's, the
march's and, past the stability range, the unconstrained march's.  Each may
have any number of terms up to what the ray was laid out for, so a term's warp
may sit out steps at the start, in the middle or at the end of the march; the
mailboxes that the CTAs of a cluster exchange through have to follow the steps
it took part in.  On one CTA and on clusters, sums over all terms and over pairs.

Bars as in test_gpu_parity: TL line 1e-3 dB, complex pressure 1e-6 relative.
"""
import numpy as np
import pytest

from cupyram_b200.engine import Engine
from cupyram_b200.pade import compute_pade_coefficients
from oracle import oracle
from test_gpu_reg import _batch

FREQ, C0, DR, NP = 100.0, 1500.0, 25.0, 8


def _sets(counts):
    """One set per count (0: the engine's own), each the expansion of its own order; the
    self-starter's is the product of 1 / (1 - X / 2^j)."""
    sets = {}
    for which, (n, ip, ns) in enumerate(zip(counts, (0, 2, 1, 1), (0, 1, 1, 0))):
        if n and which == 0:
            sets[which] = np.zeros(n, complex), -0.5 ** np.arange(n) + 0j
        elif n:
            sets[which] = compute_pade_coefficients(FREQ, C0, n, ns, DR, ip)
    return sets


@pytest.mark.gpu
@pytest.mark.parametrize("counts", [(0, 3, 0, 0), (0, 0, 5, 0), (0, 0, 0, 2), (2, 0, 0, 0), (3, 1, 0, 4), (1, 8, 2, 7),
                                    (8, 4, 1, 8)])
@pytest.mark.parametrize("nz,rays", [(140, 1), (700, 1), (2400, 1), (224, 300), (352, 300)])
def test_sets_of_unequal_length_vs_oracle(cuda_device, nz, rays, counts):
    sets = _sets(counts)
    b = _batch(nz, NP, rays, True)
    b.rays["rs"] = 140.0  # the last set from the fifth of ten steps on
    with Engine(b) as eng:
        for ray in range(rays):
            for which, (p1, p2) in sets.items():
                eng.set_pade(ray, which, p1, p2)
        out = eng.run()
        assert eng.stats()["rays_failed"] == 0 and eng.stats()["n_tiles"] == 0
    for key, width in (("cpl", b.line_len), ("cpg", b.grid_len)):
        v = out[key][:width].reshape(rays, -1)
        assert (v == v[0]).all(), key
    one = _batch(nz, NP, 1, True)
    one.rays["rs"] = 140.0
    ref = oracle.run(one, "plain", sets=sets)
    n = one.line_len
    assert np.abs(out["tll"][:n] - ref["tll"][:n]).max() < 1e-3
    assert np.abs(out["cpl"][:n] - ref["cpl"][:n]).max() < 1e-6 * np.abs(ref["cpl"][:n]).max()
    g = one.grid_len
    assert np.abs(out["cpg"][:g] - ref["cpg"][:g]).max() < 1e-6 * np.abs(ref["cpg"][:g]).max()


def test_oracle_takes_sets_in_place_of_its_own():
    """The oracle with its own sets handed back, and with others."""
    b = _batch(140, NP, 1, False)
    b.rays["rs"] = 140.0
    same = {w: oracle.pade(FREQ, C0, NP, ns, DR, ip) for w, ns, ip in ((1, 1, 2), (2, 1, 1), (3, 0, 1))}
    same[0] = np.zeros(1, complex), np.full(1, -1.0 + 0j)
    ref = oracle.run(b, "plain")["cpl"]
    assert np.array_equal(oracle.run(b, "plain", sets=same)["cpl"], ref)
    for w in range(4):
        other = oracle.run(b, "plain", sets=_sets([3 if q == w else 0 for q in range(4)]))["cpl"]
        assert not np.array_equal(other, ref), w
