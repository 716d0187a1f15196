"""The register-resident column march (complex128) at the edges of its shapes.

A ray's column is cut over 1 to 16 CTAs, a CTA's slice over 32 lanes of at most
12 rows: the depths below put slices at, just under and just over whole lanes
and the longest segments, on one CTA and on clusters, with every number of
Pade terms from 1 to 10, moving bottoms, profile updates and decimated grids.
Single rays get many CTAs, batches of copies few (the engine's plan); copies
must agree bit for bit.

Bars as in test_gpu_parity: TL line 1e-3 dB, complex pressure 1e-6 relative
(the Pade coefficients of device and host agree to 1e-8).
"""
import numpy as np
import pytest

from cupyram_b200 import batch as B
from cupyram_b200.engine import Engine
from oracle import oracle

pytestmark = pytest.mark.gpu

SINGLE = [(40, 1), (63, 2), (64, 3), (127, 4), (129, 5), (383, 6), (385, 7), (1000, 8), (1025, 9), (2400, 10), (4097, 6),
          (6144, 6), (6145, 6)]
COPIES = [(96, 1), (97, 2), (128, 3), (129, 10), (161, 4), (192, 5), (193, 6), (255, 7), (257, 8), (320, 9), (321, 6),
          (384, 10), (385, 6), (768, 4), (769, 8), (1537, 2)]


def _batch(nz, npd, rays, grids):
    """`rays` copies of one ray of nz rows (dz 1 m) over a sloping bottom, three profiles, 10 steps of 25 m."""
    freq, lyrw = 100.0, 0.5
    floor = nz + 1 - lyrw * 15.0          # bottom of the sediment: zmax = floor + lyrw * lambda
    depth = floor - 12.0
    dip = min(6.0, 0.3 * depth)
    z = np.array([0.0, 0.4 * depth, depth])
    cw = np.array([[1500.0, 1503.0, 1498.0], [1490.0, 1493.0, 1496.0], [1505.0, 1502.0, 1500.0]])
    args = [np.full(rays, freq), np.full(rays, 0.3 * depth), np.full(rays, 0.4 * depth),
            [z] * rays, [np.array([0.0, 90.0, 160.0])] * rays, [cw] * rays,
            [np.array([0.0, 12.0])] * rays, [np.array([0.0])] * rays, [np.array([[1600.0], [1700.0]])] * rays,
            [np.array([[1.4], [1.6]])] * rays, [np.array([[0.3], [0.5]])] * rays,
            [np.array([[0.0, 0.6 * depth], [140.0, 0.6 * depth + dip], [300.0, 0.6 * depth + 1.0]])] * rays]
    kw = dict(batch_size=rays, per_ray=True, rmax=275.0, dr=25.0, dz=1.0, np=npd, lyrw=lyrw, c0=np.full(rays, 1500.0),
              ndr=2, ndz=3, compute_grids=grids)
    envs, p, zs, zr, pr = B.prepare(*args, kw)
    b = B.build_batch(envs, p, zs, zr, pr, grids)
    assert set(b.nz.tolist()) == {nz}
    return b


def _check(b, out, ray0):
    ref = oracle.run(b, "plain")
    n, g = b.line_len, b.grid_len
    assert np.abs(out["tll"][:n] - ref["tll"][:n]).max() < 1e-3
    assert np.abs(out["cpl"][:n] - ref["cpl"][:n]).max() < 1e-6 * np.abs(ref["cpl"][:n]).max()
    if g:
        assert np.abs(ray0[:g] - ref["cpg"][:g]).max() < 1e-6 * np.abs(ref["cpg"][:g]).max()


@pytest.mark.parametrize("nz,npd", SINGLE)
def test_single_ray_vs_oracle(cuda_device, nz, npd):
    b = _batch(nz, npd, 1, True)
    with Engine(b) as eng:
        out = eng.run()
        assert eng.stats()["rays_failed"] == 0
    _check(b, out, out["cpg"])


@pytest.mark.parametrize("nz,npd", COPIES)
def test_batch_of_copies_vs_oracle(cuda_device, nz, npd):
    rays = 330
    b = _batch(nz, npd, rays, True)
    with Engine(b) as eng:
        out = eng.run()
        assert eng.stats()["rays_failed"] == 0 and eng.stats()["n_tiles"] == 0
    for key, width in (("tll", b.line_len), ("cpl", b.line_len), ("tlg", b.grid_len), ("cpg", b.grid_len)):
        v = out[key][:width].reshape(rays, -1)
        assert (v == v[0]).all(), key
    one = _batch(nz, npd, 1, True)
    _check(one, {k: out[k] for k in ("tll", "cpl")}, out["cpg"])


def test_changed_order_of_a_set(cuda_device):
    """cr_set_pade with fewer terms than the ray was laid out for: the idle warps
    take part in the CTA's barriers only."""
    from cupyram_b200.pade import compute_pade_coefficients
    b = _batch(700, 6, 1, False)
    small = _batch(700, 3, 1, False)
    with Engine(b) as eng, Engine(small) as ref:
        for which, ip, ns in ((1, 2, 1), (2, 1, 1), (3, 1, 0)):
            p1, p2 = compute_pade_coefficients(100.0, 1500.0, 3, ns, 25.0, ip)
            eng.set_pade(0, which, p1, p2)
            ref.set_pade(0, which, p1, p2)
        a, c = eng.run(), ref.run()
    n = b.line_len
    assert np.abs(a["cpl"][:n] - c["cpl"][:n]).max() < 1e-6 * np.abs(c["cpl"][:n]).max()


# segments of 7, 9 and 11 rows at their edges; the sum over all terms or over pairs (8 and 10 terms leave less room)
@pytest.mark.parametrize("nz,npd", [(193, 1), (224, 6), (193, 8), (224, 10), (257, 3), (288, 6), (288, 7), (321, 2),
                                    (352, 6), (352, 8), (160, 8), (160, 10), (320, 6)])
def test_odd_segments_and_sums_vs_oracle(cuda_device, nz, npd):
    rays = 300
    b = _batch(nz, npd, rays, True)
    with Engine(b) as eng:
        out = eng.run()
        assert eng.stats()["rays_failed"] == 0 and eng.stats()["n_tiles"] == 0
    _check(_batch(nz, npd, 1, True), {k: out[k] for k in ("tll", "cpl")}, out["cpg"])
