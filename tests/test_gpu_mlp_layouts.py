"""Weights, gradients and moments in a user's own layouts: column ranges of wider
matrices, and views that do not start on 16-byte boundaries.  The whole-network
calls take dense, aligned matrices; every other layout has to give the same
results as dense copies of it, to the last bit, and write nothing beside it."""
import pytest

pytestmark = pytest.mark.gpu

DIMS, BATCH = [128, 384, 256, 256], 256


def _wide(t):
    """t as a column range of a wider matrix (rows still on 16-byte boundaries)."""
    import torch
    big = torch.full((t.shape[0], t.shape[1] + 32), 7.0, dtype=t.dtype, device=t.device)
    big[:, 16:-16] = t
    return big[:, 16:-16], big


def _shifted(t, by):
    """t dense, `by` elements off a 16-byte boundary."""
    import torch
    flat = torch.full((t.numel() + 16,), 7.0, dtype=t.dtype, device=t.device)
    flat[by:by + t.numel()] = t.reshape(-1)
    return flat[by:by + t.numel()].view(t.shape), flat


def _untouched(v, big):
    """Nothing outside the view v of `big` was written."""
    if big.dim() == 2:
        return bool((big[:, :16] == 7.0).all() and (big[:, -16:] == 7.0).all())
    off = v.storage_offset()
    return bool((big[:off] == 7.0).all() and (big[off + v.numel():] == 7.0).all())


@pytest.mark.parametrize("layout", ["weights", "transposes", "gradients", "all", "shifted", "one_layer_shifted"])
def test_training_step_in_other_layouts(cuda_device, layout):
    import torch
    from cupyram_b200 import surrogate as S
    a, b = S.MLP(DIMS, seed=4), S.MLP(DIMS, seed=4)
    kept = []

    def move(name, f, layers=range(len(DIMS) - 1)):
        lst = getattr(b, name)
        for l in layers:
            lst[l], big = f(lst[l])
            kept.append((lst[l], big))
    if layout in ("weights", "all"):
        move("Wb", _wide)
    if layout in ("transposes", "all"):
        move("WTb", _wide)
    if layout in ("gradients", "all"):
        move("gW", _wide)
    if layout == "all":
        for name in ("W", "mW", "vW"):
            move(name, _wide)
    if "shifted" in layout:
        layers = [1] if layout.startswith("one") else range(len(DIMS) - 1)
        for name in ("W", "mW", "vW"):
            move(name, lambda t: _shifted(t, 1), layers)
        move("gW", lambda t: _shifted(t, 2), layers)  # the contraction stores pairs
    g = torch.Generator(device="cuda").manual_seed(1)
    S.tc_error_flag().zero_()
    for step in range(2):
        X = torch.randn(BATCH, DIMS[0], generator=g, device="cuda").to(torch.bfloat16)
        d = torch.randn(BATCH, DIMS[-1], generator=g, device="cuda").to(torch.bfloat16)
        for m in (a, b):
            m.forward(X)
            m.backward(d)
            m.step(1e-3, weight_decay=0.01)
        assert torch.equal(a.forward(X), b.forward(X)), step
        for name in ("gW", "gb", "W", "b", "mW", "vW", "mb", "vb", "Wb", "WTb"):
            for l, (x, y) in enumerate(zip(getattr(a, name), getattr(b, name))):
                assert torch.equal(x, y), (name, l, step)
    assert all(_untouched(v, big) for v, big in kept)
    assert int(S.tc_error_flag().item()) == 0


def test_predict_with_weights_in_a_wider_matrix(cuda_device):
    import torch
    from cupyram_b200 import surrogate as S
    a, b = (S.Ensemble(3, [128, 256, S.NZ_OUT * S.NR_OUT], seed=1) for _ in range(2))
    b.models[1].Wb = [_wide(w)[0] for w in b.models[1].Wb]
    X = torch.randn(256, 128, generator=torch.Generator(device="cuda").manual_seed(2), device="cuda").to(torch.bfloat16)
    (m0, s0), (m1, s1) = a.predict(X), b.predict(X)
    # the members' outputs are the same; the statistics' own FP32 rounding of values up to 150
    assert (m0 - m1).abs().max() <= 150 * 2 ** -22
    assert (s0 - s1).abs().max() <= 1e-3
