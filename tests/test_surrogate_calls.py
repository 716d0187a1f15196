"""What the surrogate's whole-network calls refuse, on the host: no case here reaches a launch."""
import ctypes
from types import SimpleNamespace

import pytest

from cupyram_b200 import surrogate as S

FAKE = 4096  # an aligned device address that is never read


def _net(dims):
    L = len(dims) - 1
    ptrs = (ctypes.c_void_p * L)(*[FAKE] * L)
    d = (ctypes.c_int * (L + 1))(*dims)
    net = S._Net(layers=L, dims=ctypes.addressof(d))
    for name, _ in S._Net._fields_[2:]:
        setattr(net, name, ctypes.addressof(ptrs))
    net.keep = ptrs, d
    return net


@pytest.mark.parametrize("widths", [(256, 512), (512, 256), (256, 256, 384), (128, 128, 128, 128, 256)])
@pytest.mark.parametrize("tc", [0, 1])
def test_ensemble_members_must_have_one_output_width(lib_built, widths, tc):
    nets = [_net([128, w]) for w in widths]
    n = len(nets)
    rc = S.kernels().cr_mlp_ensemble_predict((ctypes.c_void_p * n)(*[ctypes.addressof(t) for t in nets]), n, 128, FAKE,
                                             128, (ctypes.c_void_p * n)(*[FAKE] * n), tc, 1.0, 0.0, 0.0, 1.0, FAKE,
                                             FAKE, FAKE, None)
    assert rc == 1  # CR_MLP_EBADSHAPE, before any launch


@pytest.mark.parametrize("d_out", [4096, 16384])
def test_predict_refuses_members_of_another_field_size(d_out):
    """The results hold 64 x 128 values a request: members with fewer or more outputs were
    never accepted, and would be written past the results' end."""
    torch = pytest.importorskip("torch")
    ens = S.Ensemble.__new__(S.Ensemble)
    ens.models = [SimpleNamespace(dims=[S.D_IN, d_out], Wb=[]) for _ in range(2)]
    with pytest.raises(ValueError, match="outputs"):
        ens.predict(torch.zeros(128, S.D_IN, dtype=torch.bfloat16), check=False)
