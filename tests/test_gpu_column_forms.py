"""The EOS kernel over flat arrays at the sizes where its blocks of cells end."""

import numpy as np
import pytest

from oracle import ocean_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 255, 257, 769, 1023, 1024, 1025, 700001])
@pytest.mark.parametrize("kind", ["linear", "seos", "teos10"])
def test_density_matches_oracle(kind, n):
    import torch
    from hydrostatic_ocean_core_benchmark_b200 import _lib
    rng = np.random.default_rng(n)
    T, S, z = 2.0 + 18.0 * rng.random(n), 33.0 + 3.0 * rng.random(n), 4000.0 * rng.random(n)
    if kind == "teos10":
        want = orc.rho_teos10(T, S, z)
    else:
        want = orc.rho_anomaly(kind, T, S, z, 1025.0, 2.0e-4, 7.4e-4, 10.0, 35.0)
    dT, dS, dz = (torch.as_tensor(a, device="cuda:0") for a in (T, S, z))
    out = torch.full((n + 4,), -7.0, dtype=torch.float64, device="cuda:0")
    stream = torch.cuda.current_stream()
    _lib.check(_lib.load().oc_density(("linear", "seos", "teos10").index(kind), 1025.0, 2.0e-4, 7.4e-4, 10.0, 35.0,
                                      dT.data_ptr(), dS.data_ptr(), dz.data_ptr(), out.data_ptr(), n,
                                      stream.cuda_stream), None, "oc_density")
    got = out.cpu().numpy()
    assert np.array_equal(got[:n], want)
    assert np.all(got[n:] == -7.0)
