"""FP32 fields cross to and from the host at the sizes where the conversion moves
from the host to the device, in pageable and pinned memory."""
import numpy as np
import pytest

from hydist_c_b200 import scenario as S

pytestmark = pytest.mark.gpu


# (N+3)*(M+3) values: 2048 and 2050, 8190 and 8196, 131072 and 131076
@pytest.mark.parametrize("N,M", [(61, 29), (47, 38), (88, 87), (680, 9), (253, 509), (393, 328)])
@pytest.mark.parametrize("pinned", [False, True])
def test_round_trip(hyd, N, M, pinned):
    import torch
    with hyd.Simulation(S.make_channel(N=N, M=M, seed=4), precision=hyd.FP32) as sim:
        a = torch.empty(sim.shape, dtype=torch.float64)
        out = torch.empty(sim.shape, dtype=torch.float64)
        if pinned:
            a, out = a.pin_memory(), out.pin_memory()
        a, out = a.numpy(), out.numpy()
        a[:] = np.random.default_rng(N).standard_normal(sim.shape) * 1e3
        a[2, 3:6] = [np.inf, -np.inf, np.nan]
        for f in ("u", "FS"):
            sim.upload(f, a)
            sim.download(f, out=out)
            np.testing.assert_array_equal(out, a.astype(np.float32).astype(np.float64))
