"""The FP32 form's concentration keeps the accuracy of a solve with few chunks."""
import numpy as np
import pytest

from hydist_c_b200 import scenario as S

pytestmark = pytest.mark.gpu


def scenario(N, M, seed):
    b = S.make_channel(N=N, M=M, seed=seed, dx=5.0, dt=2.0, hours=1, inflow=3.0 * M,
                       tide_amp=0.3, fw=(0.005, 0.0755), sediment=True, sediment_start=0.0, n_bumps=0)
    i, j = np.arange(N + 3.0)[:, None], np.arange(M + 3.0)[None, :]
    sc = b["scenario"]
    sc["z0"] = 0.05 * np.cos(0.2 * i + 0.1 * j + seed)
    sc["FS0"] = sc["FS0"] * (1 + 0.4 * np.sin(6 * np.pi * i / N) * np.cos(2 * np.pi * j / M))
    return b


# the 2-norm of the error against FP64 over that of the field, after 20 steps, mean
# of four scenarios: lines of four chunks had 1.0e-7; a third more is allowed (a
# reduction over 7 to 16 chunks in FP32 gave 1.6e-7 to 1.9e-7)
@pytest.mark.parametrize("N,M,bound", [(64, 32, 1.35e-7)])
def test_error_against_fp64(hyd, N, M, bound):
    far = []
    for seed in range(4):
        f = []
        for p in (hyd.FP64, hyd.FP32):
            with hyd.Simulation(scenario(N, M, seed), precision=p) as s:
                s.step_graph(20)
                f.append(s.download("FS"))
        far.append(np.linalg.norm(f[1] - f[0]) / np.linalg.norm(f[0]))
    assert np.mean(far) <= bound, far
