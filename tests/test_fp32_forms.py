"""The FP32 forms' hydraulic sweeps keep their rows and order of operations.

Beside a dry cell the momentum rows switch a one-sided second difference on by
the sign of the cross velocity, so a rounding that turns the sign of a nearly
vanishing cross velocity moves a cell by 1e-3 of the velocities' scale. In these
channels such a cell is met within 10 or 20 steps, and sweeps that rounded
otherwise (velocities alone, solved for their changes, in staged lines) parted
there from the FP64 form by 9.5e-4 to 9e-3 of the scale."""
import numpy as np
import pytest

from hydist_c_b200 import scenario as S

pytestmark = pytest.mark.gpu

N, M = 128, 48


def channel(seed):
    """A flat-bedded channel with long waves in its initial level."""
    b = S.make_channel(N=N, M=M, seed=seed, dx=5.0, dt=2.0, hours=1, inflow=0.6 * M * 5.0,
                       tide_amp=0.3, n_bumps=0)
    sc = b["scenario"]
    rng = np.random.default_rng(seed)
    sc["h"] = np.where(sc["h"] > 0, 4.0, 0.0)
    i, j = np.arange(N + 3.0)[:, None], np.arange(M + 3.0)[None, :]
    z = np.zeros((N + 3, M + 3))
    for _ in range(3):
        a, k, l, p = rng.uniform(0.02, 0.08), *rng.uniform(-0.3, 0.3, 2), rng.uniform(0, 6.28)
        z = z + a * np.cos(k * i + l * j + p)
    sc["z0"] = z
    return b


# 1e-5 is ten times the largest rounding error of 20 steps (an ulp of FP32 is
# 1.2e-7, a sweep rounds some ten times along a row), a hundredth of a jump
@pytest.mark.parametrize("form,seed,steps", [("FP32", 2895, 10), ("FP32", 6291, 20),
                                             ("FP32", 10548, 20), ("FP32_REFINE", 3950, 10),
                                             ("FP32_REFINE", 10548, 20)])
def test_no_jump_beside_the_banks(hyd, form, seed, steps):
    got = []
    for precision in (hyd.FP64, getattr(hyd, form)):
        sims = [hyd.Simulation(channel(seed), precision=precision) for _ in range(2)]
        ens = hyd.Ensemble(sims)
        ens.step(steps)
        got.append([sims[0].download(f) for f in ("u", "v", "z")])
        ens.close()
        for s in sims:
            s.close()
    for f, want, have in zip(("u", "v", "z"), *got):
        scale = np.maximum(np.sqrt(np.mean(want ** 2)), np.abs(want))
        off = np.abs(have - want) / scale
        assert off.max() <= 1e-5, (f, off.max(), np.unravel_index(off.argmax(), off.shape))
