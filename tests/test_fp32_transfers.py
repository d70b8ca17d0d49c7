"""Host transfers of the FP32 form's fields, converted on the device: every
value that FP32 holds comes back as it went, others rounded to the nearest
FP32, infinities and NaN kept, on sizes around the conversion's blocks; and a
transfer between half-steps leaves the step's result as it is."""
import numpy as np
import pytest

from hydist_c_b200 import scenario as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,M", [(8, 8), (29, 29), (64, 32), (130, 61)])
def test_round_trip(hyd, N, M):
    sim = hyd.Simulation(S.make_channel(N=N, M=M, seed=4, inflow=20.0), precision=hyd.FP32)
    rng = np.random.default_rng(N)
    a = rng.standard_normal(sim.shape) * 10.0 ** rng.integers(-30, 30, sim.shape)
    a[1, 1:5] = [np.inf, -np.inf, np.nan, 1e300]
    for f in ("u", "FS", "Kx"):
        sim.upload(f, a)
        with np.errstate(over="ignore"):
            want = a.astype(np.float32).astype(np.float64)
        np.testing.assert_array_equal(sim.download(f), want)


def test_transfer_between_half_steps(hyd):
    b = S.make_channel(N=64, M=32, seed=5, sediment=True, sediment_start=0.0)
    one, two = hyd.Simulation(b, precision=hyd.FP32), hyd.Simulation(b, precision=hyd.FP32)
    for _ in range(3):
        for half in (0, 1):
            one.half_step(half)
            two.half_step(half)
            two.upload("u", two.download("u"))
            two.upload("FS", two.download("FS"))
    for f in ("u", "v", "z", "FS", "tFS"):
        np.testing.assert_array_equal(one.download(f), two.download(f))
