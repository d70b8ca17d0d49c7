"""Rows of 512 threads in the staged row solver, and its shared memory's limit.

Meshes of few rows: the narrowest and a wide row of 512 threads, and the last
row that one CTA's shared memory holds and the first that it does not in each form
(9344 cells FP64, 14016 FP32, 8009 refined: there the sweep hands over to the
chunked solver, and k_fs_rows is switched on). There the reference's y sweep
writes columns up to N only, so one mesh has as many rows as columns. From the
oracle's state one step agrees to 1e-10 of a field's magnitude in FP64, to 1e-4
in the FP32 forms (the bounds of the parity tests)."""
import numpy as np
import pytest

from hydist_c_b200 import scenario as S

STATE = ["u", "v", "z", "t_u", "t_v", "t_z", "H_moi", "Htdu", "Htdv", "FS", "tFS"]


def _one_step(hyd, oracle_mod, N, M, form, before):
    b = S.make_channel(N=N, M=M, seed=41 + M, dx=10.0, sediment=True, sediment_start=0.0, n_bumps=3,
                       inflow=0.5 * M * 10)
    h = b["scenario"]["h"]
    h[h > 0] += 2.0
    for q in range(1, 5):  # several segments a row
        h[N // 3:N // 3 + 4, q * M // 5:q * M // 5 + 7] = 0.0
    orc = oracle_mod.OracleSim(b, nthreads=8)
    orc.step(before)
    with hyd.Simulation(b, precision=getattr(hyd, form)) as sim:
        for f in STATE:
            sim.upload(f, orc.get(f))
        sim.upload("khouot", orc.get("khouot"))
        sim.t = orc.t
        orc.step(1)
        sim.step(1)
        sim.sync()
        tol = 1e-10 if form == "FP64" else 1e-4
        for f in ("u", "v", "z", "t_u", "t_v", "t_z", "FS", "tFS"):
            a, r = sim.download(f), orc.get(f)
            assert np.abs(a - r).max() <= tol * max(np.abs(r).max(), 1e-300), f


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["FP64", "FP32", "FP32_REFINE"])
@pytest.mark.parametrize("M", [2306, 2400, 5000, 8010, 8011, 9345, 9346, 14017, 14018])
def test_one_step_matches_oracle(hyd, oracle_mod, M, form):
    _one_step(hyd, oracle_mod, 20, M, form, 6)


@pytest.mark.gpu
def test_as_many_rows_as_columns(hyd, oracle_mod):
    _one_step(hyd, oracle_mod, 2404, 2402, "FP64", 1)
