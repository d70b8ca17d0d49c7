"""The x sweeps where the column groups just fill, just exceed and more than twice
exceed one round of CTAs (148 SMs: 592 and 1184 columns in groups of four), at and
above the lengths from which a part of a second round goes to the chunked solver
(640 cells, refined 850): one step from the oracle's state, and batched members as alone on
both sides of the second round's end."""
import numpy as np
import pytest

from hydist_c_b200 import scenario as S

STATE = ["u", "v", "z", "t_u", "t_v", "t_z", "H_moi", "Htdu", "Htdv", "FS", "tFS"]


def _mesh(N, M, seed=5):
    b = S.make_channel(N=N, M=M, seed=seed, dx=10.0, sediment=True, sediment_start=0.0, n_bumps=2,
                       inflow=0.5 * M * 10)
    h = b["scenario"]["h"]
    h[h > 0] += 2.0
    for q in range(3):
        h[N * (q + 1) // 4:N * (q + 1) // 4 + 6, M // 3 + 3 * q:M // 3 + 3 * q + 9] = 0.0
    return b


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["FP64", "FP32", "FP32_REFINE"])
@pytest.mark.parametrize("mesh", [(641, 600), (642, 593), (642, 594), (642, 595), (642, 596), (700, 1190),
                                  (851, 600), (852, 595), (852, 596)])
def test_one_step_matches_oracle(hyd, oracle_mod, mesh, form):
    b = _mesh(*mesh)
    orc = oracle_mod.OracleSim(b, nthreads=8)
    orc.step(3)
    with hyd.Simulation(b, precision=getattr(hyd, form)) as sim:
        for f in STATE:
            sim.upload(f, orc.get(f))
        sim.upload("khouot", orc.get("khouot"))
        sim.t = orc.t
        orc.step(1)
        sim.step(1)
        sim.sync()
        tol = 1e-10 if form == "FP64" else 1e-4
        for f in ("u", "v", "z", "t_u", "t_v", "t_z", "FS"):
            a, r = sim.download(f), orc.get(f)
            assert np.abs(a - r).max() <= tol * max(np.abs(r).max(), 1e-300), f


# 2 x 75 groups (a part of a second round) and 4 x 75 (more than two)
@pytest.mark.gpu
@pytest.mark.parametrize("form", ["FP64", "FP32_REFINE"])
@pytest.mark.parametrize("members", [2, 4])
def test_members_as_alone(hyd, form, members):
    prec, rtol = getattr(hyd, form), 1e-11 if form == "FP64" else 1e-4
    alone = []
    for k in range(members):
        with hyd.Simulation(_mesh(870, 300, 5 + k), precision=prec) as sim:
            sim.step(4)
            alone.append({f: sim.download(f) for f in ("u", "v", "z", "FS")})
    sims = [hyd.Simulation(_mesh(870, 300, 5 + k), precision=prec) for k in range(members)]
    ens = hyd.Ensemble(sims)
    ens.step(4)
    ens.sync()
    for k, sim in enumerate(sims):
        for f, ref in alone[k].items():
            assert np.linalg.norm(sim.download(f) - ref) <= rtol * np.linalg.norm(ref), (k, f)
    ens.close()
    for s in sims:
        s.close()
