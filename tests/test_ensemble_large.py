"""Batched members whose launches the small ensembles do not reach: columns
beyond the staged solver's limit (the chunked solver's line groups of several
members on one scratch, k_fs_rows), the last column group ragged, and more
cells in all than dependent launches take. Each member against the same scenario
alone, in the 2-norm: beside a bank a rounding can move a single cell of the FP32
forms by 1e-3 (pairgen.cuh)."""
import numpy as np
import pytest

from hydist_c_b200 import scenario as S

RTOL = {"FP64": 1e-11, "FP32": 1e-4, "FP32_REFINE": 1e-4}


def _member(N, M, k):
    b = S.make_channel(N=N, M=M, seed=900 + k, dx=10.0, dt=2.0, hours=1.0, sediment=True,
                       sediment_start=0.0, n_bumps=2, inflow=(3.0 + k) * M)
    h = b["scenario"]["h"]
    h[h > 0] += 2.0
    h[N // 2:N // 2 + 9, M // 3 + k:M // 3 + 8 + k] = 0.0  # an island, elsewhere in each member
    b["options"]["bed_change"] = 1
    return b


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["FP64", "FP32", "FP32_REFINE"])
@pytest.mark.parametrize("mesh", [(1201, 61), (700, 520), (1300, 421)])
def test_members_as_alone(hyd, mesh, form):
    prec, fields = getattr(hyd, form), ("u", "v", "z", "FS", "dH")
    alone = []
    for k in range(3):
        with hyd.Simulation(_member(*mesh, k), precision=prec) as sim:
            sim.step(6)
            alone.append({f: sim.download(f) for f in fields})
    sims = [hyd.Simulation(_member(*mesh, k), precision=prec) for k in range(3)]
    ens = hyd.Ensemble(sims)
    ens.step(6)
    ens.sync()
    for k, sim in enumerate(sims):
        for f, ref in alone[k].items():
            off = np.linalg.norm(sim.download(f) - ref)
            # (the bed change is a small difference of fluxes: three digits less)
            assert off <= RTOL[form] * (1e3 if f == "dH" else 1) * np.linalg.norm(ref), (k, f)
    assert np.linalg.norm(alone[0]["u"] - alone[1]["u"]) > 1e-2 * np.linalg.norm(alone[0]["u"])
    ens.close()
    for s in sims:
        s.close()
