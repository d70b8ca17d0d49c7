"""The sweeps' solvers at the edges of what each takes, and the segment scan's
one-launch and skipped forms.

Meshes: rows of one to sixteen warps a row and columns of four to sixteen
warps a group, the last column group ragged, columns one cell below and above
the staged solver's limit (1100 cells), rows beyond the staged solver's in
every form, islands that leave several segments in rows and columns, more columns than rows (the reference's y sweep writes
columns up to N only). From the oracle's state after 8 steps one step on each
agrees to 1e-10 of a field's magnitude in FP64, to 1e-4 in the FP32 forms
(the bounds of the parity tests)."""
import numpy as np
import pytest

from hydist_c_b200 import scenario as S

STATE = ["u", "v", "z", "t_u", "t_v", "t_z", "H_moi", "Htdu", "Htdv", "FS", "tFS"]
MESHES = [(9, 8), (33, 30), (66, 34), (131, 67), (162, 161), (259, 353), (354, 64), (520, 1155),
          (1101, 41), (1102, 41), (2307, 24), (20, 18200)]


def _mesh(N, M):
    b = S.make_channel(N=N, M=M, seed=77 + N, dx=10.0, sediment=True, sediment_start=0.0, n_bumps=3,
                       inflow=0.5 * M * 10)
    h = b["scenario"]["h"]
    h[h > 0] += 2.0
    if N > 60:
        for q in range(3):
            i, j = N * (q + 1) // 4, M // 3 + 3 * q
            h[i:i + N // 20, j:j + M // 8 + 2] = 0.0
    return b


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["FP64", "FP32", "FP32_REFINE"])
@pytest.mark.parametrize("mesh", MESHES)
def test_one_step_matches_oracle(hyd, oracle_mod, mesh, form):
    b = _mesh(*mesh)
    orc = oracle_mod.OracleSim(b, nthreads=8)
    orc.step(8)
    sim = hyd.Simulation(b, precision=getattr(hyd, form))
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


def _shelf(N, M):
    """A basin with a shelf whose shallowest patches dry in the first step and
    are wetted in the second (by the oracle: 430 cells)."""
    b = S.make_channel(N=N, M=M, seed=5, dx=10.0, n_bumps=0, inflow=0.2 * M * 10)
    h, z = b["scenario"]["h"], np.zeros((N + 3, M + 3))
    h[h > 0] = 3.0
    i, j = np.arange(N + 3)[:, None], np.arange(M + 3)[None, :]
    shelf = (i > N // 4) & (i < 3 * N // 4) & (j > M // 3) & (j < 2 * M // 3)
    h[shelf] = 0.25
    z += -0.224 + 0.008 * np.sin(2 * np.pi * i / 40) * np.cos(2 * np.pi * j / 25)
    b["scenario"]["z0"] = z
    return b


@pytest.mark.gpu
@pytest.mark.parametrize("mesh", [(256, 100), (258, 100)])
def test_drying_rebuilds_the_tables(hyd, oracle_mod, mesh):
    """Cells dry and are wetted: on a mesh scanned in one launch and on
    one scanned in two, the mask follows the oracle's step by step from the
    oracle's state (so a table left as it was would show in the next step),
    and away from the fronts the level does too."""
    b = _shelf(*mesh)
    orc, sim = oracle_mod.OracleSim(b, nthreads=8), hyd.Simulation(b)
    dried = 0
    for _ in range(12):
        orc.step(1)
        sim.step(1)
        sim.sync()
        k = orc.get("khouot")
        assert np.array_equal(sim.download("khouot"), k)
        dried = max(dried, int((k == 1).sum()))
        near = k != 0
        for _ in range(4):
            near = near | np.roll(near, 1, 0) | np.roll(near, -1, 0) | np.roll(near, 1, 1) | np.roll(near, -1, 1)
        z, zo = sim.download("z"), orc.get("z")
        assert np.abs(z - zo)[~near].max() <= 1e-6
        for f in STATE:  # (the mask is not uploaded: that would rescan)
            sim.upload(f, orc.get(f))
    assert dried > 20


def _runs_by_words(wet, lim):
    """k_runs_lines: the line's wet cells as 32-bit words, a run's start and
    end by the neighbouring bits, numbered by bit counts."""
    n = 8
    words = [sum(int(wet(2 + 32 * w + b)) << b for b in range(32) if 2 + 32 * w + b <= lim) for w in range(n)] + [0]
    w2, w1 = lim >= 4 and wet(lim - 2), lim >= 3 and wet(lim - 1)
    dau, cuoi = [], []
    for w in range(n):
        for lane in range(32):
            p = 2 + 32 * w + lane
            is_ = words[w] >> lane & 1
            before = words[w] >> (lane - 1) & 1 if lane else (words[w - 1] >> 31 if w else 0)
            after = words[w] >> (lane + 1) & 1 if lane < 31 else words[w + 1] & 1
            if is_ and not before and p <= lim - 2:
                dau.append(p)
            if is_ and not after and (p != lim - 1 or w2) and (p != lim or (w1 and w2)):
                cuoi.append(p)
    return dau, cuoi


def test_words_give_the_reference_runs():
    from test_scan import scan_reference
    rng = np.random.default_rng(9)
    for trial in range(1500):
        lim = int(rng.choice([4, 5, 6, 7, 32, 33, 34, 65, 66, 200, 256, 257]))
        K = np.where(rng.random(lim + 3) < rng.choice([0.05, 0.3, 0.6]), 1, 0)
        got = _runs_by_words(lambda p: K[p] == 0, lim)
        assert got == tuple(scan_reference(K, lim)), (lim, K)
