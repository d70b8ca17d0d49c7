"""A step however it is launched (launch by launch, by a replayed graph, inside
a caller's capture; each kernel waiting for the one before or starting in its
tail, by the mesh's size), the shortest wet segments, and the diffusivity around
its bounds."""
import numpy as np
import pytest

from hydist_c_b200 import scenario as S

FIELDS = ("u", "v", "z", "FS", "dH", "khouot")


def _channel(N, M, **kw):
    b = S.make_channel(N=N, M=M, seed=11, dx=10.0, sediment=True, sediment_start=8.0, inflow=5.0 * M,
                       **kw)
    b["options"]["bed_change"] = 1
    b["options"]["bed_change_start"] = 16.0
    return b


def _launches(sim, n):  # the two half-steps launch by launch
    for _ in range(n):
        sim.half_step(0)
        sim.half_step(1)


def _single(sim, n):  # by launches first, then by graphs
    for _ in range(n):
        sim.step(1)


WAYS = {"calls": lambda s: s.step(30), "graph": lambda s: s.step_graph(30),
        "single": lambda s: _single(s, 30),
        "mixed": lambda s: (s.step(3), _launches(s, 4), s.step(12), s.step_graph(2), _single(s, 9))}


# 40x33: kernels that start in the tail of the one before; 1100x1000: above the
# size up to which they do
@pytest.mark.gpu
@pytest.mark.parametrize("form", ["FP64", "FP32"])
@pytest.mark.parametrize("mesh", [(40, 33), (1100, 1000)])
def test_ways_to_step_agree_to_the_bit(hyd, mesh, form):
    """30 steps through the starts of sediment and bed change: the same kernels
    on the same values, so the same bits."""
    b = _channel(*mesh)
    sim = hyd.Simulation(b, precision=getattr(hyd, form))
    _launches(sim, 30)
    sim.sync()
    ref, t = {f: sim.download(f) for f in FIELDS}, sim.t
    assert np.isfinite(ref["u"]).all() and np.abs(ref["u"]).max() > 1e-3 and np.abs(ref["dH"]).max() > 0
    for name, way in WAYS.items():
        s = hyd.Simulation(b, precision=getattr(hyd, form))
        way(s)
        s.sync()
        assert s.t == t
        for f in FIELDS:
            assert np.array_equal(s.download(f), ref[f]), (name, f)


@pytest.mark.gpu
def test_step_inside_a_callers_capture(hyd):
    """Steps captured on the handle's stream after a copy and a kernel of the
    caller's; the replay gives what the steps give."""
    import torch
    b = _channel(40, 33)
    ref, sim = hyd.Simulation(b), hyd.Simulation(b)
    ref.step(40)
    ref.sync()
    st = torch.cuda.ExternalStream(sim.stream)
    src, dst = torch.ones(1000, device="cuda"), torch.zeros(1000, device="cuda")
    sim.step(37)
    sim.sync()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st):
        dst.copy_(src)
        dst.mul_(2)
        sim.step(3)
        dst.add_(1)
    with torch.cuda.stream(st):
        g.replay()
    torch.cuda.synchronize()
    assert sim.t == ref.t and bool((dst == 3).all())
    for f in FIELDS:
        assert np.array_equal(sim.download(f), ref.download(f)), f


def _short_runs(N=60, M=56):
    """Pairs of islands that leave runs of two and three wet cells between them,
    in rows and in columns, and runs as short at both banks."""
    b = S.make_channel(N=N, M=M, seed=3, dx=10.0, sediment=True, sediment_start=0.0, n_bumps=0,
                       inflow=0.5 * M * 10)
    h = b["scenario"]["h"]
    h[h > 0] += 2.0
    for k, gap in enumerate((2, 3, 4)):
        for q in range(2):
            r = 10 + 12 * k + 6 * q
            for j in (14 + 8 * k, 14 + 8 * k + gap):
                h[r - 1:r + 2, j - 1:j + 1] = 0
            for i in (10 + 12 * k, 10 + 12 * k + gap):
                h[i - 1:i + 1, 39 + 6 * q:42 + 6 * q] = 0
        h[13 + 12 * k:16 + 12 * k, 3 + k:5 + k] = 0
        h[13 + 12 * k:16 + 12 * k, M - 3 - k:M - 1 - k] = 0
    return b


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["FP64", "FP32", "FP32_REFINE"])
def test_short_segments_match_oracle(hyd, oracle_mod, form):
    """Bounds as in the other one-step comparisons: 1e-10 of a field's magnitude
    in FP64, 1e-4 in the FP32 forms."""
    b = _short_runs()
    orc, sim = oracle_mod.OracleSim(b), hyd.Simulation(b, precision=getattr(hyd, form))
    orc.step(5)
    for kind in (0, 1):
        first, last, n = orc.segments(kind)
        lens = [last[i, k] - first[i, k] + 1 for i in range(len(n)) for k in range(n[i])]
        assert lens.count(2) >= 4 and lens.count(3) >= 4
    for f in ("u", "v", "z", "t_u", "t_v", "t_z", "H_moi", "Htdu", "Htdv", "FS", "tFS"):
        sim.upload(f, orc.get(f))
    sim.upload("khouot", orc.get("khouot"))
    sim.t = orc.t
    orc.step(1)
    sim.step(1)
    sim.sync()
    tol = 1e-10 if form == "FP64" else 1e-4
    for f in ("u", "v", "z", "t_u", "t_v", "t_z", "FS"):
        a, r = sim.download(f), orc.get(f)
        assert np.isfinite(r).all() and np.abs(a - r).max() <= tol * np.abs(r).max(), f


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["FP64", "FP32"])
@pytest.mark.parametrize("Ks", [1.0, 30.0, 50.0, 60.0, 90.0])
def test_diffusivity_around_its_bounds(hyd, oracle_mod, Ks, form):
    """Roughness heights that put the quotient on both sides of 5 and 100 and
    the logarithm's argument on both sides of 1. A value below 100 has a
    logarithm above 0.03, which amplifies a rounding of its argument by at most
    33: with the velocities of one step, 1e-9 in FP64, 1e-3 in FP32."""
    b = S.make_channel(N=90, M=70, seed=3, dx=10.0, sediment=True, sediment_start=0.0, n_bumps=4,
                       inflow=6 * 70 * 10)
    h = b["scenario"]["h"]
    h[h > 0] += 2
    b["params"]["Ks"] = Ks
    orc, sim = oracle_mod.OracleSim(b), hyd.Simulation(b, precision=getattr(hyd, form))
    orc.step(40)
    for f in ("u", "v", "z", "t_u", "t_v", "t_z", "H_moi", "Htdu", "Htdv", "FS", "tFS", "Kx", "Ky"):
        sim.upload(f, orc.get(f))
    sim.upload("khouot", orc.get("khouot"))
    sim.t = orc.t
    orc.step(1)
    sim.step(1)
    sim.sync()
    for f in ("Kx", "Ky"):
        a, r = sim.download(f), orc.get(f)
        if Ks > 40 and f == "Kx":
            assert ((r > 5) & (r < 5.2)).sum() >= 5 and (r == 5).any() and (r == 100).any()
        assert np.abs(a - r).max() <= (1e-9 if form == "FP64" else 1e-3) * 100, f
