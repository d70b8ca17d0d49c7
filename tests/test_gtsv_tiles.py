"""The batched solver's paths for long systems (tiles of 2304 rows) and its
length classes: every way a system can end in its last tile, the edges of the
classes' shared memory, many tiles, alone and beside short systems, and
offsets of both alignments, against the oracle's FP64 Thomas.

Tolerances: the systems have |d| >= |a| + |c| + 0.1 with |a|, |c| <= 1, so a
row's condition is at most 21: a few tens of roundings of a value of order
one, 1e-14 in FP64 and 5e-6 in FP32."""
import numpy as np
import pytest

from hydist_c_b200 import capi

T = 2304
CASES = {
    "last tile joined": [3 * T + 1], "last tile of two": [3 * T + 2], "whole tiles": [3 * T],
    "one short of it": [3 * T - 1], "first above the classes": [6145], "many tiles": [200 * T + 17],
    "mixed": [6145, 3, 9000, 1, 4 * T + 1, 33, 5 * T + 2, 511, 7777],
    "class edges": [512, 513, 1024, 1025, 1536, 1537, 2048, 2049, 3072, 3073, 4096, 4097, 6144],
}


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["float64", "float32"])
@pytest.mark.parametrize("name", CASES)
def test_long_systems_match_oracle(hyd, oracle_mod, name, dtype):
    import torch
    from hydist_c_b200 import scenario as S
    a, d, c, b, off, ln = S.tridiag_batch(lengths=np.array(CASES[name]), seed=31)
    ref = oracle_mod.thomas_batched(a, d, c, b, off, ln)
    t = [torch.from_numpy(v).cuda().to(getattr(torch, dtype)) for v in (a, d, c, b)]
    for algo in (capi.GTSV_AUTO, capi.GTSV_PARTITION, capi.GTSV_THOMAS):
        x = torch.full_like(t[1], float("nan"))
        hyd.gtsv_batched(*t, torch.from_numpy(off), torch.from_numpy(ln), algo=algo, x=x)
        torch.cuda.synchronize()
        err = np.abs(x.double().cpu().numpy() - ref) / np.maximum(np.abs(ref), 1.0)
        assert np.isfinite(err).all() and err.max() <= (1e-14 if dtype == "float64" else 5e-6), err.max()


@pytest.mark.gpu
def test_batches_on_two_streams_share_the_scratch(hyd, oracle_mod):
    """Batches queued one after another on two streams, with no wait between:
    the second call reuses the first one's lists and tile values only after
    the first batch is done."""
    import torch
    from hydist_c_b200 import scenario as S
    st = [torch.cuda.Stream(), torch.cuda.Stream()]
    work = []
    for k in range(6):
        lens = np.full(2000, 40 + 60 * k) if k % 2 else np.full(8, 7000 + 900 * k)
        a, d, c, b, off, ln = S.tridiag_batch(lengths=lens, seed=50 + k)
        work.append(([torch.from_numpy(v).cuda() for v in (a, d, c, b)], torch.from_numpy(off).cuda(),
                     torch.from_numpy(ln).cuda(), oracle_mod.thomas_batched(a, d, c, b, off, ln)))
    torch.cuda.synchronize()
    xs = []
    for k, (t, off, ln, _) in enumerate(work):
        with torch.cuda.stream(st[k % 2]):
            xs.append(hyd.gtsv_batched(*t, off, ln))
    torch.cuda.synchronize()
    for x, w in zip(xs, work):
        assert np.abs(x.cpu().numpy() - w[3]).max() <= 1e-13 * max(1.0, np.abs(w[3]).max())


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["float64", "float32"])
@pytest.mark.parametrize("shift", [0, 1])
def test_many_short_systems_beside_a_long_one(hyd, oracle_mod, dtype, shift):
    """Short systems staged by bulk copies (more of them than one wave of
    warps, and a longer system in the batch), at the classes' edges, from
    offsets of every alignment; with arrays that are not 16-byte aligned the
    warps' own copies. Rows around the systems stay as they were."""
    import torch
    from hydist_c_b200 import scenario as S
    edges = [1, 2, 3, 31, 32, 33, 34, 65, 95, 127, 128, 129, 191, 255, 256, 257, 320, 511, 512]
    a, d, c, b, off, ln = S.tridiag_batch(lengths=np.array(edges * 40 + [600]), seed=77)
    ref = oracle_mod.thomas_batched(a, d, c, b, off, ln)
    dt = getattr(torch, dtype)

    def place(v):
        t = torch.full((len(v) + 2,), float("nan"), dtype=dt, device="cuda")
        t[shift:shift + len(v)] = torch.from_numpy(v).to(dt).cuda()
        return t[shift:shift + len(v)]

    t = [place(v) for v in (a, d, c, b)]
    full = torch.full((len(b) + 8,), float("nan"), dtype=dt, device="cuda")
    x = full[4:4 + len(b)]
    hyd.gtsv_batched(*t, torch.from_numpy(off), torch.from_numpy(ln), x=x)
    torch.cuda.synchronize()
    assert torch.isnan(full[:4]).all() and torch.isnan(full[-4:]).all()
    err = np.abs(x.double().cpu().numpy() - ref) / np.maximum(np.abs(ref), 1.0)
    assert np.isfinite(err).all() and err.max() <= (1e-14 if dtype == "float64" else 5e-6), err.max()
