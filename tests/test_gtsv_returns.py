"""Batches of short systems return once they are enqueued, however many they are;
a named solver is the one that runs."""
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

from hydist_c_b200 import capi

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]


def _batch(lens, seed, dtype):
    import torch
    from hydist_c_b200 import scenario as S
    a, d, c, b, off, ln = S.tridiag_batch(lengths=np.array(lens), seed=seed)
    dt = getattr(torch, dtype)
    return [torch.from_numpy(v).cuda().to(dt) for v in (a, d, c, b)], torch.from_numpy(off).cuda(), \
        torch.from_numpy(ln).cuda()


def _returns_early(hyd, dtype, algo):
    """60000 systems of 500 rows (30 M rows, 1.2 GB in FP64): hundreds of
    microseconds of solving, enqueued in a few."""
    import torch
    t, off, ln = _batch(np.full(60000, 500), 7, dtype)
    x = torch.empty_like(t[1])
    st = torch.cuda.current_stream()
    hyd.gtsv_batched(*t, off, ln, algo=algo, x=x)
    torch.cuda.synchronize()
    running = 0
    for _ in range(5):
        hyd.gtsv_batched(*t, off, ln, algo=algo, x=x)
        running += not st.query()
        torch.cuda.synchronize()
    assert running >= 4


@pytest.mark.parametrize("dtype", ["float64", "float32"])
def test_short_batch_returns_before_it_is_solved(hyd, dtype):
    _returns_early(hyd, dtype, capi.GTSV_WARP)


@pytest.mark.parametrize("dtype", ["float64", "float32"])
def test_short_untuned_batch_returns_before_it_is_solved(dtype):
    """AUTO before any tuning, so in a process of its own (the autotuner's table
    is the process's)."""
    r = subprocess.run([sys.executable, "-c", "import hydist_c_b200 as H, test_gtsv_returns as T\n"
                        f"T._returns_early(H, {dtype!r}, 0)\nprint('all well')"],
                       cwd=ROOT, env=dict(os.environ, PYTHONPATH=f"{ROOT}:{ROOT / 'tests'}"),
                       capture_output=True, text=True, timeout=300)
    assert "all well" in r.stdout, r.stdout + r.stderr


@pytest.mark.parametrize("dtype", ["float64", "float32"])
def test_named_warp_solver_beside_long_systems(hyd, dtype):
    """The short systems of a WARP batch come out bit for bit the same with
    a longer system in the batch as without one."""
    import torch
    short = [17, 33, 100, 128, 129, 250, 256, 257, 400, 512] * 90
    t, off, ln = _batch(short + [900], 8, dtype)
    n = int(off[-1])
    alone = hyd.gtsv_batched(*[v[:n].clone() for v in t], off[:-1].clone(), ln[:-1].clone(),
                             algo=capi.GTSV_WARP)
    both = hyd.gtsv_batched(*t, off, ln, algo=capi.GTSV_WARP)
    torch.cuda.synchronize()
    assert torch.equal(both[:n], alone)
