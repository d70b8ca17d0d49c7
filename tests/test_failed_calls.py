"""Host calls of the CUDA runtime that fail (a preloaded fake returns the error
code; no GPU work is involved): what the library makes of them."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    so = tmp_path_factory.mktemp("shim") / "fail_calls.so"
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-o", str(so),
                    str(ROOT / "tests" / "native" / "fail_calls.c"), "-ldl"], check=True)
    return so


def _child(shim, call, code):
    env = dict(os.environ, LD_PRELOAD=str(shim), FAIL_CALL=call, PYTHONPATH=str(ROOT))
    head = f"import ctypes\nfail = ctypes.CDLL({str(shim)!r})\n"
    r = subprocess.run([sys.executable, "-c", head + code], env=env, cwd=ROOT, capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "all well" in r.stdout


@pytest.mark.gpu
def test_step_launches_where_its_graph_cannot_be_made(shim):
    """hydist_step of eight steps and more goes on launch by launch, with the
    same result; hydist_step_graph, which promises the graph, reports it."""
    _child(shim, "cudaGraphInstantiate", """
import numpy as np
import hydist_c_b200 as H
from hydist_c_b200 import scenario as S
b = S.make_channel(N=40, M=33, seed=11, dx=10.0, inflow=5.0 * 33)
a, c = H.Simulation(b), H.Simulation(b)
for _ in range(20):
    a.half_step(0); a.half_step(1)
a.sync()
fail.fail_calls_left(1 << 20)
c.step(12)
for _ in range(7):
    c.step(1)
assert fail.fail_calls_failed() >= 1
n = fail.fail_calls_failed()
try:
    c.step_graph(1)
    raise SystemExit("no error")
except H.HydistError:
    pass
assert fail.fail_calls_failed() == n + 1
c.step(1)
c.sync()
assert c.t == a.t, (c.t, a.t)
for f in ("u", "v", "z"):
    assert np.array_equal(a.download(f), c.download(f)), f
fail.fail_calls_left(0)
c.step_graph(2)
c.sync()
print("all well")
""")


@pytest.mark.gpu
def test_batched_solver_after_a_failed_allocation(shim):
    """A first batch whose counts' host memory could not be had reports that;
    the next batch asks again and is solved."""
    _child(shim, "cudaHostAlloc", """
import numpy as np, torch
import hydist_c_b200 as H
from hydist_c_b200 import scenario as S
*rows, off, ln = S.tridiag_batch(lengths=np.array([5, 300, 900, 7000]), seed=3)
t = [torch.from_numpy(v).cuda() for v in rows]
off, ln = torch.from_numpy(off).cuda(), torch.from_numpy(ln).cuda()
fail.fail_calls_left(1)
try:
    H.gtsv_batched(*t, off, ln)
    raise SystemExit("no error")
except H.HydistError:
    pass
assert fail.fail_calls_failed() == 1
x = H.gtsv_batched(*t, off, ln)
a, d, c, b = t
r = d * x - b
for s in range(4):
    o, n = int(off[s]), int(ln[s])
    r[o + 1:o + n] += a[o + 1:o + n] * x[o:o + n - 1]
    r[o:o + n - 1] += c[o:o + n - 1] * x[o + 1:o + n]
assert float(r.abs().max()) < 1e-13 * float(b.abs().max().clamp(min=1)), float(r.abs().max())
print("all well")
""")


@pytest.mark.gpu
def test_batch_after_one_that_failed_halfway(shim):
    """A batch that fails with some of its classes launched: the next one, on
    another stream, waits for those before it uses the scratch again."""
    _child(shim, "cudaStreamWaitEvent", """
import numpy as np, torch
import hydist_c_b200 as H
from hydist_c_b200 import scenario as S
def batch(lens, seed):
    *rows, off, ln = S.tridiag_batch(lengths=np.array(lens), seed=seed)
    return [torch.from_numpy(v).cuda() for v in rows] + [torch.from_numpy(off).cuda(), torch.from_numpy(ln).cuda()]
one, two = batch([7000] * 300 + [900] * 400 + [300] * 400, 3), batch([40] * 5000 + [700] * 900, 4)
want = H.gtsv_batched(*two).clone()
st = [torch.cuda.Stream(), torch.cuda.Stream()]
torch.cuda.synchronize()
for _ in range(4):
    x = torch.full_like(want, float("nan"))
    torch.cuda.synchronize()
    # calls: the earlier batch, then the fork and the join of each class
    fail.fail_calls_after(3)
    n = fail.fail_calls_failed()
    try:
        with torch.cuda.stream(st[0]):
            H.gtsv_batched(*one)
        raise SystemExit("no error")
    except H.HydistError:
        assert fail.fail_calls_failed() == n + 1
    with torch.cuda.stream(st[1]):
        H.gtsv_batched(*two, x=x)
    torch.cuda.synchronize()
    assert torch.equal(x, want)
print("all well")
""")
