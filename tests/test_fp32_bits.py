"""The FP32 forms' u, v and z, bit for bit: their hydraulic rows and the order of
operations stay, down to which products and sums are contracted (csrc/pairgen.cuh says
why). The inputs take basic arithmetic only, the same on every host; the digests
are those of the interleaved sweeps as they first were. Meshes for each number of
chunks a line can have, alone and batched."""
import hashlib

import numpy as np
import pytest

from hydist_c_b200 import scenario as S

DIGESTS = {
    "9x8-1-FP32": "36ab766e237dfd76", "9x8-1-FP32_REFINE": "1f11a02334a73b60",
    "40x39-1-FP32": "cee5b7b250187850", "40x39-1-FP32_REFINE": "d35b0b2b9f569803",
    "66x34-1-FP32": "01062cedf21cee8d", "66x34-1-FP32_REFINE": "077b9da0f60f575d",
    "130x70-1-FP32": "3e1bcdcec99ce020", "130x70-1-FP32_REFINE": "df3f44bf49f27561",
    "260x131-1-FP32": "4679b34a0b0d6663", "260x131-1-FP32_REFINE": "c9e53556ba4d1e6e",
    "464x324-1-FP32": "9894ad5c97c1e2fc", "464x324-1-FP32_REFINE": "e5b6fb4ca059849d",
    "600x520-1-FP32": "939a104d82cdc95a", "600x520-1-FP32_REFINE": "4fed3c1992156ac5",
    "1201x61-1-FP32": "c77e9abe038babbd", "1201x61-1-FP32_REFINE": "c170323c2997c4a5",
    "40x39-5-FP32": "ac231a7b2581f6a6", "40x39-5-FP32_REFINE": "e57c03fcd33efba6",
    "133x133-3-FP32": "870640c1ca9cef0f", "133x133-3-FP32_REFINE": "0c20798e35d24771",
    "256x128-4-FP32": "44bf799ba3641d13", "256x128-4-FP32_REFINE": "85a86ec1f9373d85",
    "300x260-3-FP32": "c68927104435a4f9", "300x260-3-FP32_REFINE": "a0c253fd17f15203",
    "600x520-2-FP32": "fd4f9379cafd5c7e", "600x520-2-FP32_REFINE": "7f4349814ea7a7cf",
}


def channel(N, M, k=0):
    b = S.make_channel(N=N, M=M, seed=60 + k, dx=8.0, dt=2.0, hours=1, inflow=4.0 * M, tide_amp=0.0,
                       n_bumps=0, sediment=True, sediment_start=0.0, fw=(0.005, 0.07))
    sc = b["scenario"]
    i, j = np.arange(N + 3)[:, None], np.arange(M + 3)[None, :]
    sc["h"] = np.where(sc["h"] > 0, 4.0 + ((3 * i + 5 * j + k) % 17) * 0.0625, 0.0)
    if N > 60:  # an island: two segments a line
        sc["h"][N // 2:N // 2 + 5, M // 2:M // 2 + 4] = 0.0
    sc["z0"] = ((7 * i + 11 * j + k) % 31 - 15) * 0.00390625 + 0.0 * j
    sc["bc_right"] = 0.03125 * np.arange(len(sc["bc_right"]))
    return b


def digest(H, N, M, members, form):
    sims = [H.Simulation(channel(N, M, k), precision=getattr(H, form)) for k in range(members)]
    if members > 1:
        ens = H.Ensemble(sims)
        ens.step(12)
        ens.close()
    else:
        sims[0].step_graph(12)
    h = hashlib.sha256()
    for s in sims:
        for f in ("u", "v", "z"):
            a = s.download(f)
            assert np.isfinite(a).all() and np.abs(a).max() > 1e-3
            h.update(a.tobytes())
        s.close()
    return h.hexdigest()[:16]


CASES = [(9, 8, 1), (40, 39, 1), (66, 34, 1), (130, 70, 1), (260, 131, 1), (464, 324, 1), (600, 520, 1),
         (1201, 61, 1), (40, 39, 5), (133, 133, 3), (256, 128, 4), (300, 260, 3), (600, 520, 2)]


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["FP32", "FP32_REFINE"])
@pytest.mark.parametrize("case", CASES, ids=lambda c: "%dx%d-%d" % c)
def test_bits(hyd, case, form):
    assert digest(hyd, *case, form) == DIGESTS["%dx%d-%d-%s" % (*case, form)]
