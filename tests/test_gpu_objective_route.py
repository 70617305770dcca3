"""The FP64 objective on either side of the line between the targets a warp stages and those each lane loads for itself (by
textures, features and K), on planes whose last warp is partly filled: E against the C restatement, and which kernel ran."""
import ctypes as C

import numpy as np
import pytest
import torch
from torch.profiler import ProfilerActivity, profile

import oracle as O
from nntc_b200 import abi, materials
from nntc_b200.session import Session

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("textures,c0,c1,k,staged", [
    (2, 2, 2, 4, False), (3, 2, 4, 4, True), (3, 3, 3, 4, False), (3, 4, 4, 4, False), (3, 4, 1, 2, True), (3, 2, 3, 2, False),
    (3, 1, 1, 0, False), (4, 4, 4, 4, True), (4, 4, 4, 1, True), (4, 4, 3, 0, False), (5, 3, 4, 4, True), (5, 4, 4, 4, False),
    (5, 3, 4, 2, False), (6, 4, 4, 4, True), (6, 4, 4, 2, False), (6, 3, 4, 2, True), (6, 3, 4, 1, False)])
def test_route_and_value(textures, c0, c1, k, staged):
    w, h = 45 + textures, 31 + c0
    mat = materials.small(w + 3 * h, w, h, textures=textures, c0=c0, c1=c1, k=k, mip_min=4)
    rng = np.random.default_rng(w * h + k)
    nout, nin = 3 * textures, abi.feature_count(c0, c1)
    dw = (rng.standard_normal((nout, nin)) * 0.3).astype(np.float32)
    db = rng.random(nout).astype(np.float32)
    v0 = [(rng.random(p[0] * p[1] * c0) * 2 - 1).astype(np.float32) for p in mat.planes]
    v1 = [(rng.random(p[2] * p[3] * c1) * 2 - 1).astype(np.float32) for p in mat.planes]
    st = O.State([(p[0], p[1], p[2], p[3], mat.chain[i], v0[i], v1[i]) for i, p in enumerate(mat.planes)], c0, c1, nout, k,
                 dw, db, np.ones(nout, np.float32))
    num = den = 0.0
    for i, p in enumerate(mat.planes):
        sums = np.zeros(3)
        O.oracle().orc_objective_plane(C.byref(st.plane(i)), C.byref(st.dec), O.dptr(sums))
        num += mat.per_site[i] * sums[0]
        den += mat.per_site[i] * p[0] * p[1] * (1 + k)
    with Session(mat) as s:
        for i in range(len(mat.planes)):
            s.set_planes(i, v0[i], v1[i])
        s.set_decoder(dw, db)
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            e = s.objective(k).e
            torch.cuda.synchronize()
    assert any("k_objective_staged" in x.name for x in prof.events()) == staged
    # the same products in another order of FP64 sums (the bar of the parity tests)
    assert abs(e - num / (nout * den)) <= 1e-12 * e
