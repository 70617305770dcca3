"""The target rows staged by a warp (objective, normal equations) at every row length, on planes whose last warp holds
fewer than 32 pixels and planes of less than one warp: E and the FP64 normal equations against the C restatement."""
import ctypes as C

import numpy as np
import pytest

import oracle as O
from nntc_b200 import abi, materials
from nntc_b200.session import Session

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("textures,c0,c1,w,h", [(1, 2, 4, 37, 29), (2, 4, 4, 33, 40), (3, 1, 3, 70, 21), (4, 2, 4, 129, 19),
                                                (5, 3, 4, 41, 33), (6, 4, 2, 64, 37), (6, 4, 4, 31, 65)])
def test_objective_and_normal_equations(textures, c0, c1, w, h):
    mat = materials.small(w + 3 * h, w, h, textures=textures, c0=c0, c1=c1, mip_min=4)
    rng = np.random.default_rng(w * h)
    nout, nin = 3 * textures, abi.feature_count(c0, c1)
    dw = (rng.standard_normal((nout, nin)) * 0.3).astype(np.float32)
    db = rng.random(nout).astype(np.float32)
    v0 = [(rng.random(p[0] * p[1] * c0) * 2 - 1).astype(np.float32) for p in mat.planes]
    v1 = [(rng.random(p[2] * p[3] * c1) * 2 - 1).astype(np.float32) for p in mat.planes]
    st = O.State([(p[0], p[1], p[2], p[3], mat.chain[i], v0[i], v1[i]) for i, p in enumerate(mat.planes)], c0, c1, nout, 4,
                 dw, db, np.ones(nout, np.float32))
    mm = nin + 1
    entries = np.zeros(mm * (mm + 1) // 2 + nout * mm)
    num = den = 0.0
    for i, p in enumerate(mat.planes):
        one, sums = np.zeros_like(entries), np.zeros(3)
        O.oracle().orc_normal_equations_plane(C.byref(st.plane(i)), C.byref(st.dec), O.dptr(one))
        O.oracle().orc_objective_plane(C.byref(st.plane(i)), C.byref(st.dec), O.dptr(sums))
        entries += mat.per_site[i] * one
        num += mat.per_site[i] * sums[0]
        den += mat.per_site[i] * p[0] * p[1] * 5
    with Session(mat) as s:
        for i in range(len(mat.planes)):
            s.set_planes(i, v0[i], v1[i])
        s.set_decoder(dw, db)
        e = s.objective().e
        s.solve_decoder()
        ne = s.normal_equations()
    # the same products in another order of FP64 sums (the bar of the parity tests)
    assert abs(e - num / (nout * den)) <= 1e-12 * e
    assert np.abs(ne - entries).max() <= 1e-12 * np.abs(entries).max()
