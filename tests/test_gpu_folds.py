"""The fixed-order folds of per-block partials on a B200, at plane sizes around one and several staged chunks (a chunk
is 1536 or 2048 partials of 256 texels): the ranges and extremes are exact, the sums FP64 sums of positive terms."""
import numpy as np
import pytest

from nntc_b200 import materials
from nntc_b200.session import Session

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(16, 8), (128, 64), (768, 512), (1216, 880)])
def test_plane_folds(w, h):
    mat = materials.small(w + h, w, h, textures=1, c0=1, c1=2)
    rng = np.random.default_rng(w)
    with Session(mat) as s:
        for i, p in enumerate(mat.planes):
            s.set_planes(i, rng.random(p[0] * p[1]) * 2 - 1, rng.random(p[2] * p[3] * 2) * 2 - 1)
        s.set_decoder(rng.standard_normal((3, s.m.nin)) * 0.3, rng.random(3))
        s.set_grids(np.full(1, -1.0), np.full(1, 1.0))
        for level0 in (False, True):
            rep, _ = s.block(level0, ridge=1e-3)
            for i in range(len(mat.planes)):
                ws = s.workspace(i, level0)
                c = 1 if level0 else 2
                v = (s.get_v0(i) if level0 else s.get_v1(i)).reshape(-1, c)
                diag = ws["stencil"].reshape(-1, 5, c, c)[:, 0][:, range(c), range(c)]
                r = rep[i]
                assert r.min_diag == diag.min() and r.max_diag == diag.max()
                assert list(r.lo[:c]) == list(v.min(0)) and list(r.hi[:c]) == list(v.max(0))
                # n positive terms summed in two fixed orders: each within n eps of the exact sum at the very worst,
                # and in practice sqrt(n) eps of it: 1e-12 holds for n up to 1e6
                assert abs(r.lambda_ - 1e-3 * diag.mean()) <= 1e-12 * r.lambda_
                assert abs(r.plane2 - np.sum(v.astype(np.float64) ** 2)) <= 1e-12 * r.plane2
                assert abs(r.delta2 - np.sum(ws["x"] ** 2)) <= 1e-12 * r.delta2


@pytest.mark.parametrize("w,h,mip_min", [(12, 12, 8), (40, 24, 1), (96, 64, 1)])
def test_normal_equations_fold(w, h, mip_min):
    """One to seven planes' partials folded: the target sums against the features of a constant latent, in closed form."""
    mat = materials.small(w, w, h, textures=2, c0=2, c1=3, mip_min=mip_min)
    with Session(mat) as s:
        for i, p in enumerate(mat.planes):
            s.set_planes(i, np.full(p[0] * p[1] * 2, 0.5), np.full(p[2] * p[3] * 3, 0.25))
        s.solve_decoder()
        a = s.normal_equations()
        mm = s.m.nin + 1
        # every site's features are the same constants, so A is the outer product of them times the weighted site count
        phi = np.array([0.25] * 3 + [0.5] * 2 + [0.125] * 6 + [1.0])
        count = sum(om * p[0] * p[1] * 5 for om, p in zip(mat.per_site, mat.planes))
        want = np.array([phi[i] * phi[j] for i in range(mm) for j in range(i, mm)]) * count
        # bilinear weights sum to one within 2 float roundings each, so a feature is off by at most 4 eps_f relative
        assert np.all(np.abs(a[:want.size] - want) <= 8 * 2.0 ** -23 * np.abs(want))
