"""The tiled gather and the walk beside it against the reference-shaped assembly, bit for bit, at the edges of the tiles
(64 x 4 texels at level 0, 8 x 4 at level 1), on planes down to one texel, for every channel count, K and kind of
output weights; and the FP32 gather of the same states within the bound the adjoint form's assembly is held to."""
import numpy as np
import pytest

from nntc_b200 import abi, check, lib, materials
from nntc_b200.session import Session

pytestmark = pytest.mark.gpu


# (textures, c0, c1, w, h, mip_min, k, weights): tiles met exactly, one texel over and one short; level 1 tabled (a quarter
# of a power of two) and walked; chains that end at one texel
CASES = [(1, 2, 4, 64, 32, 8, 4, "one"), (2, 4, 4, 128, 64, 1, 4, "one"), (1, 1, 1, 65, 5, 1, 4, "one"),
         (1, 3, 2, 63, 37, 1, 4, "mixed"), (2, 2, 3, 32, 32, 1, 2, "mixed"), (1, 4, 1, 64, 64, 1, 1, "two"),
         (1, 1, 4, 256, 8, 2, 4, "mixed"), (3, 4, 4, 66, 130, 8, 4, "mixed"), (1, 2, 2, 8, 8, 1, 4, "one")]


def run(mat, cw, state, shaped, f32, k):
    dw, db, v0, v1 = state
    with Session(mat, model=abi.make_model(mat, cw=cw)) as s:
        check(lib().nntc_b200_set_option(s.d, abi.OPT_REFERENCE_SHAPED_ASSEMBLY, shaped), "option")
        check(lib().nntc_b200_set_option(s.d, abi.OPT_FP32_STENCIL, f32), "option")
        for i in range(len(mat.planes)):
            s.set_planes(i, v0[i], v1[i])
        s.set_decoder(dw, db)
        s.set_grids(np.full(mat.c0, -1.0), np.full(mat.c0, 1.0))
        out = []
        for level0 in (False, True):
            for i in range(len(mat.planes)):
                s.set_planes(i, v0[i], v1[i])
            s.block(level0, k=k)
            out.append([s.workspace(i, level0) for i in range(len(mat.planes))])
    return out


@pytest.mark.parametrize("textures,c0,c1,w,h,mip_min,k,weights", CASES)
def test_gather_matches_the_reference_shape(textures, c0, c1, w, h, mip_min, k, weights):
    mat = materials.small(w * 3 + h, w, h, textures=textures, c0=c0, c1=c1, k=k, mip_min=mip_min)
    mat.planes = [p for p in mat.planes if p[2] > 0 and p[3] > 0]
    rng = np.random.default_rng(w + 31 * h)
    nout = 3 * textures
    state = ((rng.standard_normal((nout, abi.feature_count(c0, c1))) * 0.3).astype(np.float32),
             rng.random(nout).astype(np.float32),
             [(rng.random(p[0] * p[1] * c0) * 2 - 1).astype(np.float32) for p in mat.planes],
             [(rng.random(p[2] * p[3] * c1) * 2 - 1).astype(np.float32) for p in mat.planes])
    # weights of one or two keep the monomial matrices symmetric bit for bit; the others take the general expansion
    cw = {"one": None, "two": [2.0] * nout, "mixed": list(0.3 + rng.random(nout))}[weights]
    shaped, split, f32 = (run(mat, cw, state, a, b, k) for a, b in ((1, 0), (0, 0), (0, 1)))
    for level in range(2):
        for i in range(len(mat.planes)):
            a, b, f = shaped[level][i], split[level][i], f32[level][i]
            for key in ("stencil", "grad"):
                assert np.array_equal(a[key], b[key]), (level, i, key)
                # the bound of the adjoint form's assembly against the FP64 one (its own test's, on other states)
                assert np.abs(f[key] - a[key]).max() <= 1e-5 * np.abs(a[key]).max(), (level, i, key)
