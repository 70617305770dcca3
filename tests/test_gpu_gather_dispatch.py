"""The assembly's dispatch above the sizes of the tile-edge tests: several rounds a block of the site pass (more than 227 k
pixels), level-1 planes that are not tabled in one launch of tiles and in two, against the reference-shaped assembly."""
import numpy as np
import pytest
import torch
from torch.profiler import ProfilerActivity, profile

from nntc_b200 import abi, check, lib, materials
from nntc_b200.session import Session
from test_gpu_gather import run

pytestmark = pytest.mark.gpu


def material(planes, textures, c0, c1, k):
    """Noise on planes of any sizes (a caller's chain need not halve, nor level 1 be a quarter)."""
    w, h = planes[0][:2]
    rng = np.random.default_rng(w * h + c1)
    mat = materials.Material("m", [np.zeros((h, w, 3), np.uint8)] * textures, c0, c1, k)
    mat.planes, mat.per_site = planes, materials.mip_weights(planes, "pixels", 0.5, k)
    mat.chain = [rng.random((p[1], p[0], 3 * textures)).astype(np.float32) for p in planes]
    state = ((rng.standard_normal((3 * textures, abi.feature_count(c0, c1))) * 0.3).astype(np.float32),
             rng.random(3 * textures).astype(np.float32),
             [(rng.random(p[0] * p[1] * c0) * 2 - 1).astype(np.float32) for p in planes],
             [(rng.random(p[2] * p[3] * c1) * 2 - 1).astype(np.float32) for p in planes])
    return mat, state


def gather_launches(mat, state, f32, k):
    dw, db, v0, v1 = state
    with Session(mat) as s:
        check(lib().nntc_b200_set_option(s.d, abi.OPT_FP32_STENCIL, f32), "option")
        for i in range(len(mat.planes)):
            s.set_planes(i, v0[i], v1[i])
        s.set_decoder(dw, db)
        s.set_grids(np.full(mat.c0, -1.0), np.full(mat.c0, 1.0), np.full(mat.c1, -1.0), np.full(mat.c1, 1.0))
        s.block(False, sweeps=1, k=k)
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            s.block(False, sweeps=1, k=k)
            torch.cuda.synchronize()
    names = [e.name for e in prof.events() if "k_gather" in e.name]
    return sum("k_gather_any1" in n for n in names), sum("k_gather_walk" in n for n in names)


ORDINARY = materials.plane_sizes(450, 333)          # 400 tiles, of 76.7 KB at the base and up to 80 KB below
APART = [(450, 333, 112, 83), (48, 48, 9, 9)]       # the second plane's tile takes 120 KB: one to an SM
ROUNDS = materials.plane_sizes(601, 613)


@pytest.mark.parametrize("planes,k,any1", [(ORDINARY, 4, 1), (APART, 4, 2), (APART[1:], 4, 1), (ORDINARY, 2, 1)])
@pytest.mark.parametrize("f32", [0, 1])
def test_launches_of_the_ragged_planes(planes, k, any1, f32):
    mat, state = material(planes, 1, 2, 4, k)
    assert gather_launches(mat, state, f32, k) == (any1, 0)


# ROUNDS has 1004 tiles: above the line between the tiles and the walk at K = 0 but for FP32 terms of four channels, below it
# at K = 1 and more; with FP64 terms of one or three channels the line is half as far
@pytest.mark.parametrize("c1,k,f32,tiled", [(2, 0, 0, False), (3, 0, 0, False), (2, 0, 1, False), (4, 0, 1, True),
                                            (2, 1, 0, True), (3, 1, 0, True), (2, 1, 1, True), (1, 4, 0, True)])
def test_large_ragged_planes_of_few_sites_are_walked(c1, k, f32, tiled):
    mat, state = material(ROUNDS, 1, 2, c1, k)
    assert gather_launches(mat, state, f32, k) == ((1, 0) if tiled else (0, 1))


# 7939 and 4428 tiles: the tiles are the faster up to any number at K = 2 and two FP64 channels, up to some thousands at K = 1
@pytest.mark.parametrize("w,h,c1,k,f32,tiled", [(2000, 1500, 2, 2, 0, True), (1400, 1200, 2, 1, 0, True),
                                                (1400, 1200, 3, 2, 0, False), (1400, 1200, 2, 2, 1, False)])
def test_large_ragged_planes_by_channels_and_sites(w, h, c1, k, f32, tiled):
    mat, state = material(materials.plane_sizes(w, h), 1, 2, c1, k)
    assert gather_launches(mat, state, f32, k) == ((1, 0) if tiled else (0, 1))


@pytest.mark.parametrize("c1,k", [(2, 0), (3, 1), (4, 1), (4, 4)])   # the diagonal blocks alone: walked, walked, walked, tiles
def test_diagonal_blocks_alone(c1, k):
    """The matrix-free conjugate gradients' assembly: its gradient and diagonal blocks are the full assembly's bits."""
    mat, (dw, db, v0, v1) = material(ROUNDS, 1, 2, c1, k)
    got = []
    for option in (0, 1):
        with Session(mat) as s:
            check(lib().nntc_b200_set_option(s.d, abi.OPT_ADJOINT_CG, option), "option")
            for i in range(len(mat.planes)):
                s.set_planes(i, v0[i], v1[i])
            s.set_decoder(dw, db)
            s.set_grids(np.full(2, -1.0), np.full(2, 1.0), np.full(c1, -1.0), np.full(c1, 1.0))
            s.block(False, k=k)
            got.append([s.workspace(i, False) for i in range(len(mat.planes))])
    for a, b in zip(*got):
        assert np.array_equal(a["grad"], b["grad"])
        diagonals = [x["stencil"].reshape(-1, 5, c1, c1)[:, 0] for x in (a, b)]
        assert np.array_equal(*diagonals)


@pytest.mark.parametrize("planes,textures,c0,c1,k", [(ROUNDS, 1, 2, 3, 0), (ROUNDS, 2, 4, 4, 0), (ROUNDS, 1, 4, 1, 1),
                                                     (ROUNDS, 2, 2, 4, 4), (ROUNDS, 1, 4, 3, 4), (ROUNDS, 1, 3, 2, 2),
                                                     (APART, 1, 2, 4, 4), (APART, 2, 4, 1, 4)])
def test_assembly_matches_the_reference_shape(planes, textures, c0, c1, k):
    mat, state = material(planes, textures, c0, c1, k)
    shaped, split, f32 = (run(mat, None, state, a, b, k) for a, b in ((1, 0), (0, 0), (0, 1)))
    for level in range(2):
        for i in range(len(mat.planes)):
            a, b, f = shaped[level][i], split[level][i], f32[level][i]
            for key in ("stencil", "grad"):
                assert np.array_equal(a[key], b[key]), (level, i, key)
                # the bound of the adjoint form's assembly against the FP64 one
                assert np.abs(f[key] - a[key]).max() <= 1e-5 * np.abs(a[key]).max(), (level, i, key)
