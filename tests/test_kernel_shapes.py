"""GPU kernels at the shapes where their tiles and dispatch rules turn over.

Each case runs Basic, Aggregate, Final, Aggregate through the vnlb.* entry
points on a small clip and must equal the CPU oracle bit for bit: dimensions
that leave remainders of the 8-lane chains, row counts that leave remainders of
the row tiles, ranks and matrix sizes on both sides of each kernel's range.
"""
import numpy as np
import pytest

import oracle as O
import synth
from test_gpu_parity import bits, gpu_chain

pytestmark = pytest.mark.gpu

APPLY_TILES = [
    # dimension remainders 2, 1, 4 and none; 72 = 2 x 36 takes whole chains of 9
    ("dim98_rows5", 48, 40, 3, 1, dict(block_size=7, patch_time=2, group_size=5, rank=5, cap_factor=1.0)),
    ("dim81_rows7", 48, 40, 3, 1, dict(block_size=9, group_size=7, rank=6, cap_factor=1.0)),
    ("dim100_rows13", 48, 40, 3, 1, dict(block_size=10, group_size=13, rank=13, cap_factor=1.0)),
    ("dim72_rows64", 48, 40, 3, 1, dict(block_size=6, patch_time=2, group_size=16, rank=15, tau=9000.0)),
    # covariance models (dimension 25, 27), uncoupled planes
    ("dim25_rank16", 40, 32, 3, 1, dict(block_size=5, group_size=20, rank=16, bm_range=4)),
    ("dim27_yuv", 40, 32, 2, 3, dict(block_size=3, block_step=2, group_size=9, rank=7, bm_range=3)),
    ("dim98_uncoupled", 48, 40, 3, 3, dict(block_size=7, patch_time=2, group_size=10, rank=9, chroma=0, tau=900.0)),
    # ranks of the wide tiles and on both sides of them
    ("rank16", 48, 40, 3, 1, dict(patch_time=2, group_size=16, rank=16, tau=900.0)),
    ("rank17", 48, 40, 3, 1, dict(patch_time=2, group_size=17, rank=17, tau=900.0)),
    ("rank32", 48, 40, 3, 1, dict(patch_time=2, group_size=32, rank=32, cap_factor=1.5, tau=900.0)),
    ("rank33", 48, 40, 3, 1, dict(patch_time=2, group_size=33, rank=33, cap_factor=1.0)),
    # dimensions whose blocks hold four warps (768) and, in Final, two (1200)
    ("dim768", 64, 48, 2, 3, dict(block_size=16, group_size=6, rank=4, bm_range=2)),
    ("dim1200", 64, 48, 4, 1, dict(block_size=20, patch_time=3, group_size=6, rank=4, bm_range=2)),
    # weights off, and only some on
    ("no_weights", 48, 40, 3, 1, dict(block_size=7, patch_time=2, group_size=12, rank=10, weight_alpha=0.0,
                                      weight_beta=0.0, weight_gamma=0.0)),
    ("alpha_only", 48, 40, 3, 1, dict(block_size=7, patch_time=2, group_size=12, rank=10, weight_beta=0.0)),
]

# eigen problems on both sides of each register and lane split (8, 16, 24, 32
# rows), with fewer rows than the matrix they are stored in
JACOBI = [(k, r) for k, r in ((1, 1), (2, 2), (7, 7), (8, 8), (9, 4), (15, 15), (23, 23), (24, 24), (25, 25), (31, 8))]


def check(w, h, f, planes, sigma, kw, seed):
    _, noisy = synth.make_clip(w, h, f, planes, sigma, seed=seed)
    bp = O.cpu_params(O.BASIC, sigma, **kw)
    fp = O.cpu_params(O.FINAL, sigma, **kw)
    oracle = O.Oracle("port")
    want_basic, want_final = oracle.chain(noisy, bp, fp)
    basic_stacks, basic, _, final = gpu_chain(noisy, bp, fp)
    assert np.array_equal(bits(basic_stacks), bits(oracle.stage_stacks(O.BASIC, bp, noisy)))
    assert np.array_equal(bits(basic), bits(want_basic))
    assert np.array_equal(bits(final), bits(want_final))


@pytest.mark.parametrize("name,w,h,f,planes,kw", APPLY_TILES, ids=[c[0] for c in APPLY_TILES])
def test_apply_row_tiles(name, w, h, f, planes, kw):
    check(w, h, f, planes, 20.0, kw, seed=len(name))


@pytest.mark.parametrize("k,rank", JACOBI)
def test_jacobi_sizes(k, rank):
    check(48, 40, 3, 1, 20.0, dict(patch_time=2, group_size=k, rank=rank, cap_factor=1.0), seed=k)
