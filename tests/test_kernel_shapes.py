"""GPU kernels at the shapes where their tiles and dispatch rules turn over.

Each case runs Basic, Aggregate, Final, Aggregate through the vnlb.* entry
points on a small clip and must equal the CPU oracle bit for bit: dimensions
that leave remainders of the 8-lane chains, row counts that leave remainders of
the row tiles, ranks and matrix sizes on both sides of each kernel's range.
"""
import time

import numpy as np
import pytest

import mlp_fp64
import oracle as O
import synth
import vnlbgpu_lib as lib
from test_gpu_parity import bits, gpu_chain, session_for

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
    # blocks that fill the shared memory to its last bytes but for the static arrays: four warps of
    # row tiles (Final), and the dual Gram's columns with and without the odd unit
    ("full_tiles", 24, 20, 9, 3, dict(block_size=7, patch_time=7, group_size=33, rank=4, bm_range=2, cap_factor=1.0)),
    ("full_columns", 30, 26, 5, 3, dict(block_size=11, patch_time=3, group_size=48, rank=1, bm_range=4)),
    ("full_columns_even", 32, 30, 6, 1, dict(block_size=13, patch_time=4, group_size=80, rank=1, bm_range=5)),
    # weights off, and only some on
    ("no_weights", 48, 40, 3, 1, dict(block_size=7, patch_time=2, group_size=12, rank=10, weight_alpha=0.0,
                                      weight_beta=0.0, weight_gamma=0.0)),
    ("alpha_only", 48, 40, 3, 1, dict(block_size=7, patch_time=2, group_size=12, rank=10, weight_beta=0.0)),
]

# eigen problems on both sides of each register and lane split (8, 16, 24, 32
# rows), with fewer rows than the matrix they are stored in
JACOBI = [(k, r) for k, r in ((1, 1), (2, 2), (7, 7), (8, 8), (9, 4), (15, 15), (23, 23), (24, 24), (25, 25), (31, 8))]

# buffers of one, two and four words per lane and larger ones, fronts of up to
# 32 and more, block sizes with and without a kernel of their own
MATCH = [
    ("buffer32", 48, 40, 3, 1, dict(group_size=8, rank=8, tau=3000.0)),
    ("buffer33", 48, 40, 3, 1, dict(group_size=11, rank=8, cap_factor=3.0, tau=3000.0)),
    ("buffer64", 48, 40, 3, 1, dict(patch_time=2, group_size=16, rank=8, tau=5000.0)),
    ("buffer128", 48, 40, 3, 1, dict(patch_time=2, group_size=32, rank=8, tau=9000.0)),
    ("buffer129", 48, 40, 3, 1, dict(patch_time=2, group_size=32, rank=8, cap_factor=4.03, tau=9000.0)),
    ("front33", 48, 40, 3, 1, dict(patch_time=2, group_size=33, rank=8, cap_factor=1.5, tau=5000.0)),
    ("block10", 53, 41, 3, 1, dict(block_size=10, block_step=5, patch_time=2, group_size=16, rank=15, tau=2000.0)),
    ("block9", 48, 40, 3, 1, dict(block_size=9, patch_time=2, group_size=12, rank=8, tau=2000.0)),
    ("block5_tau", 48, 40, 3, 1, dict(block_size=5, group_size=16, rank=8, tau=1200.0)),
    # four planes and more: later planes from the list, from every candidate, and of none
    ("planes6", 64, 48, 4, 3, dict(block_size=7, block_step=5, patch_time=2, bm_range=13, group_size=16, rank=15)),
    ("planes6_all", 64, 48, 3, 3, dict(block_size=7, block_step=7, patch_time=2, group_size=16, rank=8, tau=90000.0)),
    ("planes6_block10", 48, 40, 3, 3, dict(block_size=10, block_step=9, patch_time=2, group_size=16, rank=8)),
    ("planes5", 48, 40, 7, 1, dict(patch_time=5, group_size=40, rank=8, cap_factor=1.0)),
    # windows clipped to a few candidates
    ("tiny_frame", 10, 9, 2, 1, dict(group_size=8, rank=2, block_step=2)),
]

# dense and sparse grids (step against window), many slots, odd planes
GRIDS = [
    ("step1", 40, 32, 2, 1, dict(block_size=6, block_step=1, group_size=8, rank=6, bm_range=4)),
    ("step16_window5", 90, 70, 2, 1, dict(block_step=16, group_size=6, rank=4, bm_range=2)),
    ("wide", 700, 17, 2, 1, dict(block_step=3, group_size=8, rank=6, bm_range=3)),
    ("tall", 19, 400, 2, 1, dict(block_step=3, group_size=8, rank=6, bm_range=3)),
    ("slots6", 45, 37, 6, 3, dict(patch_time=2, radius=2, group_size=12, rank=8, block_step=6)),
    ("slots9_uncoupled", 45, 37, 9, 3, dict(radius=4, group_size=8, rank=6, bm_range=4, chroma=0)),
    ("window_off", 45, 37, 3, 3, dict(weight_gamma=0.0, patch_time=2, group_size=12, rank=8)),
]


def check(w, h, f, planes, sigma, kw, seed, noisy=None):
    if noisy is None:
        _, noisy = synth.make_clip(w, h, f, planes, sigma, seed=seed)
    bp = O.cpu_params(O.BASIC, sigma, **kw)
    fp = O.cpu_params(O.FINAL, sigma, **kw)
    oracle = O.Oracle("port")
    want_basic, want_final = oracle.chain(noisy, bp, fp)
    basic_stacks, basic, _, final = gpu_chain(noisy, bp, fp)
    assert np.array_equal(bits(basic_stacks), bits(oracle.stage_stacks(O.BASIC, bp, noisy)))
    assert np.array_equal(bits(basic), bits(want_basic))
    assert np.array_equal(bits(final), bits(want_final))
    # the same frames normalised on the device
    for stage, p, ref, want in ((lib.STAGE_BASIC, bp, None, want_basic), (lib.STAGE_FINAL, fp, want_basic, want_final)):
        s = session_for(stage, p, noisy, ref)
        got = s.render_clip()
        s.close()
        assert np.array_equal(bits(got), bits(want))


@pytest.mark.parametrize("name,w,h,f,planes,kw", APPLY_TILES, ids=[c[0] for c in APPLY_TILES])
def test_apply_row_tiles(name, w, h, f, planes, kw):
    check(w, h, f, planes, 20.0, kw, seed=len(name))


@pytest.mark.parametrize("k,rank", JACOBI)
def test_jacobi_sizes(k, rank):
    check(48, 40, 3, 1, 20.0, dict(patch_time=2, group_size=k, rank=rank, cap_factor=1.0), seed=k)


@pytest.mark.parametrize("k", [8, 16, 24, 32])
def test_jacobi_groups_that_rotate_apart(k):
    """Neighbouring groups of one warp rotate at different steps, some never:
    noise of very different strength column by column, smooth ramps and repeated
    rows, so that at every step some lanes update what others only read."""
    rng = np.random.default_rng(k)
    noise = rng.normal(0.0, 1.0, (4, 1, 40, 64))
    strength = 10.0 ** -np.tile(np.repeat(np.arange(8) % 5, 8), 1)  # 1 ... 1e-4, 8 columns each
    ramp = np.add.outer(np.arange(40) / 80.0, np.arange(64) / 128.0)
    noisy = (ramp + 0.1 * noise * strength).astype(np.float32)
    noisy[:, :, 20:30] = noisy[:, :, 20:21]
    check(64, 40, 4, 1, 5.0, dict(patch_time=2, block_step=4, group_size=k, rank=k, cap_factor=1.0), 0, noisy)


@pytest.mark.parametrize("block", [3, 4, 5, 7])
@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_eigenvalues_beside_nan(block, value):
    """One chroma sample that is no number, uncoupled planes: its column makes one
    entry of the covariance's diagonal NaN beside finite ones, which have to be
    sorted all the same.  Whatever that sample cannot reach (twice the window's
    4 columns to either side, the block, the neighbours of a match) is the
    oracle's, and the session renders on."""
    kw = dict(block_size=block, block_step=2, group_size=9, rank=4, bm_range=2, chroma=0)
    _, noisy = synth.make_clip(64, 32, 2, 3, 20.0, seed=block)
    noisy[:, 1, 12, 6] = value
    bp = O.cpu_params(O.BASIC, 20.0, **kw)
    oracle = O.Oracle("port")
    want = oracle.aggregate(oracle.stage_stacks(O.BASIC, bp, noisy), noisy, bp.search_bwd, bp.search_fwd, bp.patch_time)
    s = session_for(lib.STAGE_BASIC, bp, noisy)
    for _ in range(2):
        got = s.render_clip()
        assert np.array_equal(bits(got[..., 32:]), bits(want[..., 32:]))
    s.close()


@pytest.mark.parametrize("name,w,h,f,planes,kw", MATCH, ids=[c[0] for c in MATCH])
def test_match_selection(name, w, h, f, planes, kw):
    check(w, h, f, planes, 15.0, kw, seed=len(name) + 40)


def test_search_region_limit():
    """The largest search region a session can be made for: the staged planes,
    the window's distances, the reference patch and the buffer within 200 KB.
    Four planes with 8 x 8 blocks and buffers of 64: windows up to 89 x 89."""
    noisy = np.zeros((5, 1, 104, 120), np.float32)
    kw = dict(patch_time=4, group_size=16, rank=1)
    session_for(lib.STAGE_BASIC, O.cpu_params(O.BASIC, 20.0, bm_range=44, **kw), noisy).close()
    with pytest.raises(lib.VNLBError, match="does not fit in shared memory"):
        session_for(lib.STAGE_BASIC, O.cpu_params(O.BASIC, 20.0, bm_range=45, **kw), noisy)


@pytest.mark.parametrize("planes,patch_time,tau", [(1, 1, 0.0), (1, 1, 400.0), (3, 2, 0.0)])
def test_match_ties(planes, patch_time, tau):
    """Flat areas and repeated columns: most distances tie, many at zero."""
    rng = np.random.default_rng(planes + 10 * patch_time)
    noisy = np.full((4, planes, 40, 48), 0.5, np.float32)
    noisy[:, :, :, 24:] = np.tile(rng.random((4, planes, 40, 4)).astype(np.float32), (1, 1, 1, 6))
    noisy[:, :, 8:14, 4:12] = rng.random((4, planes, 6, 8)).astype(np.float32)
    check(48, 40, 4, planes, 10.0, dict(patch_time=patch_time, group_size=12, rank=8, tau=tau, block_step=5), 0, noisy)


@pytest.mark.parametrize("name,w,h,f,planes,kw", GRIDS, ids=[c[0] for c in GRIDS])
def test_grids_and_tiles(name, w, h, f, planes, kw):
    check(w, h, f, planes, 15.0, kw, seed=len(name) + 70)


def test_paste_waits_run_out_and_report():
    """The paste mask's waits for the grid row above are bounded: with rows told
    to publish nothing the first wait runs out, all others give up with it (100
    grid rows of 8 batches, 16 rows at a time, would wait 50 times as long), and
    the render raises.  The session then renders as a fresh one does."""
    kw = dict(block_step=4, group_size=8, rank=6, bm_range=3)
    _, noisy = synth.make_clip(1000, 400, 2, 1, 15.0, seed=5)
    bp = O.cpu_params(O.BASIC, 15.0, **kw)
    fresh = session_for(lib.STAGE_BASIC, bp, noisy)
    want = fresh.render_clip()
    fresh.close()
    s = session_for(lib.STAGE_BASIC, bp, noisy)
    s.stall_paste_waits(True)
    start = time.perf_counter()
    with pytest.raises(lib.VNLBError, match="timed out waiting for the grid row above"):
        s.render_clip()
    assert time.perf_counter() - start < 2.0
    s.stall_paste_waits(False)
    assert np.array_equal(bits(s.render_clip()), bits(want))
    s.close()


@pytest.mark.parametrize("batch,inputs,hidden,layers,outputs", [
    (1, 3, 5, 1, 7), (63, 45, 128, 3, 65), (129, 27, 64, 2, 1083), (300, 45, 128, 3, 5445), (700, 16, 16, 1, 16),
    (5, 27, 64, 2, 1536), (5, 27, 64, 2, 1537), (66, 27, 64, 2, 6144), (66, 27, 64, 2, 6201)])
def test_network_products(batch, inputs, hidden, layers, outputs):
    """Products with whole tiles, remainders and splits, against float64, each
    layer's weight and bias gradients against their own largest.  FP32 roundings
    along a path of n terms add up like a random walk, to sqrt(n) 2^-24 of the
    values; six times that leaves room for the largest of all elements."""
    import torch

    rng = np.random.default_rng(batch)
    shape = (inputs, hidden, layers, outputs)
    net = lib.MLP(*shape, max_batch=batch, seed=batch)
    x = rng.normal(0.0, 1.0, (batch, inputs)).astype(np.float32)
    t = rng.integers(0, outputs, (batch, 8)).astype(np.int32)
    dx, dt = torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda()
    out = torch.empty((batch, outputs), device="cuda")
    torch.cuda.synchronize()
    grads, loss = net.gradients(dx.data_ptr(), dt.data_ptr(), batch, 8)
    net.logits(dx.data_ptr(), batch, out.data_ptr())
    want_loss, want = mlp_fp64.loss_and_gradients(net.get_weights(), shape, x, t)
    z = mlp_fp64.forward_logits(net.get_weights(), shape, x)
    bound = 6.0 * (inputs + layers * hidden + outputs + batch) ** 0.5 * 2.0**-24
    assert abs(loss - want_loss) <= bound * max(1.0, abs(want_loss))
    for got_arrays, want_arrays in zip(mlp_fp64.unpack(grads, *shape), mlp_fp64.unpack(want, *shape)):
        for l, (g, v) in enumerate(zip(got_arrays, want_arrays)):
            assert np.abs(g - v).max() <= bound * np.abs(v).max(), (l, g.shape)
    assert np.abs(out.cpu().numpy() - z).max() <= bound * np.abs(z).max()


def test_network_workspace_follows_the_batch():
    """A network for batches of one row holds no workspace for large ones: its
    few small arrays stay within the driver's 2 MiB units."""
    import torch

    lib.MLP(3, 5, 1, 7, max_batch=1, seed=0)  # the library's kernels are loaded
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    net = lib.MLP(3, 5, 1, 7, max_batch=1, seed=0)
    assert before - torch.cuda.mem_get_info()[0] <= 4 << 20
    del net
