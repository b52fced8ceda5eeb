"""The resident-weight 3^3 kernel where it marches along z: a block owns many output planes, its piece of the plane list spans one to three
runs, the three-plane accumulator window wraps around the slot ring, the last plane of a volume commits on its own.  Full-size layers of
the benchmark's network (the shapes the benchmark times) against the oracle on identical MX operands, random operands within 1e-3 relative
L2 and exact operands bit for bit; then small ragged grids cut into few blocks with umx_conv_r_block_cap, which reach the same code paths
(several runs a piece, wrapped windows, both column-tile widths, one and two blocks a multiprocessor) in seconds."""
import numpy as np
import pytest

import gpu_util as G
import orc
import synth
from test_oracle import exact_operands

pytestmark = pytest.mark.gpu
TOL = 1e-3

FULL = [
    # N, Ci, Co, D: the level-0 and level-1 3^3 convs of the benchmark's network at their full sizes
    (1, 32, 32, 128),        # enc0.c2, dec0.c2: one input block, two blocks a multiprocessor
    (1, 64, 32, 128),        # dec0.c1: two input blocks
    (1, 64, 64, 64),         # enc1.c2, dec1.c2: 64-channel column tile, one block a multiprocessor
    (1, 128, 64, 64),        # dec1.c1: four input blocks
    (2, 32, 32, 128),        # a batch: pieces that cross from one sample into the next
    (2, 64, 64, 64),
]


def run(kind, mx, w, b, N, Ci, D, H, W, Co, bits, want_kernel=1):
    got = G.run_pm32(kind, mx, w, b, N, Ci, D, H, W, Co, bits)
    assert G.L().umx_conv_last_kernel() == want_kernel, "the launch did not take the resident-weight kernel"
    return got


@pytest.mark.parametrize("bits", [8, 4])
@pytest.mark.parametrize("N,Ci,Co,D", FULL)
def test_full_size_layers_random_operands(dev, N, Ci, Co, D, bits):
    S = D ** 3
    x = synth.rng(301).standard_normal(N * Ci * S).astype(np.float32)
    w, b = synth.kaiming(302, Co, Ci, 27), synth.bias(303, Co, 0.1)
    mx, want = orc.conv_case("conv3", x, w, b, N, Ci, D, D, D, Co, bits)
    del x
    got = run("conv3", mx, w, b, N, Ci, D, D, D, Co, bits)
    assert np.isfinite(got).all()
    e = orc.rel_l2(got, want)
    print("3^3 %d -> %d on %d^3 x %d, MX-fp%d: rel-L2 %.3g, max abs %.3g" % (Ci, Co, D, N, bits, e, np.abs(got - want).max()))
    assert e < TOL


@pytest.mark.parametrize("bits", [8, 4])
@pytest.mark.parametrize("N,Ci,Co,D", [(1, 32, 32, 128), (1, 128, 64, 64), (1, 64, 32, 128)])
def test_full_size_layers_exact_operands(dev, N, Ci, Co, D, bits):
    S = D ** 3
    x = exact_operands(311, (N, Ci, D, D, D), 1).reshape(-1)
    w = exact_operands(312, (Co, Ci, 27), 1)
    b = (synth.rng(313).integers(-8, 8, Co) * 0.5).astype(np.float32)
    mx, want = orc.conv_case("conv3", x, w, b, N, Ci, D, D, D, Co, bits)
    del x
    got = run("conv3", mx, w, b, N, Ci, D, D, D, Co, bits)
    assert np.array_equal(got, want), "%d of %d differ" % (np.count_nonzero(got != want), want.size)


SMALL = [
    # N, Ci, Co, D, H, W, cap: `cap` blocks per column tile
    (1, 32, 32, 13, 19, 16, 3),     # 4 tiles x 13 planes over 3 blocks: 17-plane pieces, two or three runs each
    (1, 32, 32, 9, 19, 48, 5),      # 12 tiles
    (2, 64, 32, 7, 19, 16, 3),      # batch: pieces cross samples; two input blocks
    (1, 64, 64, 11, 16, 16, 2),     # 64-channel column tile (one block a multiprocessor)
    (1, 128, 64, 5, 35, 16, 1),     # one block takes every plane of six tiles: a run per tile, four input blocks
    (1, 96, 128, 12, 19, 16, 2),    # three input blocks, four column tiles of 32 channels
    (2, 32, 96, 6, 16, 32, 2),      # three column tiles of 32 channels
    (1, 32, 32, 1, 64, 32, 1),      # single planes: sixteen runs of one plane, each first and last at once
    (1, 32, 32, 1, 16, 16, 0),      # fewer planes than blocks: one plane a block
    (1, 32, 32, 2, 33, 16, 1),
]


@pytest.mark.parametrize("bits", [8, 4])
@pytest.mark.parametrize("N,Ci,Co,D,H,W,cap", SMALL)
def test_small_grids_in_few_blocks(dev, N, Ci, Co, D, H, W, cap, bits):
    L = G.L()
    S = D * H * W
    x = synth.rng(321).standard_normal(N * Ci * S).astype(np.float32)
    w, b = synth.kaiming(322, Co, Ci, 27), synth.bias(323, Co, 0.1)
    mx, want = orc.conv_case("conv3", x, w, b, N, Ci, D, H, W, Co, bits)
    xe = exact_operands(324, (N, Ci, D, H, W), 1).reshape(-1)
    we = exact_operands(325, (Co, Ci, 27), 1)
    mxe, wante = orc.conv_case("conv3", xe, we, None, N, Ci, D, H, W, Co, bits)
    L.umx_conv_r_block_cap(cap)
    try:
        got = run("conv3", mx, w, b, N, Ci, D, H, W, Co, bits)
        gote = run("conv3", mxe, we, None, N, Ci, D, H, W, Co, bits)
        # the InstanceNorm path through the same launch geometry
        c = G.Conv("conv3", w, b, Co, Ci, bits)
        raw, _ = c.fwd(mx, N, D, H, W, G.OUT_H16B)
        y, coef = c.fwd_norm(mx, N, D, H, W, epilogue_stats=True)
        assert L.umx_conv_last_kernel() == 1
        L.umx_conv_r_block_cap(0)
        y_free, coef_free = c.fwd_norm(mx, N, D, H, W, epilogue_stats=True)      # the same layer cut into as many blocks as the device holds
        same_kernel = L.umx_conv_last_kernel() == 1          # (a few of these grids then go to the general kernel: another summation order)
        c.free()
    finally:
        L.umx_conv_r_block_cap(0)
    e = orc.rel_l2(got, want)
    assert np.isfinite(got).all() and e < TOL, "relative L2 %.3g" % e
    assert np.array_equal(gote, wante), "%d of %d differ" % (np.count_nonzero(gote != wante), wante.size)
    assert np.array_equal(raw.view(np.uint16), y.view(np.uint16))
    assert np.array_equal(raw.view(np.float16), orc.pm_to_blocked(got, N, Co, S).astype(np.float16))
    # the epilogue's InstanceNorm sums: the oracle's fp64 statistics bit for bit, whatever the partition of the planes over blocks
    assert np.array_equal(coef, orc.in_coef(orc.in_sums(y.astype(np.float32), N, Co, S), N, Co, S))
    if same_kernel:
        assert np.array_equal(y_free.view(np.uint16), y.view(np.uint16)) and np.array_equal(coef, coef_free)


@pytest.mark.parametrize("N,Ci,Co,D,H,W,bits,cap", [(1, 32, 32, 3, 16, 16, 8, 0), (2, 32, 24, 4, 19, 16, 8, 0), (1, 64, 64, 3, 9, 48, 8, 0), (1, 32, 96, 5, 16, 32, 4, 0), (1, 64, 33, 12, 5, 16, 8, 0), (1, 32, 1, 2, 16, 16, 8, 0),
                                                    (1, 128, 64, 6, 20, 16, 8, 1)])       # a stage of three of the four input items, then one of the fourth (blocked halves leave room for all four)
def test_plane_major_halves(dev, N, Ci, Co, D, H, W, bits, cap):
    """the plane-major fp16 epilogue: the values of the blocked fp16 one, at partial tiles, channel counts that end inside a block or a pair, one and several
    column tiles; an output that is not on a 16-byte boundary takes the general epilogue"""
    import ufsm_b200
    from ufsm_b200 import DevBuf
    S, nbi, nbo, r = D * H * W, (Ci + 31) // 32, (Co + 31) // 32, synth.rng(701)
    x = DevBuf(data=np.concatenate([r.integers(0, 120, N * nbi * S * 4 * bits, dtype=np.uint8), r.integers(118, 128, N * nbi * S, dtype=np.uint8)]))
    c = G.Conv("conv3", synth.kaiming(702, Co, Ci, 27), synth.bias(703, Co, 0.1), Co, Ci, bits)

    def run(nbytes, shift, mode):
        y = DevBuf(data=np.full(nbytes + shift, 0x5a, np.uint8))
        dev.umx_conv_r_block_cap(cap)
        try:
            assert dev.umx_conv_fwd(c.h, x.ptr, N, D, H, W, y.ptr + shift, mode, 0, 0, 0, None, 1) == 0
        finally:
            dev.umx_conv_r_block_cap(0)
        assert dev.umx_conv_last_kernel() == 1
        ufsm_b200.check()
        return y.download()[shift:].copy().view(np.uint16)
    want = run(N * nbo * S * 64, 0, 0).reshape(N, nbo, S, 32).transpose(0, 1, 3, 2).reshape(N, nbo * 32, S)[:, :Co]
    for shift in (0, 2):
        assert np.array_equal(run(N * Co * S * 2, shift, 3).reshape(N, Co, S), want)


@pytest.mark.parametrize("bits", [8, 4])
@pytest.mark.parametrize("N,Ci,Co,D,H,W,cap", [
    (1, 32, 64, 41, 37, 19, 2),        # odd grid, runs of many planes: windows that wrap around the slot ring, pieces of several runs
    (2, 64, 96, 24, 33, 8, 3),         # even depth (the last plane completes on an odd input plane), 32-channel column tiles, pieces that cross samples
    (1, 32, 32, 1, 40, 50, 0),         # one input plane: a stage that starts and completes its output
    (1, 160, 40, 9, 16, 16, 1),        # the widest input in MX-fp8, one block a column tile
    (2, 33, 64, 7, 5, 3, 0),           # grids smaller than a tile, a second input block of one channel
])
def test_stride2_runs_and_wraps(dev, N, Ci, Co, D, H, W, cap, bits):
    """The resident-weight stride-2 kernel on exact operands (every product and partial sum representable): the oracle's bits, whatever the pieces."""
    x = exact_operands(331, (N, Ci, D, H, W), 1).reshape(-1)
    w = exact_operands(332, (Co, Ci, 27), 1)
    b = (synth.rng(333).integers(-8, 8, Co) * 0.5).astype(np.float32)
    mx, want = orc.conv_case("conv3s2", x, w, b, N, Ci, D, H, W, Co, bits)
    dev.umx_conv_r_block_cap(cap)
    try:
        got = run("conv3s2", mx, w, b, N, Ci, D, H, W, Co, bits, want_kernel=4)
    finally:
        dev.umx_conv_r_block_cap(0)
    assert np.array_equal(got, want), "%d of %d differ" % (np.count_nonzero(got != want), want.size)


@pytest.mark.parametrize("bits", [8, 4])
@pytest.mark.parametrize("N,Ci,Co,D,H,W,cap", [
    (1, 32, 32, 33, 17, 13, 2),        # rows of every alignment, runs of many planes
    (2, 64, 64, 12, 31, 21, 3),        # two input blocks, 64-channel tiles, pieces that cross samples
    (1, 96, 32, 9, 18, 35, 2),         # three input blocks: in MX-fp4 the second item's second block is not there
    (2, 32, 64, 40, 5, 3, 1),          # a grid narrower than a tile
    (1, 1, 32, 20, 16, 30, 1),         # even width, one channel
    (1, 64, 64, 11, 19, 24, 2),        # whole tile rows: the plane-major epilogue's wide stores behind a gathered window
    (1, 32, 33, 7, 16, 40, 1),
    (1, 64, 32, 7, 17, 13, 2),         # scale bytes that end inside a word, in MX-fp4 of an item with both blocks
    (1, 64, 32, 24, 1, 5, 2),          # planes of a few voxels
    (1, 64, 32, 25, 1, 2, 2),
])
def test_widths_that_tma_does_not_take(dev, N, Ci, Co, D, H, W, cap, bits):
    """Scale planes whose rows are not multiples of 16 bytes: the scale warp gathers its window.  Random operands within 1e-3 of the oracle (the order of the fp32 sums is the only
    freedom), exact operands the oracle's bits; fp16 plane-major, blocked fp16 and MX outputs equal to those of the fp32 output, with nothing written behind the tensor (blocked halves
    of several MX-fp8 items are the general kernel's, on exact operands the same)."""
    import ufsm_b200
    from ufsm_b200 import DevBuf
    S, nbo = D * H * W, (Co + 31) // 32
    x = synth.rng(341).standard_normal(N * Ci * S).astype(np.float32) * np.exp2(synth.rng(344).integers(-6, 7, N * Ci * S)).astype(np.float32)
    w, b = synth.kaiming(342, Co, Ci, 27), synth.bias(343, Co, 0.1)
    mx, want = orc.conv_case("conv3", x, w, b, N, Ci, D, H, W, Co, bits)
    xe = exact_operands(345, (N, Ci, D, H, W), 1).reshape(-1)
    we = exact_operands(346, (Co, Ci, 27), 1)
    mxe, wante = orc.conv_case("conv3", xe, we, None, N, Ci, D, H, W, Co, bits)
    dev.umx_conv_r_block_cap(cap)
    try:
        got = run("conv3", mx, w, b, N, Ci, D, H, W, Co, bits)
        gote = run("conv3", mxe, we, None, N, Ci, D, H, W, Co, bits)
        c = G.Conv("conv3", w, b, Co, Ci, bits)
        h16, _ = c.fwd(mx, N, D, H, W, G.OUT_PM16)
        q, _ = c.fwd(mx, N, D, H, W, G.OUT_MXRAW, 8)
        assert dev.umx_conv_last_kernel() == 1
        c.free()
        blocked = []
        for w_, b_, m_ in ((w, b, mx), (we, None, mxe)):
            c = G.Conv("conv3", w_, b_, Co, Ci, bits)
            xd, yd = DevBuf(data=G.to_split(m_, N, (Ci + 31) // 32 * 32, S, bits)), DevBuf(N * nbo * S * 64 + 256).fill(0x5a)
            assert dev.umx_conv_fwd(c.h, xd.ptr, N, D, H, W, yd.ptr, G.OUT_H16B, 0, 0, 0, None, 3) == 0
            ufsm_b200.check()
            assert dev.umx_conv_last_kernel() == (0 if bits == 8 and Ci > 32 else 1)
            c.free()
            raw = yd.download()
            assert (raw[N * nbo * S * 64:] == 0x5a).all()
            blocked.append(raw[:N * nbo * S * 64].view(np.float16))
    finally:
        dev.umx_conv_r_block_cap(0)
    if not (bits == 8 and Ci > 32):
        assert np.array_equal(blocked[0], orc.pm_to_blocked(got, N, Co, S).astype(np.float16))
    assert np.array_equal(blocked[1], orc.pm_to_blocked(wante, N, Co, S).astype(np.float16))
    e = orc.rel_l2(got, want)
    assert np.isfinite(got).all() and e < TOL, "relative L2 %.3g" % e
    assert np.array_equal(gote, wante), "%d of %d differ" % (np.count_nonzero(gote != wante), wante.size)
    assert np.array_equal(h16.view(np.float16).reshape(-1), got.astype(np.float16).reshape(-1))
    assert np.array_equal(q, orc.blocked_to_mx(orc.pm_to_blocked(got, N, Co, S), 8, N, Co, S))


@pytest.mark.parametrize("kind,want_kernel,W", [("conv3", 1, 16), ("conv3", 1, 13), ("conv3s2", 4, 16), ("conv1", 2, 16), ("tconv2", 2, 16)])
def test_nan_scales_stay_in_their_sample(dev, kind, want_kernel, W):
    """MX-fp4 with an odd number of blocks: the last item's second block has zero weights, and its scales are not those of the next sample (0xff, of a block with a NaN, would make NaN
    of zero codes times zero weights)."""
    N, Ci, Co, D, H = 2, 96, 32, 6, 16
    S = D * H * W
    x = synth.rng(351).standard_normal(N * Ci * S).astype(np.float32)
    xn = x.copy()
    xn[Ci * S:] = np.nan
    w, b = synth.kaiming(352, Co, Ci, {"conv1": 1, "tconv2": 8}.get(kind, 27), transposed=kind == "tconv2"), synth.bias(353, Co, 0.1)
    mx, want = orc.conv_case(kind, x, w, b, N, Ci, D, H, W, Co, 4)
    mxn, _ = orc.conv_case(kind, xn, w, b, N, Ci, D, H, W, Co, 4)
    dev.umx_conv_r_block_cap(1)
    try:
        got = run(kind, mx, w, b, N, Ci, D, H, W, Co, 4, want_kernel)
        gotn = run(kind, mxn, w, b, N, Ci, D, H, W, Co, 4, want_kernel)
    finally:
        dev.umx_conv_r_block_cap(0)
    half = got.size // 2
    assert np.isfinite(got).all() and np.array_equal(got.reshape(-1)[:half], gotn.reshape(-1)[:half])
    assert np.isnan(gotn.reshape(-1)[half:]).any()


@pytest.mark.parametrize("N,Ci,Co,D,H,W,bits,kernels", [
    (3, 32, 96, 24, 20, 32, 8, (0, 1)),       # several column tiles: one wave of the general kernel's blocks alone, more in the batch
    (3, 32, 96, 24, 20, 32, 4, (0, 1)),
    (2, 96, 96, 24, 20, 32, 8, (0, 0)),       # MX-fp8 of several input items: an order of its own, so by one sample
    (2, 64, 256, 24, 20, 32, 8, (1, 1)),      # more than one wave alone
    (2, 96, 96, 24, 20, 32, 4, (0, 1)),       # a padded item
    (4, 32, 32, 33, 31, 30, 8, (0, 1)),       # rows that TMA does not take
    (4, 64, 32, 33, 31, 30, 8, (0, 0)),
    (4, 64, 32, 33, 31, 30, 4, (0, 1)),
    (8, 128, 128, 20, 16, 16, 8, (0, 0)),     # K split alone, so split in the batch too
])
def test_a_batch_may_take_the_other_kernel(dev, N, Ci, Co, D, H, W, bits, kernels):
    """In MX-fp4 and with one input item the general kernel and the z-marching kernel add in one order, so that the choice between them may follow the batch: a sample's bits are those it
    has alone."""
    S = D * H * W
    x = synth.rng(361).standard_normal(N * Ci * S).astype(np.float32) * np.exp2(synth.rng(362).integers(-6, 7, N * Ci * S)).astype(np.float32)
    w, b = synth.kaiming(363, Co, Ci, 27), synth.bias(364, Co, 0.1)
    got = run("conv3", orc.pm_to_mx(x, 0, N, Ci, S, bits, 32), w, b, N, Ci, D, H, W, Co, bits, kernels[1])
    alone = run("conv3", orc.pm_to_mx(x[-Ci * S:], 0, 1, Ci, S, bits, 32), w, b, 1, Ci, D, H, W, Co, bits, kernels[0])
    assert np.isfinite(got).all() and np.array_equal(got.reshape(N, -1)[-1], alone.reshape(-1))


@pytest.mark.parametrize("Ci,bits,kernel", [(64, 8, 0), (32, 8, 1), (64, 4, 1)])
def test_network_layers_keep_their_order_of_sums(dev, Ci, bits, kernel):
    """Rows that TMA does not take, blocked halves out (a network's layer): several MX-fp8 input items are added item by item, by the general kernel, at every size.  The planes that a
    volume of the first six has in common with the whole one have its bits, although the general kernel takes the small one in every case; and the halves are the oracle's."""
    N, Co, D, H, W, d = 1, 32, 40, 64, 40, 6
    S, s = D * H * W, d * H * W
    x = synth.rng(371).standard_normal(N * Ci * S).astype(np.float32) * np.exp2(synth.rng(374).integers(-6, 7, N * Ci * S)).astype(np.float32)
    w, b = synth.kaiming(372, Co, Ci, 27), synth.bias(373, Co, 0.1)
    c = G.Conv("conv3", w, b, Co, Ci, bits)
    mx, want = orc.conv_case("conv3", x, w, b, N, Ci, D, H, W, Co, bits)
    y, _ = c.fwd(mx, N, D, H, W, G.OUT_H16B)
    assert dev.umx_conv_last_kernel() == kernel
    z, _ = c.fwd(orc.pm_to_mx(np.ascontiguousarray(x.reshape(Ci, S)[:, :s]).reshape(-1), 0, N, Ci, s, bits, 32), N, d, H, W, G.OUT_H16B)
    assert dev.umx_conv_last_kernel() == 0
    c.free()
    y, z, same = y.view(np.float16), z.view(np.float16), (d - 1) * H * W * 32
    assert np.array_equal(y[:same], z[:same])
    e = orc.rel_l2(y.astype(np.float32), orc.pm_to_blocked(want, N, Co, S))
    assert np.isfinite(y).all() and e < TOL, "relative L2 %.3g" % e
