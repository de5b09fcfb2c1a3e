"""The narrowing convolutions at the edges of their tiles, against the oracle: 8-pixel-wide tiles with shared rows (ragged
maps, several channel blocks, weights resident or not, 64- and 128-column tiles, masks and side codes), the thin layer's
operands of 32-byte rows, the gradient-and-update call, and the short roundings of the stand-alone kernels."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from niti_b200 import ops, ti_torch  # noqa: E402
from niti_b200._lib import lib  # noqa: E402
from niti_b200.compat import cutlassconv_cuda  # noqa: E402
from oracle import niti_oracle as O  # noqa: E402
from oracle import philox  # noqa: E402
from tests.test_gpu_launch_forms import Layer, kernels  # noqa: E402

DEV = "cuda:0"


def rnd8(rng, shape):
    return rng.integers(-127, 128, size=shape).astype(np.int8)


def cu(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(DEV)


def same(got, want):
    assert np.array_equal(got.cpu().numpy(), want)


@pytest.mark.parametrize("N,H,W,C,K", [
    (1, 16, 8, 16, 16), (2, 17, 9, 48, 80), (1, 33, 31, 32, 64), (3, 15, 13, 144, 64), (2, 20, 24, 128, 48), (1, 32, 32, 272, 128),
    (2, 12, 8, 64, 144), (5, 30, 16, 112, 112)])
@pytest.mark.parametrize("parking", [False, True])
@pytest.mark.parametrize("mode", [0, 1])
def test_tiles_that_share_rows(N, H, W, C, K, parking, mode):
    rng = np.random.default_rng(N + H + 3 * W + C + K)
    x, w, err = np.maximum(rnd8(rng, (N, H, W, C)), 0), rnd8(rng, (K, 3, 3, C)), rnd8(rng, (N, H, W, K))
    seed, ea = ops.seed_tensor(9, DEV), torch.zeros((), dtype=torch.int32, device=DEV)
    acc, back = O.conv_fprop(x, w), O.conv_dgrad(err, w)
    want = O.relu_fwd(O.act_calc(acc, 0, mode, philox.random_u32_tensor(9, 3, acc.shape))[0])
    want_e = np.where(x > 0, O.err_calc(back, mode, philox.random_u32_tensor(9, 4, back.shape))[0], 0).astype(np.int8)
    old = ops.set_accumulator_parking(parking)
    try:
        fwd, bwd = ops.new_requant_state(DEV), ops.new_requant_state(DEV)
        nbytes = ops.conv_dgrad_side_bytes(N, H, W, C, K, 3, 3, 1)
        side = torch.empty(nbytes, dtype=torch.uint8, device=DEV) if nbytes else None
        for _ in range(2):  # a streaming layer guesses wrong first and right afterwards
            same(ops.conv_fprop_fused(cu(x), cu(w), fwd, 1, mode, seed, 3, 0, True, ea, ea)[0], want)
            same(ops.conv_dgrad_fused(cu(err), cu(w), bwd, 1, mode, seed, 4, 0, ea, ea, relu_mask=cu(x), side=side)[0], want_e)
    finally:
        ops.set_accumulator_parking(old)
    ops.check_status(DEV)


@pytest.mark.parametrize("N,H,W,C,K", [(2, 18, 8, 16, 16), (1, 22, 16, 144, 64), (3, 26, 8, 48, 80), (2, 30, 4, 128, 128), (1, 38, 2, 32, 272),
                                       (4, 20, 8, 64, 48)])
@pytest.mark.parametrize("mode", [0, 1])
def test_pooling_in_the_same_launch_on_maps_of_any_even_height(N, H, W, C, K, mode):
    """Maps whose height does not split into tiles of an even number of rows (18, 22, 26, 30, 38) pool in the launch too."""
    assert ops.conv_fprop_pool_fused_supported(N, H, W, C, K, 3, 3, 1)
    rng = np.random.default_rng(N + H + W + C + K)
    x, w = rnd8(rng, (N, H, W, C)), rnd8(rng, (K, 3, 3, C))
    ea, st = torch.zeros((), dtype=torch.int32, device=DEV), ops.new_requant_state(DEV)
    y8, yp, _, _ = ops.conv_fprop_pool_fused(cu(x), cu(w), st, 1, mode, ops.seed_tensor(9, DEV), 3, 0, True, ea, ea)
    acc = O.conv_fprop(x, w)
    want = O.relu_fwd(O.act_calc(acc, 0, mode, philox.random_u32_tensor(9, 3, acc.shape))[0])
    same(y8, want)
    same(yp, O.maxpool_fwd(want))
    ops.check_status(DEV)


@pytest.mark.parametrize("N,H,W,C,K", [
    (1, 8, 8, 512, 512), (32, 4, 4, 272, 512),    # eight and four thread blocks to a tile; tiles of 64 and of 128 pixels
    (1, 16, 16, 384, 512),                        # four (16-pixel rows: pooling leaves a block whole pairs of image rows)
    (20, 8, 8, 144, 272), (70, 10, 10, 240, 112), # four; two, in tiles of 100 pixels
    (1, 3, 5, 288, 208), (3, 2, 2, 144, 512), (2, 2, 130, 192, 176)])
@pytest.mark.parametrize("mode,offset", [(0, 0), (1, 0), (1, 5), (2, 0)])
def test_tiles_that_share_a_reduction(N, H, W, C, K, mode, offset):
    """So few tiles that a cluster of thread blocks works on each: rows, columns and reduction blocks that do not divide evenly,
    masks, pooling, every rounding, and random words that start inside a block of four."""
    rng = np.random.default_rng(N + H + 3 * W + C + K)
    x, w, err = np.maximum(rnd8(rng, (N, H, W, C)), 0), rnd8(rng, (K, 3, 3, C)), rnd8(rng, (N, H, W, K))
    seed, ea = ops.seed_tensor(9, DEV), torch.full((), 3, dtype=torch.int32, device=DEV)
    acc, back = O.conv_fprop(x, w), O.conv_dgrad(err, w)
    y, _, shift = O.act_calc(acc, 0, mode, philox.random_u32_tensor(9, 3, acc.shape, offset))
    e, shift_e = O.err_calc(back, mode, philox.random_u32_tensor(9, 4, back.shape, offset))
    fwd, bwd = ops.new_requant_state(DEV), ops.new_requant_state(DEV)
    for relu in (False, True):
        want = O.relu_fwd(y) if relu else y
        got, exp, _ = ops.conv_fprop_fused(cu(x), cu(w), fwd, 1, mode, seed, 3, offset, relu, ea, ea)
        same(got, want)
        assert int(exp) == shift + 6
        if ops.conv_fprop_pool_fused_supported(N, H, W, C, K, 3, 3, 1):
            got, pooled, exp, _ = ops.conv_fprop_pool_fused(cu(x), cu(w), fwd, 1, mode, seed, 3, offset, relu, ea, ea)
            same(got, want)
            same(pooled, O.maxpool_fwd(want))
    for mask in (None, cu(x)):
        got, exp, _ = ops.conv_dgrad_fused(cu(err), cu(w), bwd, 1, mode, seed, 4, offset, ea, ea, relu_mask=mask)
        same(got, e if mask is None else np.where(x > 0, e, 0).astype(np.int8))
        assert int(exp) == shift_e + 6
    ops.check_status(DEV)


def test_more_than_2_to_the_31_output_rows():
    """16 channels in and out, 34 GB each: images at both ends and in the middle come out as they do alone, the others stay zero."""
    N, C = (1 << 21) + 5, 16
    torch.cuda.empty_cache()
    if torch.cuda.mem_get_info()[0] < (80 << 30):
        pytest.skip("needs 80 GB of device memory")
    rng = np.random.default_rng(8)
    few, w, at = cu(rnd8(rng, (4, 32, 32, C))), cu(rnd8(rng, (16, 3, 3, C))), [0, 1 << 20, N - 2, N - 1]
    ea = torch.zeros((), dtype=torch.int32, device=DEV)
    want = ops.conv_fprop_fused(few, w, ops.new_requant_state(DEV), 1, 0, None, 0, 0, False, ea, ea)[0]
    x = torch.zeros((N, 32, 32, C), dtype=torch.int8, device=DEV)
    x[at] = few
    got = ops.conv_fprop_fused(x, w, ops.new_requant_state(DEV), 1, 0, None, 0, 0, False, ea, ea)[0]
    ops.check_status(DEV)
    assert torch.equal(got[at], want)
    got[at] = 0
    assert not any(bool(part.any()) for part in got.split(1 << 17))
    del x, got
    torch.cuda.empty_cache()


@pytest.mark.parametrize("C,K", [(128, 128), (64, 64), (256, 64), (144, 128)])  # weights resident, weights in the ring; two tile widths
def test_stage_cap_reaches_the_kernels_that_share_rows(C, K):
    """NITI_OPT_STAGE_CAP: the same bytes from a ring of one, two or all stages, and with one stage, where every load waits for
    the products of the stage before it, a longer time (more than twice; a tenth is asserted)."""
    rng = np.random.default_rng(C + K)
    x, w, ea = cu(rnd8(rng, (40, 32, 32, C))), cu(rnd8(rng, (K, 3, 3, C))), torch.zeros((), dtype=torch.int32, device=DEV)
    old, out, times = ops.set_accumulator_parking(False), [], []
    try:
        for cap in (0, 2, 1):
            lib.niti_set_option(3, cap)
            st = ops.new_requant_state(DEV)
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            for i in range(60):
                if i == 20:
                    a.record()
                y = ops.conv_fprop_fused(x, w, st, 1, 0, None, 0, 0, False, ea, ea)[0]
            b.record()
            b.synchronize()
            out.append(y)
            times.append(a.elapsed_time(b))
    finally:
        lib.niti_set_option(3, 0)
        ops.set_accumulator_parking(old)
    assert torch.equal(out[0], out[1]) and torch.equal(out[0], out[2])
    assert times[2] > 1.1 * times[0], times
    ops.check_status(DEV)


@pytest.mark.parametrize("N,H,W,C,K", [(80, 32, 32, 144, 48), (90, 30, 28, 272, 64), (76, 32, 32, 160, 112), (90, 30, 28, 144, 128)])
@pytest.mark.parametrize("mode", [0, 1])
def test_tiles_that_share_rows_over_several_rounds_of_the_ring(N, H, W, C, K, mode):
    """More than four tiles per thread block with the weights in the ring: accumulators and stages are used again, 64-column
    tiles are dealt to two pairs of warp groups.  Against the int32 products, narrowed by the stand-alone kernel."""
    rng = np.random.default_rng(N + C + K)
    x, w, err = cu(np.maximum(rnd8(rng, (N, H, W, C)), 0)), cu(rnd8(rng, (K, 3, 3, C))), cu(rnd8(rng, (N, H, W, C)))
    wb = cu(rnd8(rng, (C, 3, 3, K)))  # error-backward of a layer K -> C has K output columns
    mask = cu(rnd8(rng, (N, H, W, K)))
    seed, ea = ops.seed_tensor(9, DEV), torch.zeros((), dtype=torch.int32, device=DEV)
    want, e, s = ops.requant(*ops.conv_fprop_acc(x, w), ops.CALC_ACT, 7, mode, seed, 3, relu=True, exp_a=ea, want_shift=True)
    want_b = ops.relu_bwd(mask, ops.requant(*ops.conv_dgrad_acc(err, wb), ops.CALC_ERR, 7, mode, seed, 4)[0])
    old = ops.set_accumulator_parking(False)
    try:
        fwd, bwd = ops.new_requant_state(DEV), ops.new_requant_state(DEV)
        side = torch.empty(ops.conv_dgrad_side_bytes(N, H, W, K, C, 3, 3, 1), dtype=torch.uint8, device=DEV)
        for _ in range(2):
            y, ey, sy = ops.conv_fprop_fused(x, w, fwd, 1, mode, seed, 3, 0, True, ea, None)
            assert torch.equal(y, want) and int(ey) == int(e) and int(sy) == int(s)
            assert torch.equal(ops.conv_dgrad_fused(err, wb, bwd, 1, mode, seed, 4, 0, None, None, relu_mask=mask, side=side)[0], want_b)
    finally:
        ops.set_accumulator_parking(old)
    ops.check_status(DEV)


@pytest.mark.parametrize("K", [16, 112, 272])  # one column tile of 64, of 128, two of 256
@pytest.mark.parametrize("parking", [False, True])
@pytest.mark.parametrize("mode", [0, 1, 2])
def test_accumulators_that_need_no_shift(K, parking, mode):
    """A maximum of 128 has 7 bits: the low bytes as they are, so that 128 wraps to -128 (and ends as 0 behind a ReLU)."""
    rng = np.random.default_rng(K)
    x, w = np.zeros((2, 9, 10, 16), np.int8), rng.integers(-2, 3, size=(K, 3, 3, 16)).astype(np.int8)
    x[0, 2, 2, 0], x[1, 6, 7, 3], x[1, 1, 1, 5] = 64, -64, 9
    acc = O.conv_fprop(x, w)
    assert np.abs(acc).max() == 128 and O.act_calc(acc, 0)[2] == 0
    err = np.zeros((2, 9, 10, K), np.int8)
    err[0, 2, 2, 0], err[1, 6, 7, K - 1], err[1, 1, 1, 5] = 64, -64, 9
    back = O.conv_dgrad(err, w)
    assert np.abs(back).max() == 128
    seed, z = ops.seed_tensor(9, DEV), torch.zeros((), dtype=torch.int32, device=DEV)
    old = ops.set_accumulator_parking(parking)
    try:
        for relu in (False, True):
            st = ops.new_requant_state(DEV)
            for _ in range(2):
                y, _, shift = ops.conv_fprop_fused(cu(x), cu(w), st, 1, mode, seed, 3, 0, relu, z, z)
                same(y, np.maximum(O.wrap_int8(acc), 0) if relu else O.wrap_int8(acc))
                assert int(shift) == 0
        e, _, shift = ops.conv_dgrad_fused(cu(err), cu(w), ops.new_requant_state(DEV), 1, mode, seed, 4, 0, z, z)
        same(e, O.wrap_int8(back))
        assert int(shift) == 0
    finally:
        ops.set_accumulator_parking(old)
    ops.check_status(DEV)


@pytest.mark.parametrize("N,H,W,K", [(1, 1, 1, 16), (1, 4, 4, 16), (3, 7, 12, 80), (2, 5, 9, 144), (9, 32, 32, 48), (1, 3, 260, 64)])
def test_thin_layer(N, H, W, K):
    """Rows of whole words take the staged gather, the others the general one; fewer pixels than a tile; 16 to 144 filters."""
    rng = np.random.default_rng(N + H + W + K)
    x, w, err = rnd8(rng, (N, H, W, 3)), rnd8(rng, (K, 3, 3, 3)), rnd8(rng, (N, H, W, K))
    ea, st = torch.zeros((), dtype=torch.int32, device=DEV), ops.new_requant_state(DEV)
    acc = O.conv_fprop(x, w)
    for _ in range(2):
        same(ops.conv_fprop_fused(cu(x), cu(w), st, 1, 0, None, 0, 0, False, ea, ea)[0], O.act_calc(acc, 0)[0])
    same(ops.conv_fprop_acc(cu(x), cu(w))[0], acc)
    same(ops.conv_wgrad_acc(cu(x), cu(err), 3, 3, 1)[0], O.conv_wgrad(x, err, 3, 3, 1))


@pytest.mark.parametrize("N,H,W", [(1, 1, 4), (3, 6, 10), (2, 5, 7), (40, 32, 32)])
def test_input_quantisation_of_three_planes(N, H, W):
    x = np.random.default_rng(N + H + W).standard_normal((N, 3, H, W)).astype(np.float32)
    want, want_e = O.float_to_int8(x)
    got, e = ops.quantize_input(cu(x))
    same(got, np.ascontiguousarray(want.transpose(0, 2, 3, 1)))
    assert int(e) == want_e


@pytest.mark.parametrize("N,H,W,C,K,mode", [(2, 5, 7, 16, 16, 2), (3, 8, 8, 48, 80, 2), (1, 4, 4, 144, 128, 1),
                                            (7, 4, 4, 512, 528, 2), (1, 2, 2, 1040, 1024, 2)])  # more weights than stay in registers; two waves
def test_gradient_and_update_in_one_call(N, H, W, C, K, mode):
    rng = np.random.default_rng(N + C + K)
    x, w, err = rnd8(rng, (N, H, W, C)), rnd8(rng, (K, 3, 3, C)), rnd8(rng, (N, H, W, K))
    g = O.conv_wgrad(x, err, 3, 3, 1)
    wd = cu(w)
    g32, mx = ops.conv_wgrad_update(cu(x), cu(err), wd, 1, 5, mode, ops.seed_tensor(7, DEV), 18)
    same(g32, g)
    assert int(mx) == int(np.abs(g).max())
    same(wd, O.weight_update(w, g, 5, mode, philox.random_u32_tensor(7, 18, g.shape))[0])
    # the same in one launch, over the layer's own words, which every call leaves zero
    st = ops.new_update_state(DEV)
    for _ in range(2):
        w1 = cu(w)
        g1, m1 = ops.conv_wgrad_update(cu(x), cu(err), w1, 1, 5, mode, ops.seed_tensor(7, DEV), 18, st)
        same(g1, g)
        assert torch.equal(w1, wd) and int(m1) == int(mx) and not bool(st.any())
    ops.check_status(DEV)
    # operands that do not start on a 16-byte boundary are served too, as by the separate calls
    odd = torch.empty(x.size + 1, dtype=torch.int8, device=DEV)[1:].view(x.shape)
    odd.copy_(cu(x))
    w2 = cu(w)
    same(ops.conv_wgrad_update(odd, cu(err), w2, 1, 5, mode, ops.seed_tensor(7, DEV), 18)[0], g)
    assert torch.equal(w2, wd)


@pytest.mark.parametrize("n", [1, 3, 16, 2055, 300001])
@pytest.mark.parametrize("top", [0, 90, 129, 1 << 15, (1 << 30) - 1, (1 << 31) - 1])
def test_roundings_of_the_stand_alone_kernels(n, top):
    """All three roundings from no shift at all to accumulators that fill 31 bits (the short forms end at 30)."""
    rng = np.random.default_rng(n + top % 97)
    acc = rng.integers(-top, top + 1, size=n).astype(np.int32)
    acc[rng.integers(n)] = top
    mx, seed = ops.absmax(cu(acc)), ops.seed_tensor(5, DEV)
    for mode in (0, 1, 2):
        words = philox.random_u32_tensor(5, 2, acc.shape)
        same(ops.requant(cu(acc), mx, ops.CALC_ACT, 7, mode, seed, 2)[0], O.act_calc(acc, 0, mode, words)[0])
        w = rnd8(rng, (n,))
        wd = cu(w)
        ops.update(wd, cu(acc), mx, 5, mode, seed, 2)
        same(wd, O.weight_update(w, acc, 5, mode, words)[0])


@pytest.mark.parametrize("n", [1, 4, 6, 1023, 4096])
@pytest.mark.parametrize("shift", [1, 4, 10, 23])
def test_roundings_by_a_shift_that_the_data_exceed(n, shift):
    """RoundShift and StoShift take any shift, niti_requant_i8 any target width: int32 values whose rounded quotients (and
    whose sums with half a unit) pass both ends of the range are clamped like all others, in whole words and in the tail."""
    rng = np.random.default_rng(n + shift)
    lim = np.iinfo(np.int32)
    x = rng.choice(np.array([lim.max, lim.max - (1 << shift >> 1), lim.max - (1 << shift) + 2, (127 << shift) + 1, 127 << shift, 5, 0, -5,
                             -(127 << shift) - 1, lim.min + (1 << shift), lim.min + 1, lim.min], dtype=np.int32), size=n)
    words = philox.random_u32_tensor(3, 0, x.shape)
    ti_torch.set_seed(3, DEV)
    same(ti_torch.RoundShift(cu(x), shift), O.round_shift(x, shift))
    same(ti_torch.StoShift(cu(x), shift), O.sto_shift(x, shift, words))
    same(ti_torch.PstoShift(cu(x), shift), O.psto_shift(x, shift))
    same(ops.requant(cu(x), cu(np.array([lim.max], np.int32)), ops.CALC_ACT, 31 - shift, 0, relu=True)[0], np.maximum(O.round_shift(x, shift), 0))


@pytest.mark.parametrize("M,N,K,ta,tb", [
    (4097, 50, 128, False, True), (700, 10, 2448, False, True), (1000, 101, 256, False, True), (513, 1024, 50, False, False),
    (10, 2064, 1003, True, False), (99, 512, 500, True, False), (130, 4096, 33, True, False)])
def test_products_of_any_row_pitch(M, N, K, ta, tb):
    rng = np.random.default_rng(M + N + K)
    a, b = rnd8(rng, (M, K)), rnd8(rng, (K, N))
    want = O.int8_mm(a, b)
    c, mx = ops.gemm_acc(cu(a.T if ta else a), cu(b.T if tb else b), ta, tb)
    same(c, want)
    assert int(mx) == int(np.abs(want).max())
    ops.check_status(DEV)


def test_launches_are_counted_by_shape():
    """Gather, product and conditional second launch of a thin layer; row copies of a padded product and none of others."""
    def counted(fn, *args):
        before = ops.LAUNCHES
        fn(*args)
        return ops.LAUNCHES - before

    rng = np.random.default_rng(0)
    z = torch.zeros((), dtype=torch.int32, device=DEV)
    for C, fused, grad in ((3, 3, 3), (16, 2, 2)):
        x, w, err = cu(rnd8(rng, (2, 8, 8, C))), cu(rnd8(rng, (16, 3, 3, C))), cu(rnd8(rng, (2, 8, 8, 16)))
        assert counted(ops.conv_fprop_fused, x, w, ops.new_requant_state(DEV), 1, 0, None, 0, 0, False, z, z) == fused
        assert counted(ops.conv_wgrad_acc, x, err) == grad
    for M, N, K, ta, tb, n in [(500, 1024, 100, False, False, 2), (1000, 101, 256, False, True, 2), (700, 33, 1000, False, True, 1),
                               (99, 1024, 500, True, False, 2), (64, 64, 64, False, True, 1), (5, 3, 7, False, False, 1)]:
        a, b = rnd8(rng, (K, M) if ta else (M, K)), rnd8(rng, (N, K) if tb else (K, N))
        assert counted(ops.gemm_acc, cu(a), cu(b), ta, tb) == n, (M, N, K)


@pytest.mark.parametrize("N,H,W,C,K", [(16, 5, 7, 32, 48), (32, 4, 4, 144, 128)])
def test_partial_sums_instead_of_reductions_in_every_weight_gradient(N, H, W, C, K):
    """NITI_OPT_WGRAD_TMA_REDUCE = 0 sends the update call and the batch-innermost form through niti_conv_wgrad_i8."""
    rng = np.random.default_rng(N + C)
    x, w, err = rnd8(rng, (N, H, W, C)), rnd8(rng, (K, 3, 3, C)), rnd8(rng, (N, H, W, K))
    g, wd = O.conv_wgrad(x, err, 3, 3, 1), cu(w)
    old = lib.niti_set_option(2, 0)
    ops.PROFILE = []
    try:
        g32, mx = ops.conv_wgrad_update(cu(x), cu(err), wd, 1, 5, 2, None, 18)
        dis = cutlassconv_cuda.sp_conv_optimized(cu(x.transpose(3, 1, 2, 0)), cu(err.transpose(3, 1, 2, 0)), 1, 1)
        names = [p[0] for p in ops.PROFILE]
    finally:
        ops.PROFILE = None
        lib.niti_set_option(2, old)
    assert names == ["niti_conv_wgrad_i8", "niti_update_i8", "niti_conv_wgrad_i8"]
    same(g32, g)
    assert int(mx) == int(np.abs(g).max())
    same(wd, O.weight_update(w, g, 5, 2)[0])
    same(dis, g.transpose(3, 1, 2, 0))


@pytest.mark.parametrize("N,H,W,C,K,forward,pooled,backward", [
    (1, 8, 8, 512, 512, 8, 8, 8), (1, 16, 16, 384, 512, 8, 4, 8),  # 16-pixel rows: a block of a pooling call keeps pairs of them
    (12, 8, 8, 256, 512, 4, 4, 8), (20, 8, 8, 400, 512, 2, 2, 2),
    (75, 4, 4, 384, 496, 2, 2, 4), (44, 5, 7, 400, 272, 2, 0, 2)])  # tiles of 105 pixels, maps that no pool divides
def test_as_many_thread_blocks_to_a_tile_as_the_rule_says(N, H, W, C, K, forward, pooled, backward):
    """Eight, four and two thread blocks to a tile, in both directions and with pooling, whatever the rounding; results as above."""
    seed, layer = ops.seed_tensor(9, DEV), Layer(N, H, W, C, K)
    O.set_backend("int_mm")
    try:
        for mode in (0, 1, 2):
            def call(fn, x, *more):
                st = ops.new_requant_state(DEV)
                return kernels(lambda: fn(x, layer.dw, st, 1, mode, seed, 3, 0, *more))
            assert call(ops.conv_fprop_fused, layer.dx, False, layer.z, layer.z) == [(True, forward)]
            assert call(ops.conv_dgrad_fused, layer.derr, layer.z, layer.z) == [(True, backward)]
            if pooled:
                assert call(ops.conv_fprop_pool_fused, layer.dx, False, layer.z, layer.z) == [(True, pooled)]
            else:
                assert not ops.conv_fprop_pool_fused_supported(N, H, W, C, K, 3, 3, 1)
            test_tiles_that_share_a_reduction(N, H, W, C, K, mode, 0)
    finally:
        O.set_backend("int64")


@pytest.mark.parametrize("offset", [(1 << 34) - 16, (1 << 34) + 64, (1 << 34) - 16 * 1001, (1 << 36) - 32, 3 << 40])
@pytest.mark.parametrize("N,H,W,C,K,parking", [(2, 9, 7, 48, 80, False), (2, 9, 7, 48, 80, True), (3, 8, 8, 128, 256, True),
                                               (3, 8, 8, 144, 64, False), (1, 8, 8, 512, 512, True)])
def test_random_words_where_their_block_number_leaves_32_bits(N, H, W, C, K, parking, offset):
    """A sample offset may put a tensor's elements anywhere in 64 bits: block numbers (four elements each) that carry into their high
    word inside a row of outputs, inside the tensor and before it, in the streaming, the parked and the shared kernels."""
    rng = np.random.default_rng(N + H + C + K)
    x, w, err = np.maximum(rnd8(rng, (N, H, W, C)), 0), rnd8(rng, (K, 3, 3, C)), rnd8(rng, (N, H, W, K))
    seed, z = ops.seed_tensor(9, DEV), torch.zeros((), dtype=torch.int32, device=DEV)
    acc, back = O.conv_fprop(x, w), O.conv_dgrad(err, w)
    want = O.act_calc(acc, 0, 1, philox.random_u32_tensor(9, 3, acc.shape, offset))[0]
    want_e = O.err_calc(back, 1, philox.random_u32_tensor(9, 4, back.shape, offset))[0]
    old = ops.set_accumulator_parking(parking)
    try:
        fwd, bwd = ops.new_requant_state(DEV), ops.new_requant_state(DEV)
        for _ in range(2):
            for relu in (False, True):
                same(ops.conv_fprop_fused(cu(x), cu(w), fwd, 1, 1, seed, 3, offset, relu, z, z)[0], np.maximum(want, 0) if relu else want)
            same(ops.conv_dgrad_fused(cu(err), cu(w), bwd, 1, 1, seed, 4, offset, z, z)[0], want_e)
    finally:
        ops.set_accumulator_parking(old)
    ops.check_status(DEV)
