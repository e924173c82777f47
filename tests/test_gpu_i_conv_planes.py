"""Convs staged as whole image planes (shape[11] = 3): 3 x 3 windows on images whose rows are no 16-byte multiples."""
import numpy as np
import pytest

import bfuse_project_b200 as bf
from bfuse_project_b200 import workloads as wl
from pair_oracle import check_against_oracle
from test_gpu_b_pairs import BLOCK_PATTERNS, run_and_check

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rt():
    r = bf.Runtime(0)
    yield r
    r.close()


# n, ci, h = w, co, stride, pad, k-slices
SHAPES = [
    (1, 32, 14, 40, 1, 1, 1),      # one image, a tile and a half; ragged channel tile
    (3, 64, 7, 128, 1, 1, 2),      # a tile over three images, the second one partly filled; one group of channels a slice
    (5, 128, 14, 136, 2, 1, 4),    # stride 2 on an even width (8-byte reads), tiles of whole images
    (4, 256, 7, 130, 1, 1, 8),     # eight slices
    (11, 64, 5, 128, 1, 0, 1),     # no padding: nine pixels an image, fifteen images a tile
    (9, 96, 10, 64, 2, 2, 1),      # padding 2
    (9, 96, 13, 64, 1, 2, 2),      # two slices of two and one channel groups
]


@pytest.mark.parametrize("n,ci,hw,co,stride,pad,split", SHAPES)
def test_planes_against_the_oracle_and_unfused(rt, n, ci, hw, co, stride, pad, split):
    """The tolerances are the tf32 conv's (pair_oracle); fused == unfused bit for bit."""
    rng = np.random.default_rng(ci + hw)
    a = wl.conv2d("planes", rng, bf.OP_CONV2D_TF32, n, ci, hw, hw, co, 3, stride, pad, bn=128, split=split, mode=3)
    b = wl.gemm("g", rng, bf.OP_GEMM_TF32, 1, 100, 64, 64, w_std=1.0, bn=64, split=1)
    run_and_check(rt, wl.PairSpec("planes", a, b, "tf32", "hbm"), BLOCK_PATTERNS if split == 1 else [(bf.ZIGZAG, 1, 1), (bf.RANGE_SPLIT, 0, 0)])
    if split == 1:
        run_and_check(rt, wl.PairSpec("planes_twice", a, a, "tf32", "hbm"), [(bf.WORK_QUEUE, 1, 1), (bf.THREAD_SPLIT, 0, 0)])


def test_the_runtime_takes_planes_for_small_images_of_a_batch(rt):
    def mode(n, ci, hw, co, flags=0):
        d = rt.describe("c", bf.OP_CONV2D_TF32, (n, ci, hw, hw, co, 3, 3, 1, 1, 0, 0, 0), flags=flags)
        return d.shape[11], d.shape[10]
    assert mode(32, 512, 7, 512, bf.flag_share(1)) == (3, 4) and mode(32, 256, 14, 256, bf.flag_share(1)) == (3, 1)
    assert mode(1, 512, 7, 512)[0] == 2 and mode(32, 128, 28, 128)[0] == 1      # a lone image; rows of 16-byte multiples


def test_planes_that_cannot_be_are_rejected(rt):
    for n, ci, hw, co, k, bn, split in ((4, 40, 7, 64, 3, 128, 1), (4, 64, 7, 64, 1, 128, 1), (4, 64, 7, 64, 3, 64, 1), (4, 64, 7, 64, 3, 128, 4), (4, 64, 62, 64, 3, 128, 1)):
        with pytest.raises(bf.BfuseError) as err:
            rt.describe("c", bf.OP_CONV2D_TF32, (n, ci, hw, hw, co, k, k, 1, k // 2, bn, split, 3))
        assert err.value.code == 2


def test_ctas_that_walk_several_tiles_and_values_outside_a_window(rt):
    """A grid smaller than the tile count writes the same bits; an infinity reaches only the windows that hold it,
    although a tap outside its image reads whatever lies beside the plane."""
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    n, ci, hw, co = 40, 32, 7, 136
    x = torch.randn(n, ci, hw, hw, device="cuda", generator=g)
    w = torch.randn(co, ci, 3, 3, device="cuda", generator=g) * 0.05
    outs = []
    for grid in (None, (3, 1, 1), (1, 1, 1)):
        y = torch.zeros(n, co, hw, hw, device="cuda")
        d = rt.describe("c", bf.OP_CONV2D_TF32, (n, ci, hw, hw, co, 3, 3, 1, 1, 128, 1, 3), [x.data_ptr(), w.data_ptr(), y.data_ptr()], grid=grid)
        k = rt.register_kernel(d)
        rt.launch_kernel(k)
        assert rt.read_status() == 0
        outs.append(y)
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    x[1, 3, 0, 0] = float("inf")                     # a corner: the next row's end and the next image's start lie beside it
    rt.launch_kernel(k)
    assert rt.read_status() == 0
    touched = torch.zeros(n, 1, hw, hw, dtype=torch.bool, device="cuda")
    touched[1, 0, :2, :2] = True
    assert torch.equal(outs[2][~touched.expand_as(outs[2])], outs[0][~touched.expand_as(outs[0])])
    assert not torch.isfinite(outs[2][1, :, :2, :2]).any()


@pytest.mark.parametrize("n,ci,hw,co,stride", [(8, 256, 14, 256, 1), (32, 64, 7, 96, 2), (32, 256, 14, 40, 1)])
def test_a_launch_recorded_for_the_gathered_form_is_still_accepted(rt, n, ci, hw, co, stride):
    """The runtime's choice is whole planes; a window too small for them, the gathered form's grid, or both register and run gathered."""
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(7)
    x = torch.randn(n, ci, hw, hw, device="cuda", generator=g)
    w = torch.randn(co, ci, 3, 3, device="cuda", generator=g) * 0.05
    o = (hw - 1) // stride + 1
    shape = (n, ci, hw, hw, co, 3, 3, stride, 1)
    # (registered at once: the planes' own launch and one that fits neither form)
    planes = rt.describe("c", bf.OP_CONV2D_TF32, shape + (128, 0, 3))
    gathered = rt.describe("c", bf.OP_CONV2D_TF32, shape + (0, 0, 2))

    def run(**launch):
        y = torch.zeros(n, co, o, o, device="cuda")
        sh = (0, 0, 2) if launch.pop("mode", 0) == 2 else (128, planes.shape[10], 3)
        k = rt.register_kernel(rt.describe("c", bf.OP_CONV2D_TF32, shape + sh, [x.data_ptr(), w.data_ptr(), y.data_ptr()], **launch))
        rt.launch_kernel(k)
        assert rt.read_status() == 0
        return y
    want = run(mode=2)
    grid = gathered.GridDim.tuple()
    for launch in (dict(smem=gathered.smem_bytes), dict(grid=grid), dict(grid=grid, smem=gathered.smem_bytes)):
        if launch.get("grid") and grid[0] * grid[1] * grid[2] <= planes.GridDim.size():
            continue   # a grid the planes can walk as it is
        assert torch.equal(run(**launch), want), launch
    for launch in (dict(smem=4096), dict(grid=(grid[0] + 1, grid[1], grid[2] + 1))):
        with pytest.raises(bf.BfuseError) as err:
            run(**launch)
        assert err.value.code == 2


def test_thread_split_beside_a_wide_window(rt):
    """Thread split lays both windows side by side: the planes' raw slots are given up first, and where even two of them do
    not fit beside the partner the conv runs gathered, as the fusion's own sequential mode does."""
    rng = np.random.default_rng(21)
    planes = wl.conv2d("planes", rng, bf.OP_CONV2D_TF32, 5, 128, 14, 14, 64, 3, 1, 1, bn=128, split=1, mode=3)
    rows = wl.conv2d("rows", rng, bf.OP_CONV2D_TF32, 2, 512, 28, 28, 128, 3, 1, 1, bn=128, split=1, mode=1)
    for smem, retiled in ((130 * 1024, False), (200 * 1024, True)):
        rows.smem = smem
        for order in ((planes, rows), (rows, planes)):
            pair = wl.DevicePair(rt, wl.PairSpec("wide", *order, "tf32", "hbm"))
            f = pair.fusion(bf.THREAD_SPLIT, 0, 0)
            info = rt.fusion_info(f)
            assert any(info["retiled_unsplit"]) == retiled, (smem, info)
            pair.clear_outputs()
            rt.launch_sequential(f)
            want = pair.read_outputs()
            pair.clear_outputs()
            rt.launch_fused(f)
            got = pair.read_outputs()
            assert rt.read_status() == 0
            for k, ks in enumerate(order):
                assert np.array_equal(want[k][0], got[k][0]), (smem, ks.name)
                check_against_oracle(ks, got[k], ks.name)


def test_planes_beside_an_operator_of_another_cluster_width(rt):
    """The runtime splits this conv in four slices as whole planes and would leave it unsplit gathered: beside a GEMM of two
    k-slices it runs in one, as a pair and in a group, and the records it needs for that are released with them."""
    rng = np.random.default_rng(22)
    conv = wl.conv2d("planes", rng, bf.OP_CONV2D_TF32, 8, 256, 14, 14, 256, 3, 1, 1)
    gemm = wl.gemm("g", rng, bf.OP_GEMM_TF32, 1, 100, 64, 1024, w_std=0.05, bn=64, split=2)
    pair = wl.DevicePair(rt, wl.PairSpec("widths", conv, gemm, "tf32", "hbm"))
    f = pair.fusion(bf.ZIGZAG, 1, 1)
    assert rt.fusion_info(f)["retiled_unsplit"] == (True, False)
    pair.clear_outputs()
    rt.launch_sequential(f)
    want = pair.read_outputs()
    check_against_oracle(conv, want[0], "planes")
    check_against_oracle(gemm, want[1], "gemm")
    g = rt.register_group([pair.kernels[1], pair.kernels[0]], bf.ZIGZAG, 1, 1)
    for launch in (lambda: rt.launch_fused(f), lambda: rt.launch_group(g)):
        pair.clear_outputs()
        launch()
        got = pair.read_outputs()
        assert rt.read_status() == 0
        assert np.array_equal(got[0][0], want[0][0]) and np.array_equal(got[1][0], want[1][0])
    with pytest.raises(bf.BfuseError):
        rt.unregister_kernel(pair.kernels[0])
    rt.unregister_group(g)
    rt.unregister_fusion(pair.fusions.pop((bf.ZIGZAG, 1, 1)))
    for k in pair.kernels:
        rt.unregister_kernel(k)
    # an explicit width that the gathered form would not have come without stays refused
    four = wl.conv2d("four", rng, bf.OP_CONV2D_TF32, 1, 512, 7, 7, 64, 3, 1, 1)
    pair = wl.DevicePair(rt, wl.PairSpec("widths", four, gemm, "tf32", "hbm"))
    with pytest.raises(bf.BfuseError) as err:
        pair.fusion(bf.ZIGZAG, 1, 1)
    assert err.value.code == 7


@pytest.mark.parametrize("n,ci,hw,co,stride,share", [(8, 256, 14, 130, 1, 2), (32, 128, 7, 64, 1, 2), (40, 64, 15, 96, 2, 2), (24, 128, 7, 256, 2, 3)])
def test_the_runtime_s_own_choice_against_the_oracle_and_in_a_group(rt, n, ci, hw, co, stride, share):
    """Shape fields left to the runtime: alone against the oracle, and beside a gathered conv and a GEMM in one launch, bit for bit."""
    rng = np.random.default_rng(ci + hw + n)
    planes = wl.conv2d("planes", rng, bf.OP_CONV2D_TF32, n, ci, hw, hw, co, 3, stride, 1)
    planes.flags = bf.flag_share(share)
    split = rt.describe("c", planes.op, planes.shape, flags=planes.flags).shape
    assert split[11] == 3
    beside = wl.conv2d("gathered", rng, bf.OP_CONV2D_TF32, 2, 32, 9, 9, 40, 3, 1, 1, bn=32, split=split[10], mode=2) if split[10] == 1 else \
        wl.conv2d("gathered", rng, bf.OP_CONV2D_TF32, 1, 256, 9, 9, 40, 3, 1, 1, bn=32, split=split[10], mode=2)
    gemm = wl.gemm("g", rng, bf.OP_GEMM_TF32, 1, 70, 64, 64, w_std=1.0, bn=64, split=1)
    pair = run_and_check(rt, wl.PairSpec("own", planes, beside, "tf32", "hbm"), [(bf.ZIGZAG, 1, 1)])
    other = wl.DevicePair(rt, wl.PairSpec("own", gemm, beside, "tf32", "hbm"))
    rt.launch_kernel(other.kernels[0])
    want = [pair.read_outputs(), other.read_outputs()]
    for p in (pair, other):
        p.clear_outputs()
    group = rt.register_group([pair.kernels[0], other.kernels[0], pair.kernels[1]], bf.ZIGZAG, 1, 1)
    rt.launch_group(group)
    got = [pair.read_outputs(), other.read_outputs()]
    assert rt.read_status() == 0
    assert np.array_equal(got[0][0][0], want[0][0][0]) and np.array_equal(got[0][1][0], want[0][1][0])
    assert np.array_equal(got[1][0][0], want[1][0][0])
