"""Fused launches in which the CTAs of a row-wise operator beside a tensor-memory operator take runs of blocks."""
import numpy as np
import pytest

import bfuse_project_b200 as bf
from bfuse_project_b200 import workloads as wl
from test_gpu_b_pairs import run_and_check

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rt():
    r = bf.Runtime(0)
    yield r
    r.close()


# enough blocks for runs of 2, 4 and more; a last run cut short, a last block of fewer rows, rows wider than a warp
@pytest.mark.parametrize("row", [
    lambda rng: wl.softmax("sm", rng, 7001, 512, 0.125),
    lambda rng: wl.softmax("sm", rng, 6145, 1024, 0.125),
    lambda rng: wl.softmax("sm", rng, 20000, 128, 1.0),
    lambda rng: wl.layernorm("ln", rng, 5003, 768, 1e-5, residual=True),
    lambda rng: wl.rmsnorm("rms", rng, 4501, 2048, 1e-5),
    lambda rng: wl.rope("rope", rng, 4099, 8, 128, 500000.0),
])
@pytest.mark.parametrize("pattern", [(bf.ZIGZAG, 1, 1), (bf.RANGE_SPLIT, 0, 0)])
def test_runs_equal_one_block_per_cta(rt, row, pattern):
    rng = np.random.default_rng(11)
    g = wl.gemm("g", rng, bf.OP_GEMM_TF32, 2, 200, 256, 64, causal=True, w_std=1.0, bn=256, split=1)   # a window of half an SM
    for a, b in ((row(rng), g), (g, row(rng))):
        pair = run_and_check(rt, wl.PairSpec("runs", a, b, "tf32", "hbm"), [pattern])
        f = pair.fusion(*pattern)
        info = rt.fusion_info(f)
        assert info["launched_ctas"] < info["GridDim"][0]
        assert len(rt.trace_fused(f)[0]) == info["GridDim"][0]


def test_runs_of_clusters(rt):
    """A k-split GEMM: its partner's CTAs are dealt in clusters, a run to each."""
    rng = np.random.default_rng(12)
    g = wl.gemm("g", rng, bf.OP_GEMM_TF32, 1, 256, 256, 1024, w_std=0.05, bn=128, split=4)
    pair = run_and_check(rt, wl.PairSpec("runs", wl.softmax("sm", rng, 7001, 512, 0.125), g, "tf32", "hbm"), [(bf.ZIGZAG, 1, 1), (bf.RANGE_SPLIT, 0, 0)])
    info = rt.fusion_info(pair.fusion(bf.ZIGZAG, 1, 1))
    assert info["launched_ctas"] < info["GridDim"][0]


@pytest.mark.parametrize("split", [1, 4])
@pytest.mark.parametrize("pattern", [(bf.ZIGZAG, 1, 1), (bf.ZIGZAG, 3, 2), (bf.PROPORTIONAL, 3, 0), (bf.SM_STRIPED, 0, 0), (bf.SM_STRIPED, 37, 0),
                                     (bf.RANGE_SPLIT, 0, 0)])
def test_slots_describe_the_launch(rt, pattern, split):
    """Block map, trace and timeline of a launch whose CTAs take runs: every block of both operators in exactly one slot,
    a run in consecutive slots on one SM with its CTA's time marks, as many CTAs as the fusion says it launches."""
    rng = np.random.default_rng(13)
    g = wl.gemm("g", rng, bf.OP_GEMM_TF32, 1, 256, 256, 1024, w_std=0.05, bn=128, split=split)
    rows = wl.layernorm("ln", rng, 5003, 768, 1e-5)
    for order in ((rows, g), (g, rows)):
        pair = run_and_check(rt, wl.PairSpec("runs", *order, "tf32", "hbm"), [pattern])
        f = pair.fusion(*pattern)
        info = rt.fusion_info(f)
        row = order.index(rows)
        per = info["blocks_per_cta"][row]
        blocks = [k.launch[0][0] * k.launch[0][1] * k.launch[0][2] for k in order]
        assert per > 1 and info["blocks_per_cta"][1 - row] == 1 and info["launched_ctas"] < info["GridDim"][0]
        kern, vb, sm = rt.trace_fused(f)
        used = sum(blocks)
        assert (kern[used:] == -1).all() and used <= len(kern) < used + 2 * split
        for k in range(2):
            assert sorted(vb[kern == k].tolist()) == list(range(blocks[k]))
        for i in range(len(kern)):
            assert rt.map_block(f, i) == (None if i >= used else (int(kern[i]), int(vb[i])))
        marks = rt.fused_timeline([f])[0]
        assert (marks[:used] > 0).all() and (marks[:, 0] <= marks[:, 1]).all() and (marks[:, 1] <= marks[:, 2]).all()
        where = np.nonzero(kern == row)[0]
        for lo in range(0, blocks[row], per):
            slots = where[lo:lo + per]      # an operator's blocks are handed out in ascending order
            assert (np.diff(slots) == 1).all() and (vb[slots] == np.arange(lo, lo + len(slots))).all()
            assert len(set(sm[slots].tolist())) == 1 and (marks[slots] == marks[slots[0]]).all()


@pytest.mark.parametrize("cols", [128, 1024])
def test_rows_of_infinities_and_nan_beside_finite_ones(rt, cols):
    """Softmax rows taken two at a time: a row without a finite value, with an infinity or a NaN, or masked but for one value
    writes what it writes alone, and the rows that share its thread or its warp are not touched."""
    rng = np.random.default_rng(14)
    rows = wl.softmax("sm", rng, 6145, cols, 0.125)
    x = rows.host[0]
    x[0] = -np.inf
    x[5, 3] = np.nan
    x[9, :-1] = -np.inf
    x[64, 7] = np.inf
    x[65] = np.finfo(np.float32).min
    x[6144] = np.nan
    odd = [0, 5, 64, 6144]
    g = wl.gemm("g", rng, bf.OP_GEMM_TF32, 2, 200, 256, 64, causal=True, w_std=1.0, bn=256, split=1)
    pair = run_and_check(rt, wl.PairSpec("odd", rows, g, "tf32", "hbm"), [(bf.ZIGZAG, 1, 1)], check_oracle=False)
    info = rt.fusion_info(pair.fusion(bf.ZIGZAG, 1, 1))
    assert info["blocks_per_cta"][0] >= 2
    y = pair.read_outputs()[0][0]
    ok = np.ones(len(y), bool)
    ok[odd] = False
    assert not np.isfinite(y[odd]).all(1).any()
    assert np.abs(y[ok].sum(1) - 1).max() <= 1e-5 and y[9, -1] == 1 and np.allclose(y[65], 1 / cols, rtol=1e-5)
