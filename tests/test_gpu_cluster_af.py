"""The cluster-resident autofocus engine (one thread-block cluster per frame,
distributed shared memory) against the FP64 oracle, through the C ABI."""
import numpy as np
import pytest

import oracle
from tests.helpers import golden_echo, make_frame, rel_l2
from tests.test_gpu_parity import TOL_IMG, ctx_for, from_dev, to_dev

pytestmark = pytest.mark.gpu


def _cut(M, N, seed, full=False):
    e, _ = make_frame(M, N, seed=seed, full=full)
    rp = oracle.radar(M, N)
    y, _ = oracle.range_align(e, rp)
    _, cut, _ = oracle.center_cut(y, rp)
    return cut.astype(np.complex64)


def _cluster_or_skip(ctx, cl):
    mx = ctx.tuning().af_cluster_max
    if cl > mx:
        pytest.skip("cluster of %d CTAs not launchable here (max %d)" % (cl, mx))


@pytest.mark.parametrize("cl", [4, 8, 16])
@pytest.mark.parametrize("M,N,seed", [(128, 512, 1), (256, 1024, 2), (512, 2048, 3), (1024, 2048, 4)])
def test_cluster_fast_entropy_matches_oracle(torch_cuda, gb300, M, N, seed, cl):
    torch = torch_cuda
    cut = _cut(M, N, seed)
    want, tw = oracle.fast_entropy(cut)
    with ctx_for(gb300, torch, M, N) as ctx:
        _cluster_or_skip(ctx, cl)
        ctx.set_tuning(af_cluster=cl)
        dc = to_dev(torch, cut)
        ctx.stage_fast_entropy(dc, 120)
        got = from_dev(torch, dc).reshape(M, 512)
        tr = ctx.trace()
    assert tr["unit2_num"] == tw["unit2_num"]
    assert np.array_equal(tr["bins"], tw["bins"])
    assert tr["af_iterations"] == 120
    assert np.isfinite(tr["af_entropy"])
    assert rel_l2(got, want) < TOL_IMG


def test_cluster_many_bins_reload_path(torch_cuda, gb300):
    """M = 1024 with U = 256 bins: a cluster of 4 caches 16 of each CTA's 64
    bins and reloads the rest every iteration."""
    torch = torch_cuda
    M = 1024
    rng = np.random.default_rng(5)
    cut = (rng.standard_normal((M, 512)) + 1j * rng.standard_normal((M, 512))).astype(np.complex64) * 300
    # 280 constant-magnitude bright bins -> tgt_num 280, U = 256
    cut[:, 100:380] = (6000 * np.exp(2j * np.pi * rng.random((M, 280)))).astype(np.complex64)
    want, tw = oracle.fast_entropy(cut, iters=10)
    assert tw["unit2_num"] == 256
    with ctx_for(gb300, torch, M, 2048) as ctx:
        _cluster_or_skip(ctx, 4)
        ctx.set_tuning(af_cluster=4)
        dc = to_dev(torch, cut)
        ctx.stage_fast_entropy(dc, 10)
        got = from_dev(torch, dc).reshape(M, 512)
        tr = ctx.trace()
    assert tr["unit2_num"] == tw["unit2_num"]
    assert rel_l2(got, want) < TOL_IMG


# Bins per CTA from none (U = 2 on 16 CTAs: most CTAs only take part in the
# exchange; half a warp owns a bin alone at 128 pulses) to more than the
# rounds kept in shared memory (U = 256 on 4 CTAs), at every transform split.  One
# update at U = 2: two bins of random phase are ill conditioned, further
# updates amplify any FP32 rounding.
@pytest.mark.parametrize("bright,U,iters", [(3, 2, 1), (9, 8, 8), (280, 256, 8)])
@pytest.mark.parametrize("M,cl", [(128, 4), (128, 16), (256, 4), (256, 16), (512, 4), (512, 8), (1024, 8), (1024, 16)])
def test_cluster_few_and_many_bins(torch_cuda, gb300, M, cl, bright, U, iters):
    torch = torch_cuda
    rng = np.random.default_rng(M + bright)
    cut = (rng.standard_normal((M, 512)) + 1j * rng.standard_normal((M, 512))).astype(np.complex64) * 100
    cut[:, 100:100 + bright] = (6000 * np.exp(2j * np.pi * rng.random((M, bright)))).astype(np.complex64)
    want, tw = oracle.fast_entropy(cut, iters=iters)
    assert tw["unit2_num"] == U
    with ctx_for(gb300, torch, M, 2048) as ctx:
        _cluster_or_skip(ctx, cl)
        ctx.set_tuning(af_cluster=cl)
        dc = to_dev(torch, cut)
        ctx.stage_fast_entropy(dc, iters)
        got = from_dev(torch, dc).reshape(M, 512)
        tr = ctx.trace()
    assert tr["unit2_num"] == U
    assert rel_l2(got, want) < TOL_IMG


# Engine 0, the cooperative grid, from few bins to 512 (profiles below one
# count, whose integer mean is 0): the oracle's result, and the trace's engine
# fields as engine 0 reports them.
@pytest.mark.parametrize("M", [128, 256, 512, 1024])
@pytest.mark.parametrize("bright,scale,U", [(40, 6000.0, 32), (280, 6000.0, 256), (512, 0.5, 512)])
def test_engine0_every_bin_count(torch_cuda, gb300, M, bright, scale, U):
    torch = torch_cuda
    rng = np.random.default_rng(3 * M + bright)
    cut = (rng.standard_normal((M, 512)) + 1j * rng.standard_normal((M, 512))).astype(np.complex64) * scale / 60
    k = (512 - bright) // 2
    cut[:, k:k + bright] = (scale * np.exp(2j * np.pi * rng.random((M, bright)))).astype(np.complex64)
    want, tw = oracle.fast_entropy(cut, iters=6)
    assert tw["unit2_num"] == U
    with ctx_for(gb300, torch, M, 2048) as ctx:
        ctx.set_tuning(af_cluster=0)
        dc = to_dev(torch, cut)
        ctx.stage_fast_entropy(dc, 6)
        got = from_dev(torch, dc).reshape(M, 512)
        tr = ctx.trace()
    assert tr["unit2_num"] == U and np.isnan(tr["af_entropy"])
    assert rel_l2(got, want) < TOL_IMG


# af_cluster 0 names the cooperative grid at every size (a poll limit of its own
# does not change the engine), and a 512-pulse context that was never tuned
# picks by bins: the 16-CTA cluster up to 256, the grid above.
@pytest.mark.parametrize("M", [128, 256, 512])
@pytest.mark.parametrize("bright,scale,U", [(40, 6000.0, 32), (280, 6000.0, 256), (512, 0.5, 512)])
def test_engine0_is_the_grid_and_the_default_picks_by_bins(torch_cuda, gb300, M, bright, scale, U):
    torch = torch_cuda
    rng = np.random.default_rng(5 * M + bright)
    cut = (rng.standard_normal((M, 512)) + 1j * rng.standard_normal((M, 512))).astype(np.complex64) * scale / 60
    k = (512 - bright) // 2
    cut[:, k:k + bright] = (scale * np.exp(2j * np.pi * rng.random((M, bright)))).astype(np.complex64)

    def run(cl=None, polls=0):
        with ctx_for(gb300, torch, M, 2048) as ctx:
            if cl is not None:
                _cluster_or_skip(ctx, cl)
                ctx.set_tuning(af_cluster=cl)
            ctx.test_barrier_timeout(polls, False)
            dc = to_dev(torch, cut)
            ctx.stage_fast_entropy(dc, 6)
            out = from_dev(torch, dc)
            tr = ctx.trace()
        assert tr["unit2_num"] == U
        return out, np.isnan(tr["af_entropy"])

    grid, none = run(0)
    assert none and np.array_equal(grid, run(0, polls=1 << 21)[0])
    cluster, none = run(16)
    assert not none and not np.array_equal(cluster, grid)
    if M == 512:
        out, none = run()
        assert none and np.array_equal(out, cluster if U <= 256 else grid)


# Row sums whose |s|^2 is a handful of the smallest float: it carries two
# roundings of half a unit, so at one unit s / |s| may be as long as sqrt(2), but
# the normalisation adds no error of its own.
@pytest.mark.parametrize("M", [128, 512, 1024])
def test_cluster_normalises_the_smallest_sums(torch_cuda, gb300, M):
    torch = torch_cuda
    rng = np.random.default_rng(M)
    base = np.exp(2j * np.pi * rng.random((M, 512)))
    a0 = (4e-23 / (512 * 1.3 * np.sqrt(M))) ** (1.0 / 3.0)   # |s| ~ 512 bins a^3 sqrt(M)
    seen = 0
    with ctx_for(gb300, torch, M, 2048) as ctx:
        _cluster_or_skip(ctx, 8)
        ctx.set_tuning(af_cluster=8)
        for k in range(-4, 5):
            dc = to_dev(torch, (base * a0 * 1.12 ** k).astype(np.complex64))
            ctx.stage_fast_entropy(dc, 1)
            torch.cuda.synchronize()
            r = np.abs(ctx.trace()["phase"].astype(np.complex128))
            r = r[np.isfinite(r)]
            seen += np.count_nonzero(np.abs(r - 1.0) > 0.1)   # sums of a few units are there
            assert np.all(r < np.sqrt(2.0) * (1.0 + 1e-5))
    assert seen > M // 16


def test_cluster_stop_criterion_equals_oracle_at_same_count(torch_cuda, gb300):
    torch = torch_cuda
    M, N = 256, 1024
    cut = _cut(M, N, 9)
    with ctx_for(gb300, torch, M, N) as ctx:
        _cluster_or_skip(ctx, 8)
        ctx.set_tuning(af_cluster=8, af_tol=1e-5, af_iters=120)
        dc = to_dev(torch, cut)
        ctx.stage_fast_entropy(dc, 120)
        got = from_dev(torch, dc).reshape(M, 512)
        tr = ctx.trace()
    k = tr["af_iterations"]
    assert 1 <= k < 120
    assert k % 4 == 0   # the criterion is checked every 4th iteration, before its update
    want, _ = oracle.fast_entropy(cut, iters=k)
    assert rel_l2(got, want) < TOL_IMG


def test_cluster_engine_whole_frame_matches_reference_golden(torch_cuda, gb300):
    import glob
    import os
    torch = torch_cuda
    for path in sorted(glob.glob(os.path.join(os.path.dirname(__file__), "golden", "*.npz"))):
        if os.path.basename(path).startswith(("pc_", "hrrp_", "ingest_")):   # stage fixtures, not frames
            continue
        z = np.load(path)
        M, N = int(z["M"]), int(z["N"])
        flags = (gb300.FLAG_HPC if bool(z["hpc"]) else 0) | (gb300.FLAG_MTRC if bool(z["mtrc"]) else 0)
        echo = golden_echo(z)
        rp = oracle.radar(M, N, B=float(z["B"]), fc=float(z["fc"]), Fs=float(z["Fs"]), Tp=float(z["Tp"]))
        _, tw = oracle.image(echo, z["velocity"], rp, hpc=bool(z["hpc"]), mtrc=bool(z["mtrc"]))
        with ctx_for(gb300, torch, M, N) as ctx:
            _cluster_or_skip(ctx, 8)
            ctx.set_tuning(af_cluster=8)
            ctx.set_ra_shifts(tw["ra_shift"])
            got = ctx.image_host(echo, z["velocity"], flags)
        assert rel_l2(got, z["img"]) < TOL_IMG, path
