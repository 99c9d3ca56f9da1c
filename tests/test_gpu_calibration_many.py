"""Statistics over many tensors in one launch against the oracle, the single-pass calibrator against the two-pass form, and the
KLD search on long, sparse and folded histograms."""
import numpy as np
import pytest
import torch

import oracle
from tpu_mlir_b200.calibration import CaliMathB200, ShardedCalibrator, kld_threshold_host

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def m():
    return CaliMathB200()


@pytest.mark.parametrize("samples", [1, 5])
def test_many_tensors_in_one_launch(m, samples):
    rng = np.random.default_rng(samples)
    sizes = [1, 3, 31, 1024, 32767, 32768, 32769, 70001]      # around the min/max chunk, odd rows (unaligned samples)
    xs = [(rng.standard_normal((samples, n)) * rng.uniform(0.1, 9)).astype(np.float32) for n in sizes]
    xs[3][:] = np.maximum(xs[3], 0)
    xs[4][0] = 0
    dev = [torch.from_numpy(x).cuda() for x in xs]
    mm = m.minmax_many(dev, samples)
    assert np.array_equal(mm[:, :, 0], np.stack([x.min(axis=1) for x in xs])) and np.array_equal(mm[:, :, 1], np.stack([x.max(axis=1) for x in xs]))
    # bins that fit four, one and no copies of the counters in shared memory, a skipped sample, thresholds that differ per sample
    nb = np.tile(np.array([2, 17, 2048, 4096, 2048, 13000, 52000, 60000], np.int32)[:, None], (1, samples))
    nb[4, 0] = 0
    th = np.abs(mm).max(axis=2).astype(np.float32) * np.linspace(1, 1.5, samples, dtype=np.float32) + np.float32(1e-3)
    hists = [torch.zeros(int(nb[t].max()) + 1, dtype=torch.int32, device="cuda") for t in range(len(xs))]
    addr = (np.array([h.data_ptr() for h in hists], np.uint64), np.array([h.numel() for h in hists], np.int64))
    m.histogram_many_into(addr, dev, th, nb)
    for t, x in enumerate(xs):
        want = np.zeros(hists[t].numel(), np.int32)
        for s in range(samples):
            if nb[t, s]:
                oracle.histogram(x[s], th[t, s], int(nb[t, s]), into=want)
        assert np.array_equal(hists[t].cpu().numpy(), want), sizes[t]


def test_single_pass_equals_two_passes(m):
    rng = np.random.default_rng(0)
    S = 11
    scale = np.array([1, 0.5, 1.3, 0.2, 40, 1, 41, 3, 300, 2, 1], np.float32)          # bins grow several times
    acts = {"grow": rng.standard_normal((S, 501)).astype(np.float32) * scale[:, None],
            "restart": rng.standard_normal((S, 64)).astype(np.float32) * np.where(np.arange(S) < 6, 1e-6, 1.0).astype(np.float32)[:, None],
            "flat": np.abs(rng.standard_normal((S, 3, 700))).astype(np.float32), "zero": np.zeros((S, 9), np.float32)}
    acts["zero"][:2] = 0
    dev = {n: torch.from_numpy(a).cuda() for n, a in acts.items()}
    batches = [(0, 4), (4, 5), (5, 11)]

    def run(**kw):
        cal = ShardedCalibrator(lambda b: {n: a[b[0]:b[1]] for n, a in dev.items()}, math=m)
        return cal, cal.run(batches, S, **kw)
    one, r1 = run()
    two, r2 = run(cache_bytes=0)
    assert r1 == r2
    assert all(torch.equal(one.histograms[n], two.histograms[n]) for n in acts)
    assert all(np.array_equal(one._shard[k], two._shard[k]) for k in ("minmax", "hist", "sizes"))


@pytest.mark.parametrize("shape", [(3, 40), (5, 40), (8, 10), (2,), ()])
def test_activations_that_are_not_the_batch_are_refused(m, shape):
    """Cut at the first tensor's batch they would count as other samples, or lose their tail: every driver refuses them."""
    bad = torch.ones(shape, device="cuda")
    for kw in ({}, dict(cache_bytes=1 << 30), dict(cache_bytes=0)):
        cal = ShardedCalibrator(lambda b: {"a": torch.ones((4, 10), device="cuda"), "bad": bad}, math=m)
        with pytest.raises((ValueError, RuntimeError, IndexError)):
            cal.run([0], 4, **kw)


def test_an_activation_that_is_the_same_in_every_sample(m):
    """One row for the whole batch (a position table, say) counts once per sample, as in the driver that keeps the activations."""
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    a, one = torch.randn((4, 100), device="cuda", generator=g), torch.randn((1, 30), device="cuda", generator=g)
    res = []
    for kw in ({}, dict(cache_bytes=1 << 30)):
        cal = ShardedCalibrator(lambda b: {"a": a * b, "one": one}, math=m)
        res.append((cal.run([1.0, 2.0], 8, **kw), cal.histograms["one"].cpu()))
    assert res[0][0] == res[1][0] and torch.equal(res[0][1], res[1][1]) and int(res[0][1].sum()) == 8 * 30


@pytest.mark.parametrize("bins", [128, 256, 2049, 5000, 45000, 131072, 300001])
def test_kld_of_long_and_sparse_histograms(m, bins):
    rng = np.random.default_rng(bins)
    h = rng.poisson(np.maximum(0.02, 400 * np.exp(-np.arange(bins) * 6 / bins))).astype(np.int32)
    h[rng.random(bins) < 0.3] = 0
    h[0] = 30_000_000                    # sums beyond 2^24: the order of the float additions shows
    th = m.find_thresholds([torch.from_numpy(h).cuda()], [0.01])
    hf, wf = oracle.fold_for_kld(h, np.float32(0.01), 128)
    assert th[0] == oracle.kl_diversity_hist(hf, wf, 128)


@pytest.mark.parametrize("bins,dst", [(2048, 256), (1290, 129), (4096, 1024), (500, 500), (45000, 200), (96, 3), (66000, 264)])
def test_kld_with_other_bin_counts(bins, dst):
    """The C symbol takes any number of bins that divides the histogram, also more than the calibration's 128."""
    rng = np.random.default_rng(bins)
    h = rng.poisson(np.maximum(0.02, 400 * np.exp(-np.arange(bins) * 6 / bins))).astype(np.int32)
    h[0] = 30_000_000
    assert kld_threshold_host(h, np.float32(0.02), dst) == oracle.kl_diversity_hist(h, np.float32(0.02), dst)
