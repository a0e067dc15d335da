"""GPU KDE kernels against the oracle.

Histograms are integer counts: bit-exact.  Smoothed pdfs are fp64 sums of
the reference's terms in the reference's order, rounded to float; exp() and
cos() come from CUDA instead of the host libm, so the tolerance is stated per
point: relative error median <= 1e-7 and 99th percentile <= 1e-6 (max <= 1e-5),
relative to the pdf's maximum.
"""
import numpy as np
import pytest
import torch

import oracle as O
from kde_cases import bivariate, univariate
from slm_b200 import kde, kernels

pytestmark = pytest.mark.gpu
SHAPES = ["tophat", "triangle", "epanechnikov", "cosine", "gaussian"]


def _close(got, want):
    scale = max(float(np.abs(want).max()), 1e-30)
    rel = np.abs(got.astype(np.float64) - want.astype(np.float64)) / scale
    assert np.median(rel) <= 1e-7, np.median(rel)
    assert np.percentile(rel, 99) <= 1e-6, np.percentile(rel, 99)
    assert rel.max() <= 1e-5, rel.max()


@pytest.mark.parametrize("kind", SHAPES)
@pytest.mark.parametrize("nb,npp", [(2048, 256), (8192, 1024)])
def test_univariate_kernels(kind, nb, npp):
    d, prm = univariate(kind, n_hist_bins=nb, n_pdf_points=npp, n=200000)
    data = np.ascontiguousarray(d.logx_data.reshape(-1), dtype=np.float32)
    hist_o = O.histogram_univariate(prm, data)
    pdf_o = O.pdf_univariate(prm, hist_o)
    data_d = torch.from_numpy(data).cuda()
    hist_d = torch.zeros(nb, dtype=torch.uint32, device="cuda")
    kernels.histogram_univariate(prm, data_d, hist_d)
    pdf_d = torch.zeros(npp, dtype=torch.float32, device="cuda")
    kernels.pdf_univariate(prm, hist_d, pdf_d)
    torch.cuda.synchronize()
    assert np.array_equal(hist_d.cpu().numpy(), hist_o)
    _close(pdf_d.cpu().numpy(), pdf_o)


@pytest.mark.parametrize("kind", SHAPES)
def test_bivariate_kernels(kind):
    d, prm = bivariate(kind, n=100000)
    nb, npp = int(d.n_hist_bins), int(d.n_pdf_points)
    data = np.ascontiguousarray(d.logxy_data, dtype=np.float32)
    hist_o = O.histogram_bivariate(prm, data)
    part_o = O.pdf_bivariate_rows(prm, hist_o)
    pdf_o = O.pdf_bivariate_cols(prm, part_o)
    data_d = torch.from_numpy(data).cuda()
    hist_d = torch.zeros(nb * nb, dtype=torch.uint32, device="cuda")
    kernels.histogram_bivariate(prm, data_d, hist_d)
    part_d = torch.zeros(nb * nb, dtype=torch.float32, device="cuda")
    kernels.pdf_bivariate_rows(prm, hist_d, part_d)
    pdf_d = torch.zeros(npp * npp, dtype=torch.float32, device="cuda")
    # the cols pass is checked on the oracle's partial pdf, the rows pass separately
    kernels.pdf_bivariate_cols(prm, torch.from_numpy(part_o).cuda(), pdf_d)
    torch.cuda.synchronize()
    assert np.array_equal(hist_d.cpu().numpy(), hist_o)
    _close(part_d.cpu().numpy(), part_o)
    _close(pdf_d.cpu().numpy(), pdf_o)


def test_estimate_univariate_pdf_end_to_end():
    d, prm = univariate("gaussian", n_hist_bins=8192, n_pdf_points=1024, n=300000)
    d.bandwidth = 2.0 / 2.0
    pdf, hist = kde.estimate_univariate_pdf(d)
    prm = kde.kde_params(d, "pdf_univariate")
    data = np.ascontiguousarray(d.logx_data.reshape(-1), dtype=np.float32)
    hist_o = O.histogram_univariate(prm, data).reshape(-1, 1)
    pdf_o = O.pdf_univariate(prm, hist_o).reshape(-1, 1)
    assert pdf.shape == (1024, 1) and hist.shape == (8192, 1)
    assert np.array_equal(hist, hist_o / (sum(hist_o) * d.bin_dx))
    _close(pdf, pdf_o / (sum(pdf_o) * d.bin_dx))


def test_estimate_bivariate_pdf_end_to_end():
    d, prm = bivariate("epanechnikov", n=50000)
    pdf, hist = kde.estimate_bivariate_pdf(d)
    assert pdf.shape == (64, 64) and hist.shape == (256, 256)
    assert abs(float(np.sum(hist) * d.bin_dx * d.bin_dy) - 1.0) < 1e-6
    assert abs(float(np.sum(pdf) * d.bin_dx * d.bin_dy) - 1.0) < 1e-4


def test_channel_threshold_from_device_pdf():
    """estimate_channel_threshold (device KDE + host consumers) equals the
    consumers run on the oracle's pdf of the same data."""
    from types import SimpleNamespace

    from slm_b200 import analysis as A
    rng = np.random.default_rng(21)
    nx, ny = 300, 280
    hill = rng.lognormal(2.5, 0.5, (nx, ny))
    chan = rng.lognormal(6.0, 0.8, (nx, ny))
    slt = np.where(rng.random((nx, ny)) < 0.08, chan, hill).astype(np.float32)
    sla = (slt * rng.uniform(0.5, 1.5, (nx, ny))).astype(np.float32)
    mask = rng.random((nx, ny)) < 0.05
    data = SimpleNamespace(slt_array=np.stack([slt, slt], 2), sla_array=np.stack([sla, sla], 2), mask_array=mask)
    d = A.compute_marginal_distribn_dslt(data)
    thr = A.estimate_channel_threshold(data)
    assert thr is not None and thr == d.channel_threshold_x
    # the same consumers on the oracle's pdf of the same selection
    prm = kde.kde_params(d, "pdf_univariate")
    x = np.ascontiguousarray(d.logx_data.reshape(-1), dtype=np.float32)
    hist_o = O.histogram_univariate(prm, x).reshape(-1, 1)
    pdf_o = O.pdf_univariate(prm, hist_o).reshape(-1, 1)
    pdf_o = pdf_o / (sum(pdf_o) * d.bin_dx)
    o = A.compute_marginal_distribn_dslt(data)  # fresh object, same data selection
    o.pdf = pdf_o.astype(np.float32)
    o.cdf = np.cumsum(o.pdf) * o.bin_dx
    o.pdf /= o.cdf[-1]
    o.cdf /= o.cdf[-1]
    for attr in ("mode_x", "channel_threshold_x"):
        if hasattr(o, attr):
            delattr(o, attr)
    o.find_modes()
    o.statistics()
    o.locate_threshold()
    assert o.mode_i == d.mode_i
    assert o.channel_threshold_i == d.channel_threshold_i


@pytest.mark.parametrize("nb,npp,n", [(256, 128, 4095), (256, 128, 4096), (2048, 256, 8191), (2048, 256, 8193),
                                      (12288, 128, 60001), (12289 + 127, 128, 60001), (64, 64, 1000003),
                                      (4096, 33, 1)])
def test_univariate_histogram_in_shared_memory_and_not(nb, npp, n):
    """Sizes on either side of the rule for counting in shared memory; the pdf
    with more, fewer and as many weights as its table holds."""
    nb -= nb % npp
    rng = np.random.default_rng(nb + n)
    d, _ = univariate("gaussian", n_hist_bins=nb, n_pdf_points=npp, n=20000, bandwidth=6.0)
    prm = kde.kde_params(d, "pdf_univariate")
    data = rng.choice(np.ascontiguousarray(d.logx_data.reshape(-1), dtype=np.float32), n)
    hist_d = torch.full((nb,), 3, dtype=torch.int32, device="cuda").view(torch.uint32)  # added to, not cleared
    kernels.histogram_univariate(prm, torch.from_numpy(data).cuda(), hist_d)
    pdf_d = torch.zeros(npp, dtype=torch.float32, device="cuda")
    hist_o = O.histogram_univariate(prm, data)
    kernels.pdf_univariate(prm, torch.from_numpy(hist_o).cuda(), pdf_d)
    torch.cuda.synchronize()
    assert np.array_equal(hist_d.cpu().numpy(), hist_o + 3)
    _close(pdf_d.cpu().numpy(), O.pdf_univariate(prm, hist_o))


@pytest.mark.parametrize("n", [1, 255, 512, 513, 131073, 1000003])
@pytest.mark.parametrize("cols", [1, 2])
def test_column_std_against_64_bits(n, cols):
    """Formed in double from n values of |x| < 30 with spread >= 0.5 and rounded
    once to float32: within 2^-24 of the 64-bit value, but for the double sums'
    own error (n 2^-53 of them, below 2^-30)."""
    rng = np.random.default_rng(n * 3 + cols)
    x = (3.0 + rng.standard_normal((n, cols)) * np.array([0.8, 0.5])[:cols]).astype(np.float32)
    got = kernels.column_std(torch.from_numpy(x if cols == 2 else x[:, 0].copy()).cuda())
    want = x.astype(np.float64).std(axis=0)
    for g, w in zip(got, want):
        assert g.dtype == np.float32 and abs(float(g) - w) <= w * (2.0 ** -24 + 2.0 ** -30)


@pytest.mark.parametrize("nb,n", [(64, 16405), (64, 16406), (2048, 39684), (2048, 39685), (12288, 855243),
                                  (12288, 855244)])
def test_univariate_histogram_on_either_side_of_the_rule(nb, n):
    rng = np.random.default_rng(nb + n)
    d, _ = univariate("gaussian", n_hist_bins=nb, n_pdf_points=64, n=20000, bandwidth=6.0)
    prm = kde.kde_params(d, "pdf_univariate")
    data = rng.choice(np.ascontiguousarray(d.logx_data.reshape(-1), dtype=np.float32), n)
    hist_d = torch.full((nb,), 3, dtype=torch.int32, device="cuda").view(torch.uint32)
    kernels.histogram_univariate(prm, torch.from_numpy(data).cuda(), hist_d)
    assert np.array_equal(hist_d.cpu().numpy(), O.histogram_univariate(prm, data) + 3)


def test_univariate_histogram_of_few_values_in_many_bins():
    """60000 values in 12288 bins are counted in memory, as in 16384: about 3 us
    (26 us in the shared memory of the one block that four values a bin leave)."""
    def us(nb):
        d, _ = univariate("gaussian", n_hist_bins=nb, n_pdf_points=64, n=60000, bandwidth=6.0)
        prm = kde.kde_params(d, "pdf_univariate")
        data = torch.from_numpy(np.ascontiguousarray(d.logx_data.reshape(-1), dtype=np.float32)).cuda()
        hist = torch.zeros(nb, dtype=torch.uint32, device="cuda")
        kernels.histogram_univariate(prm, data, hist)
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            for _ in range(20):
                kernels.histogram_univariate(prm, data, hist)
        times = []
        for _ in range(9):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            g.replay()
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b) * 50.0)
        return sorted(times)[4]

    assert us(12288) < 3.0 * us(16384)


def test_univariate_histogram_of_as_many_values_as_a_count_holds():
    """2^32 - 400 values: a chunk sixteen times over, but for its last 400."""
    nb, chunk, cut = 16384, 1 << 28, 400
    d, _ = univariate("gaussian", n_hist_bins=nb, n_pdf_points=64, n=20000, bandwidth=6.0)
    prm = kde.kde_params(d, "pdf_univariate")
    lo, span = float(d.logx_min), float(d.logx_range)
    data = torch.empty(16 * chunk, dtype=torch.float32, device="cuda")
    data[:chunk].uniform_(lo, lo + span, generator=torch.Generator(device="cuda").manual_seed(3))
    for k in range(1, 16):
        data[k * chunk:(k + 1) * chunk] = data[:chunk]
    hist = [torch.zeros(nb, dtype=torch.uint32, device="cuda") for _ in range(3)]
    for h, part in zip(hist, (data[:chunk], data[chunk - cut:chunk], data[:16 * chunk - cut])):
        kernels.histogram_univariate(prm, part, h)
    one, last, whole = (h.cpu().numpy().astype(np.int64) for h in hist)
    assert one.sum() == chunk and last.sum() == cut
    assert np.array_equal(whole, 16 * one - last)
