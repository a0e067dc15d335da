"""Kernel-density estimates of log-distributions: drop-in for the reference's
``python/streamlines/kde.py``.

``estimate_univariate_pdf(distbn)`` (kde.py:116-194) and
``estimate_bivariate_pdf(distbn)`` (kde.py:35-114) keep the reference's
contract: they read the distribution object's fields (``logx_data`` or
``logxy_data``, ``n_data``, ``bandwidth``, bin and pdf spacings, ``kernel``),
set its Silverman-scaled kernel widths in log space, run histogram + smoothing
on the device (``libslm_b200.so``), and return ``(pdf, histogram)`` normalised
exactly as the reference normalises them.  The kernel parameters are the
reference's KDE macros (pocl.py:196-222).
"""
from __future__ import annotations

import numpy as np
import torch

from . import kernels
from .device import cuda_device, download
from .params import params_from_options, compile_options
from .useful import vprint


def kde_params(distbn, kernel_fn):
    """The KDE parameter block for one kernel, as the reference's -D macros."""
    return params_from_options(compile_options(distbn, kernel_fn, job_type="kde"))


def _device(distbn):
    return cuda_device(getattr(distbn, "cl_platform", 0) or 0, getattr(distbn, "cl_device", 0) or 0)


# Data of this many values on: their spread is formed on the device, in double,
# from the copy the histogram is counted from.  np.std takes three passes over
# the host array (2 M float32: 1.5 ms; 1 M pairs, by column: 3.2 ms), the device
# 0.03 ms and one round trip.
DEVICE_STD_FROM = 1 << 16


def _std_on_device(array):
    return array.dtype == np.float32 and array.size >= DEVICE_STD_FROM


def prepare_univariate(distbn, stddev=None):
    """Silverman-scaled kernel width in log space (kde.py:151-158);
    ``stddev``: the data's standard deviation, where it is known."""
    stddev_x = np.std(distbn.logx_data) if stddev is None else stddev[0]
    distbn.kdf_width_x = 1.06 * stddev_x * np.power(distbn.n_data, -0.2) * distbn.bandwidth
    distbn.kdf_width_y = 0.0
    distbn.n_kdf_part_points_x = np.uint32(np.floor(distbn.kdf_width_x / distbn.pdf_dx)) // 2
    distbn.n_kdf_part_points_y = 0


def prepare_bivariate(distbn, stddev=None):
    """Kernel widths of both axes (kde.py:71-82); ``stddev``: the columns'
    standard deviations, where they are known."""
    sl_array = distbn.logxy_data
    stddev_x, stddev_y = (np.std(sl_array[:, 0]), np.std(sl_array[:, 1])) if stddev is None else stddev
    distbn.kdf_width_x = 1.06 * stddev_x * np.power(distbn.n_data, -0.2) * distbn.bandwidth
    distbn.kdf_width_y = 1.06 * stddev_y * np.power(distbn.n_data, -0.2) * distbn.bandwidth
    distbn.n_kdf_part_points_x = (np.uint32(np.floor(distbn.kdf_width_x / distbn.bin_dx)) // 2)
    distbn.n_kdf_part_points_y = (np.uint32(np.floor(distbn.kdf_width_y / distbn.bin_dy)) // 2)


def estimate_univariate_pdf(distbn, do_detrend=False, logx_vec=None):
    verbose = getattr(distbn, "verbose", False)
    vprint(verbose, "Estimating univariate pdf...", end="")
    dev = _device(distbn)
    sl_array = distbn.logx_data
    bin_dx = distbn.bin_dx
    nb, npp = int(distbn.n_hist_bins), int(distbn.n_pdf_points)
    with torch.cuda.device(dev):
        data_d = torch.from_numpy(np.ascontiguousarray(sl_array, dtype=np.float32).reshape(-1)).to(dev)
        prepare_univariate(distbn, kernels.column_std(data_d) if _std_on_device(sl_array) else None)
        prm = kde_params(distbn, "histogram_univariate")  # the KDE kernels share their macros
        hist_d = torch.zeros(nb, dtype=torch.uint32, device=dev)
        kernels.histogram_univariate(prm, data_d, hist_d)
        histogram_array = hist_d.cpu().numpy().reshape(nb, 1)
        if do_detrend:
            from scipy.stats import norm
            x = logx_vec
            pdf = histogram_array.copy().astype(np.float32)
            mean = (np.sum(x * pdf) / np.sum(pdf))
            stddev = np.sqrt(np.sum((x - mean) ** 2 * pdf) / np.sum(pdf))
            pdf /= norm.pdf(logx_vec, mean, stddev)
            pdf /= np.sum(pdf)
            pdf *= np.sum(histogram_array)
            histogram_array = pdf.copy().astype(np.uint32)
            hist_d = torch.from_numpy(np.ascontiguousarray(histogram_array).reshape(-1)).to(dev)
        pdf_d = torch.zeros(npp, dtype=torch.float32, device=dev)
        kernels.pdf_univariate(prm, hist_d, pdf_d)
        pdf_array = pdf_d.cpu().numpy().reshape(npp, 1)
    vprint(verbose, "done")
    # the reference normalises by Python's builtin sum over the rows: a
    # left-to-right sum in the array's own dtype, which accumulate gives
    return (pdf_array / (_row_sum(pdf_array) * bin_dx),
            histogram_array / (_row_sum(histogram_array) * bin_dx))


def _row_sum(a):
    """``sum(a)`` (builtin) of an [n, 1] array: the rows added left to right in
    a's dtype (kde.py:193-194)."""
    if a.shape[0] == 0:
        return 0
    return np.add.accumulate(a, axis=0, dtype=a.dtype)[-1]


def estimate_bivariate_pdf(distbn):
    verbose = getattr(distbn, "verbose", False)
    vprint(verbose, "Estimating bivariate pdf...", end="")
    dev = _device(distbn)
    sl_array = distbn.logxy_data
    bin_dx, bin_dy = distbn.bin_dx, distbn.bin_dy
    nb, npp = int(distbn.n_hist_bins), int(distbn.n_pdf_points)
    with torch.cuda.device(dev):
        data_d = torch.from_numpy(np.ascontiguousarray(sl_array, dtype=np.float32)).to(dev)
        prepare_bivariate(distbn, kernels.column_std(data_d) if _std_on_device(sl_array) else None)
        prm = kde_params(distbn, "histogram_bivariate")  # the KDE kernels share their macros
        hist_d = torch.zeros(nb * nb, dtype=torch.uint32, device=dev)
        kernels.histogram_bivariate(prm, data_d, hist_d)
        part_d = torch.zeros(nb * nb, dtype=torch.float32, device=dev)
        kernels.pdf_bivariate_rows(prm, hist_d, part_d)
        pdf_d = torch.zeros(npp * npp, dtype=torch.float32, device=dev)
        kernels.pdf_bivariate_cols(prm, part_d, pdf_d)
        # every pair is in one bin, so the counts sum to the number of pairs
        scale = np.uint64(sl_array.shape[0]) * bin_dx * bin_dy
        if np.asarray(scale).dtype == np.float64 and scale != 0:
            # counts over their sum and the bins' area, divided on the device
            histogram, = download((kernels.scale_counts(hist_d, scale),), "histogram", pinned=True)
            histogram = histogram.reshape(nb, nb)
        else:
            histogram = hist_d.cpu().numpy().reshape(nb, nb) / scale
        pdf_array = pdf_d.cpu().numpy().reshape(npp, npp)
    vprint(verbose, "done")
    return pdf_array / (np.sum(pdf_array) * bin_dx * bin_dy), histogram
