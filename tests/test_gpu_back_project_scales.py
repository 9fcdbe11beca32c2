"""Back projection over z scales that do not divide a chunk of 32 detector rows: a slice's
rows straddle chunks, are more than one chunk holds, or are no power of two in number.

Tolerance: the products are summed in FP64 and rounded once, 2^-24 of the value; 1.2e-7
holds it with the order of the sum (N <= 3e4 terms, N 2^-53 of their magnitudes).
"""
import numpy as np
import pytest

import phasecon_b200 as pc
from problems import make_problem, to_gpu_problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ncol,nrow,nview,nframe,mxy,mz", [
    (24, 6, 6, 1, 1, 3),
    (24, 12, 6, 1, 1, 6),
    (20, 42, 7, 1, 1, 3),       # slices across the edge of the first 32 rows
    (18, 36, 5, 2, 1, 9),
    (16, 102, 5, 1, 1, 3),      # 34 slices
    (16, 34, 4, 1, 1, 17),
    (16, 96, 5, 1, 1, 48),      # more rows a slice than lanes
    (16, 64, 5, 1, 1, 64),
    (32, 20, 9, 2, 2, 5),       # longer records
    (48, 12, 6, 1, 3, 12),
    (64, 14, 7, 1, 4, 7),
])
def test_back_projection_matches_fp64_sums(ncol, nrow, nview, nframe, mxy, mz):
    pb, _ = make_problem(ncol=ncol, nrow=nrow, nview=nview, nframe=nframe)
    s = pc.Session(to_gpu_problem(pb), mult_xy=mxy, mult_z=mz, options=pc.get_options())
    first, count, vals = s.amatrix()
    T, Z, Y, X = s.shape
    Np, Nr, Nt = s.sino_shape
    y = np.random.default_rng(7).normal(size=s.sino_shape).astype(np.float32)
    ref, mag = np.zeros((T, Z, Y, X)), np.zeros((T, Z, Y, X))
    for v in range(Np):
        f = next((f for f in range(T) if pb.recon_times[f] <= pb.proj_times[v] < pb.recon_times[f + 1]), None)
        if f is None:
            continue
        slices = y[v].astype(np.float64).reshape(Nr, Z, mz)
        sums, sizes = slices.sum(2), np.abs(slices).sum(2)
        for q in range(vals.shape[-1]):
            jj, kk = np.nonzero(count[v] > q)
            a = vals[v][jj, kk, q].astype(np.float64)[:, None]
            np.add.at(ref[f].transpose(1, 2, 0), (jj, kk), a * sums[first[v][jj, kk] + q])
            np.add.at(mag[f].transpose(1, 2, 0), (jj, kk), a * sizes[first[v][jj, kk] + q])
    back = s.back_project(y)
    s.close()
    assert np.all(np.abs(back - ref) <= 1.2e-7 * np.abs(ref) + 1e-11 * mag)
