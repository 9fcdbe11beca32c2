"""The projectors against FP64 sums over the system matrix they read.

Cases: images no tile divides, slabs of 4 to 72 rows in steps of two (each vector
width, a last chunk that is partly filled), one or an odd number of views a frame,
voxel scales with one, two and three words a record, a z scale that is no power of
two, objects with empty columns.

Tolerances: A x is summed in FP64 and rounded once, 2^-24 of the value (1.2e-7 holds
it with the order of the sum). A^T s sums twelve products in FP32 before FP64: at most
14 2^-24 of the sum of their magnitudes, and 2^-24 for the result, 1e-6 together.
"""
import numpy as np
import pytest

import phasecon_b200 as pc
from problems import make_problem, to_gpu_problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ncol,nrow,nview,nframe,mxy,mz", [
    (24, 8, 11, 1, 1, 1),
    (36, 6, 10, 2, 1, 1),       # two rows a lane
    (50, 18, 37, 2, 1, 1),
    (34, 36, 9, 1, 1, 1),       # 32 + 4 rows
    (18, 72, 5, 5, 1, 1),       # one view a frame
    (40, 32, 70, 2, 1, 2),
    (40, 16, 7, 1, 1, 8),
    (24, 12, 6, 1, 1, 3),       # a z scale that is no power of two
    (64, 8, 21, 2, 2, 2),
    (48, 6, 9, 1, 3, 1),
    (64, 20, 13, 1, 4, 4),
    (128, 4, 3, 1, 1, 1),
])
def test_projectors_match_fp64_sums(ncol, nrow, nview, nframe, mxy, mz):
    pb, _ = make_problem(ncol=ncol, nrow=nrow, nview=nview, nframe=nframe)
    s = pc.Session(to_gpu_problem(pb), mult_xy=mxy, mult_z=mz, options=pc.get_options())
    first, count, vals = s.amatrix()
    T, Z, Y, X = s.shape
    Np, Nr, Nt = s.sino_shape
    rng = np.random.default_rng(7)
    x = rng.normal(size=s.shape).astype(np.float32)
    x[:, :, rng.random((Y, X)) < 0.3] = 0
    y = rng.normal(size=s.sino_shape).astype(np.float32)
    # the frame of each view: those the frames' intervals hold, as the session assigns them
    frame = np.full(Np, -1)
    for v in range(Np):
        for f in range(T):
            if pb.recon_times[f] <= pb.proj_times[v] < pb.recon_times[f + 1]:
                frame[v] = f
    ax, mag = np.zeros((Np, Nr, Nt)), np.zeros((Np, Nr, Nt))
    aty, aty_mag = np.zeros((T, Nt, Y, X)), np.zeros((T, Nt, Y, X))
    xt = np.repeat(x.astype(np.float64), mz, axis=1)  # [T][Nt][Y][X]
    for v in range(Np):
        f = frame[v]
        if f < 0:
            continue
        for q in range(vals.shape[-1]):
            jj, kk = np.nonzero(count[v] > q)
            r, a = first[v][jj, kk] + q, vals[v][jj, kk, q].astype(np.float64)
            p = a[:, None] * xt[f][:, jj, kk].T
            np.add.at(ax[v], r, p)
            np.add.at(mag[v], r, np.abs(p))
            b = a[:, None] * y[v].astype(np.float64)[r]
            np.add.at(aty[f].transpose(1, 2, 0), (jj, kk), b)
            np.add.at(aty_mag[f].transpose(1, 2, 0), (jj, kk), np.abs(b))
    got = s.forward_project(x)
    assert np.all(np.abs(got - ax) <= 1.2e-7 * np.abs(ax) + 1e-13 * mag)
    if mz & (mz - 1):
        return  # the adjoint over such a scale has its own grouping of rows
    back = s.back_project(y)
    ref = aty.reshape(T, Z, mz, Y, X).sum(2)
    ref_mag = aty_mag.reshape(T, Z, mz, Y, X).sum(2)
    assert np.all(np.abs(back - ref) <= 1e-6 * ref_mag)
