"""The non-homogeneous selection of one cluster per frame on images beyond the
keys its threads keep in registers, with ties and with all-equal maps, bit for
bit against the oracle's restatement of VSC_based_Voxel_Line_Select
(MBIR_4D/XT_NHICD.c:164-216); and the passes with work lists against the passes
that visit every super-voxel (same selection, so the same update count)."""
import numpy as np
import pytest

import oracle as O
import phasecon_b200 as pc
from problems import make_problem, to_gpu_problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,frames,kind", [(16, 1, "random"), (34, 2, "ties"), (258, 1, "random"), (300, 2, "ties"),
                                           (64, 1, "equal")])
def test_selection_matches_oracle(n, frames, kind):
    z = np.zeros((frames * 3, 4, n), np.float32)
    ang = np.linspace(0, 3, frames * 3).astype(np.float32)
    pb = pc.Problem(z, np.ones_like(z), ang, np.arange(frames * 3, dtype=np.float32),
                    np.arange(0, frames * 3 + 1, 3, dtype=np.float32), 4, n, frames * 3, frames, rot_center=n / 2)
    s = pc.Session(pb)
    rng = np.random.default_rng(n)
    mag = rng.random((frames, n, n)).astype(np.float32)
    if kind == "ties":
        mag = np.floor(mag * 3).astype(np.float32)
    if kind == "equal":
        mag[:] = 0.25
    got = s.nh_select(mag).astype(bool)
    jj, kk = np.meshgrid(np.arange(n), np.arange(n), indexing="ij")
    mask = (kk + 0.5 - n / 2) ** 2 + (jj + 0.5 - n / 2) ** 2 < (n / 2) ** 2
    s.close()
    for f in range(frames):
        assert np.array_equal(got[f], O.vsc_select(mag[f], int(mask.sum())) & mask)


def test_work_lists_visit_the_selected_columns():
    # one super-voxel per frame in the full sweep: the same map in both runs
    pb, _ = make_problem(ncol=16, nrow=8, nview=40, nframe=2, seed=5)
    updates = []
    for lists in (1, 0):
        o = pc.get_options()
        o.mrf_p, o.nh_work_lists, o.zero_skipping, o.nhicd_passes = pb.mrf_p, lists, 0, 1
        o.sv_size, o.nh_sv_size = 16, 4
        s = pc.Session(to_gpu_problem(pb), options=o)
        s.set_object_zero()
        s.icd_iteration(1)
        updates.append(s.icd_iteration(2).voxel_updates)
        s.close()
    assert updates[0] == updates[1] > 0
