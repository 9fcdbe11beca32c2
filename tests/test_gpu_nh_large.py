"""The non-homogeneous selection where the image is filtered by a launch of its own (beyond
the 65,536 columns whose keys a cluster keeps in registers), bit for bit against the
oracle's restatement of VSC_based_Voxel_Line_Select (MBIR_4D/XT_NHICD.c:164-216): just
past the line, rows that no block divides, several frames, ties."""
import numpy as np
import pytest

import oracle as O
import phasecon_b200 as pc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,frames,kind", [(256, 2, "random"), (258, 3, "ties"), (334, 1, "random"), (514, 2, "random"),
                                           (600, 1, "equal")])
def test_large_selection_matches_oracle(n, frames, kind):
    z = np.zeros((frames * 3, 4, n), np.float32)
    ang = np.linspace(0, 3, frames * 3).astype(np.float32)
    pb = pc.Problem(z, np.ones_like(z), ang, np.arange(frames * 3, dtype=np.float32),
                    np.arange(0, frames * 3 + 1, 3, dtype=np.float32), 4, n, frames * 3, frames, rot_center=n / 2)
    s = pc.Session(pb)
    mag = np.random.default_rng(n).random((frames, n, n)).astype(np.float32)
    if kind == "ties":
        mag = np.floor(mag * 3).astype(np.float32)
    if kind == "equal":
        mag[:] = 0.25
    got = s.nh_select(mag).astype(bool)
    s.close()
    jj, kk = np.meshgrid(np.arange(n), np.arange(n), indexing="ij")
    mask = (kk + 0.5 - n / 2) ** 2 + (jj + 0.5 - n / 2) ** 2 < (n / 2) ** 2
    for f in range(frames):
        assert np.array_equal(got[f], O.vsc_select(mag[f], int(mask.sum())) & mask)
