"""The cost kernel's prior term for exponents q beyond the default 2, whose powers of small
differences leave FP64's range, against the same sum in FP64 (qGGMRF potential of
MBIR_4D/XT_ICD_update.c:82-90 over the causal neighbours of :206-298).

Tolerance: terms off by a few 2^-50 and N <= 2e5 positive terms in any order, N 2^-53.
"""
import numpy as np
import pytest

import oracle as O
import phasecon_b200 as pc
from problems import make_problem, to_gpu_problem

pytestmark = pytest.mark.gpu


def prior(g, x):
    f = np.array(g.spatial_filter).reshape(3, 3, 3)

    def rho(d, sq, sqp, c):
        a = np.abs(d.astype(np.float64))
        return a**g.q / sq / (c + a**(g.q - g.p) / sqp)

    total = 0.0
    T, Z, Y, X = x.shape
    for dz in (0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                if (dz, dy, dx) <= (0, 0, 0):
                    continue
                z, y0, y1 = slice(0, Z - dz), max(0, -dy), Y - max(0, dy)
                x0, x1 = max(0, -dx), X - max(0, dx)
                d = x[:, z, y0:y1, x0:x1] - x[:, dz:, y0 + dy:y1 + dy, x0 + dx:x1 + dx]
                total += f[1 + dz, 1 + dy, 1 + dx] * rho(d, g.sigma_s_q, g.sigma_s_q_p, g.c_s).sum()
    return total + g.time_filter * rho(x[:-1] - x[1:], g.sigma_t_q, g.sigma_t_q_p, g.c_t).sum()


@pytest.mark.parametrize("q,p,decades", [
    (2.0, 1.2, (-3, -1)),
    (3.5, 1.2, (-38, -1)),
    (6.5, 1.2, (-44, -1)),
    (6.75, 5.0, (-44, -1)),
    (8.0, 1.2, (-44, -1)),
    (10.0, 9.0, (-38, 0)),
])
def test_prior_term_over_exponents(q, p, decades):
    pb, obj = make_problem(ncol=16, nrow=8, nview=24, nframe=2, seed=3)
    pb.sig_s = pb.sig_t = 1.0  # sigma^q stays of order one
    rng = np.random.default_rng(5)
    e = rng.integers(decades[0], decades[1] + 1, size=obj.shape)
    x = (rng.normal(size=obj.shape) * 10.0**e * (rng.random(obj.shape) < 0.5)).astype(np.float32)
    x[0, :, :4] = x[1, :, :4] = (1e-32 * rng.normal(size=x[0, :, :4].shape)).astype(np.float32)  # small differences only
    opt = pc.get_options()
    opt.mrf_p, opt.mrf_q = p, q
    s = pc.Session(to_gpu_problem(pb), options=opt)
    s.set_object(x)
    got = s.cost()[2]
    s.close()
    g = O.Oracle(pb).g
    delta_recon = 12.0  # views a frame
    g.q, g.p = q, p
    g.sigma_s_q, g.sigma_s_q_p, g.sigma_t_q, g.sigma_t_q_p = 1.0, 1.0, delta_recon**q, delta_recon**(q - p)
    assert got == pytest.approx(prior(g, x), rel=1e-10)
