"""The register-blocked Schwarz factorisation at the sizes where it can go wrong: domains of 1
to 32 vertices (register blocks of 24, 48, 72 and 96 rows and their remainders), a domain whose
pivot fails, and the coarse level. The applied z = W^T W r against the oracle's dense solve; W
is FP64 rounded to FP32, so z is off by a few times 2^-24 of sum |W| |W^T| |r|: the same 1e-4
of the largest entry as the apply's other tests."""
import numpy as np
import pytest

import oracle_py as O
from mguso import Bsr, Schwarz, scenes

pytestmark = pytest.mark.gpu


def applied(a, s, r):
    import torch
    st = torch.cuda.current_stream().cuda_stream
    s.factor(st)
    rd = torch.from_numpy(r).cuda()
    zd = torch.full_like(rd, float("nan"))
    s.apply(rd.data_ptr(), zd.data_ptr(), st)
    torch.cuda.synchronize()
    return zd.cpu().numpy()


@pytest.mark.parametrize("domain", [1, 2, 7, 8, 9, 15, 16, 17, 23, 24, 25, 31, 32])
def test_domain_sizes(ctx, domain):
    nb, rp, col, val = scenes.grid_bsr(23, 5)
    N, srp, sci, svv = scenes.bsr_to_csr(nb, rp, col, val)
    a = Bsr(ctx, nb, rp, col, val)
    s = Schwarz(a, domain)
    r = np.random.default_rng(domain).standard_normal(N).astype(np.float32)
    want = O.schwarz_apply(N, srp, sci, svv, domain, r.astype(np.float64))
    assert np.abs(applied(a, s, r) - want).max() <= 1e-4 * np.abs(want).max()


@pytest.mark.parametrize("entry", [0, 17, 95])
def test_failed_pivot_falls_back_to_the_diagonal(ctx, entry):
    """One negative diagonal entry in the first domain: its factor is the floored diagonal's (1
    where that is not positive), the other domains are unaffected."""
    nb, rp, col, val = scenes.grid_bsr(23, 5)
    val = val.copy()
    N, srp, sci, svv = scenes.bsr_to_csr(nb, rp, col, val)
    dom, _ = O.schwarz_domains(N, srp, sci, 32)
    v = int(np.flatnonzero(dom == 0)[entry // 3])
    k = [k for k in range(rp[v], rp[v + 1]) if col[k] == v][0]
    val[k, entry % 3, entry % 3] = -50.0
    N, srp, sci, svv = scenes.bsr_to_csr(nb, rp, col, val)
    a = Bsr(ctx, nb, rp, col, val)
    s = Schwarz(a, 32)
    r = np.random.default_rng(1).standard_normal(N).astype(np.float32)
    want = O.schwarz_apply(N, srp, sci, svv, 32, r.astype(np.float64))
    got = applied(a, s, r)
    assert np.abs(got - want).max() <= 1e-4 * np.abs(want).max()


@pytest.mark.parametrize("domain", [3, 16, 32])
def test_coarse_level(ctx, domain):
    nb, rp, col, val = scenes.grid_bsr(40, 7)
    N, srp, sci, svv = scenes.bsr_to_csr(nb, rp, col, val)
    a = Bsr(ctx, nb, rp, col, val)
    s = Schwarz(a, domain, levels=2, weight=0.7)
    r = np.random.default_rng(2).standard_normal(N).astype(np.float32)
    want = O.schwarz_ml_apply(N, srp, sci, svv, domain, 0.7, r.astype(np.float64))
    assert np.abs(applied(a, s, r) - want).max() <= 1e-4 * np.abs(want).max()
